"""Timed cases of the transcription path, from a four-second request to an hour of audio.

Each case is one call (or one short chain of calls) that a program built on this package
makes: `PipelineEngine.transcribe_batch` / `transcribe_stream` / `encode_chunk`, the log-mel
frontend, the subsampling stage, and the linear / feed-forward / attention building blocks at
the sizes of the benchmark configurations.  Weights are the package's seeded synthetic tensors
and are laid out once per process; the inputs of a case come from its seed alone.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

pk = importlib.import_module("l4-parakeet-rs_b200")
L, ops = pk.lib, pk.ops

LAYERS = 24
MODEL_SEED = 4
CALIBRATION_SEED = 100
WIDTH, FF, HIDDEN, BINS = 1024, 4096, 640, 128
TOKEN_ROWS = 1030
HOP = 160
LIVE = 0.3                        # share of the hidden tiles that the tile threshold keeps
BATCH_UTTERANCES, BATCH_FRAMES = 8, 6000
LONG_UTTERANCES, LONG_FRAMES = 2, 12000
HOUR_FRAMES = 360000


def listed():
    return [
        # voice command, the smallest call: one short utterance on an engine sized for a batch of minutes
        dict(name="request_4s", kind="transcribe", engine="batch", frames="400"),
        # one utterance per request, the batch-1 benchmark configuration
        dict(name="request_60s", kind="transcribe", engine="batch", frames="6000"),
        # the headline workload: one GPU's share of 64 utterances of 60 s
        dict(name="batch_8x60s", kind="transcribe", engine="batch", frames=" ".join(["6000"] * 8)),
        # a batch as it arrives in serving: no two utterances of the same length, most far below the cap
        dict(name="batch_ragged", kind="transcribe", engine="batch",
             frames="331 1207 2765 598 5893 1764 901 3520"),
        # a long request with the two-layer prediction network of the reference's model (INT8 LSTM cache)
        dict(name="request_120s_two_layer", kind="transcribe", engine="long", frames="12000"),
        # bulk transcription: batches follow each other and overlap
        dict(name="stream_6_of_8x60s", kind="stream", batches=6, utterances=8, frames=6000),
        # an hour of audio as one sequence: mel upload, subsampling, blocks, encoder projection
        dict(name="encode_3600s", kind="encode", frames=HOUR_FRAMES),
        # PCM to normalised log-mel for a batch
        dict(name="frontend_8x60s", kind="frontend", utterances=8, samples=959999),
        # subsampling with E4M3 activations and weights (the long-request variant)
        dict(name="subsampling_fp8_8x60s", kind="subsampling", utterances=8, frames=6000, precision="fp8"),
        # fp16 x INT4 group-128 linear, 60 s of encoder rows
        dict(name="int4_linear_750", kind="int4_linear", rows=750, n=FF, k=WIDTH),
        # feed-forward block with 70 % zero hidden tiles, 60 s of encoder rows
        dict(name="ff_block_750", kind="ff_block", rows=750),
        # attention module over an hour: INT8 QKV, local attention, INT4 output projection
        dict(name="attention_45000", kind="attention", rows=45000),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["transcribe"] * 4 + ["long", "stream", "encode", "frontend", "subsampling", "int4_linear",
                                            "ff_block", "attention"])
    if kind == "transcribe":
        frames = [_log_int(rng, 50, BATCH_FRAMES) for _ in range(rng.randint(1, BATCH_UTTERANCES))]
        return dict(kind="transcribe", engine="batch", frames=" ".join(map(str, frames)))
    if kind == "long":
        frames = [_log_int(rng, 800, LONG_FRAMES) for _ in range(rng.randint(1, LONG_UTTERANCES))]
        return dict(kind="transcribe", engine="long", frames=" ".join(map(str, frames)))
    if kind == "stream":
        return dict(kind="stream", batches=rng.randint(2, 6), utterances=rng.randint(1, 8),
                    frames=_log_int(rng, 400, BATCH_FRAMES))
    if kind == "encode":
        return dict(kind="encode", frames=_log_int(rng, 6000, HOUR_FRAMES))
    if kind == "frontend":
        return dict(kind="frontend", utterances=rng.randint(1, 8), samples=_log_int(rng, 8000, 959999))
    if kind == "subsampling":
        return dict(kind="subsampling", utterances=rng.randint(1, 8), frames=_log_int(rng, 100, 6000),
                    precision=rng.choice(["fp16", "fp8"]))
    if kind == "int4_linear":
        return dict(kind="int4_linear", rows=_log_int(rng, 8, 6144), n=rng.choice([1024, 2048, 3072, 4096]), k=WIDTH)
    return dict(kind=kind, rows=_log_int(rng, 50, 45000 if kind == "attention" else 12000))


# ---- what a program sets up once: engines, weights, handles
_KEPT = {}


def _kept(key, make):
    if key not in _KEPT:
        _KEPT[key] = make()
    return _KEPT[key]


def _device():
    return torch.device("cuda:0")


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed))
    return g


def _normal(seed, shape, dtype=torch.float16, std=1.0):
    return (torch.randn(shape, generator=_generator(seed), device=_device()) * std).to(dtype)


def _batch_engine():
    def make():
        eng = pk.pipeline.PipelineEngine(_device(), layers=LAYERS, decoder_layers=1, seed=MODEL_SEED,
                                         max_utterances=BATCH_UTTERANCES, mel_frames=BATCH_FRAMES)
        eng.mel_dev.copy_(_normal(CALIBRATION_SEED, tuple(eng.mel_dev.shape), torch.float32))
        eng.calibrate(BATCH_UTTERANCES)
        return eng
    return _kept("batch", make)


def _engine(name):
    """The engines of other request sizes share the encoder weights of the batch engine."""
    if name == "batch":
        return _batch_engine()
    sizes = dict(long=(LONG_UTTERANCES, LONG_FRAMES, 2), hour=(1, HOUR_FRAMES, 1))[name]

    def make():
        enc = _batch_engine().enc
        eng = pk.pipeline.PipelineEngine(_device(), layers=0, decoder_layers=sizes[2], seed=MODEL_SEED,
                                         max_utterances=sizes[0], mel_frames=sizes[1])
        eng.enc = enc
        return eng
    return _kept(name, make)


def _subsampling(precision):
    return _kept(("subsampling", precision), lambda: pk.subsampling.Subsampling(
        pk.synth.subsampling_weights(MODEL_SEED), _device(), precision=precision))


def _mel_filters():
    """128 triangular filters evenly spaced on the mel scale over 0 .. 8 kHz, 257 FFT bins."""
    mel = np.linspace(0.0, 2595.0 * np.log10(1.0 + 8000.0 / 700.0), BINS + 2)
    hz = 700.0 * (10.0 ** (mel / 2595.0) - 1.0)
    bins = np.arange(257) * (16000.0 / 512.0)
    up = (bins[None, :] - hz[:-2, None]) / (hz[1:-1] - hz[:-2])[:, None]
    down = (hz[2:, None] - bins[None, :]) / (hz[2:] - hz[1:-1])[:, None]
    return np.maximum(0.0, np.minimum(up, down)).astype(np.float32)


def _frontend():
    return _kept("frontend", lambda: pk.frontend.MelFrontend(np.hanning(400).astype(np.float32), _mel_filters(),
                                                             _device()))


def _int4_weights(n, k):
    return _kept(("int4", n, k), lambda: ops.pack_weight_rows(_normal(1000 + n, (n, k), std=0.02), L.PACK_S4_G128))


def _norm_vectors(seed):
    return _normal(seed, (WIDTH,), std=0.1) + 1, _normal(seed + 1, (WIDTH,), std=0.1)


def _ff_weights():
    def make():
        w = dict(w1=ops.pack_weight_rows(_normal(2000, (FF, WIDTH), std=0.02), L.PACK_E4M3),
                 w2=ops.pack_weight_rows(_normal(2001, (WIDTH, FF), std=0.02), L.PACK_S8), ln=_norm_vectors(2002), tau=0.0)
        rows = 768                                   # the tile threshold, chosen once on a calibration input
        s = _ff_state(w, _normal(CALIBRATION_SEED, (rows, WIDTH)))
        stats = torch.zeros((rows // 128, FF // 64), dtype=torch.float32, device=_device())
        _ff_expand(s, stats)
        w["tau"] = pk.encoder.tau_for_zero_fraction(stats.cpu().numpy(), 1.0 - LIVE)
        return w
    return _kept("ff", make)


def _ff_state(w, x):
    rows = x.shape[0]
    new = lambda shape, dtype: torch.empty(shape, dtype=dtype, device=_device())
    return dict(w=w, x=x, q8=new((rows, WIDTH), torch.uint8), hidden=new((rows, FF), torch.int8),
                keep=new(((rows + 127) // 128, FF // 64), torch.uint8), out=new((rows, WIDTH), torch.float16),
                status=torch.zeros(1, dtype=torch.int32, device=_device()))


def _ff_expand(s, stats=None):
    w = s["w"]
    ops.layer_norm(s["x"], *w["ln"], mode=L.LN_E4M3_FIXED, inv_scale=56.0, out=s["q8"])
    ops.gemm(s["q8"], w["w1"][0], kind=L.KIND_E4M3, epilogue=L.EPI_SPARSE_OUT, row_scale=8.0 / 448.0,
             col_scales=w["w1"][1], out=s["hidden"], out_type=L.OUT_S8, out_scale=32.0, tau=w["tau"], keep_out=s["keep"],
             stats_out=stats, status=s["status"])


def _attention_weights():
    def make():
        pos = torch.empty((pk.encoder.POSITION_ROWS_PADDED, WIDTH), dtype=torch.float16, device=_device())
        sinus = torch.from_numpy(pk.encoder.relative_position_encoding()).to(_device())
        ops.gemm(sinus, _normal(3000, (WIDTH, WIDTH), std=0.02), kind=L.KIND_F16, out=pos)
        return dict(qkv=ops.pack_weight_rows(_normal(3001, (3 * WIDTH, WIDTH), std=0.02), L.PACK_S8),
                    out=ops.pack_weight_rows(_normal(3002, (WIDTH, WIDTH), std=0.02), L.PACK_S4_G128),
                    pos=ops.pack_position_heads(pos), u=_normal(3003, (8, 128), std=0.02),
                    v=_normal(3004, (8, 128), std=0.02), ln=_norm_vectors(3005))
    return _kept("attention", make)


# ---- inputs of one case
def _lengths(case):
    return [int(f) for f in case["frames"].split()]


def _host_mel(seed, lengths):
    """Gaussian log-mel frames in pinned host memory, zero behind each utterance's end."""
    mel = _normal(seed, (len(lengths), max(lengths), BINS), torch.float32)
    for u, f in enumerate(lengths):
        mel[u, f:] = 0
    return torch.empty(mel.shape, dtype=torch.float32, pin_memory=True).copy_(mel)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "transcribe":
        lengths = _lengths(case)
        return dict(kind=kind, engine=_engine(case["engine"]), lengths=lengths, mel=_host_mel(seed, lengths))
    if kind == "stream":
        return dict(kind=kind, engine=_engine("batch"), frames=case["frames"], batches=[
            _host_mel(seed * 64 + i, [case["frames"]] * case["utterances"]) for i in range(case["batches"])])
    if kind == "encode":
        return dict(kind=kind, engine=_engine("hour"), rows=pk.subsampling.output_frames(case["frames"]),
                    mel=_host_mel(seed, [case["frames"]])[0])
    if kind == "frontend":
        samples = case["samples"]
        # a slow loudness contour over noise: the dynamic range of the log spectrum is that of speech
        contour = torch.sin(torch.arange(samples, device=_device()) * (2 * math.pi / 16000)) ** 2 * 0.2 + 1e-3
        pcm = _normal(seed, (case["utterances"], samples), torch.float32) * contour
        counts = torch.tensor([samples - 1000 * u for u in range(case["utterances"])], dtype=torch.int32).clamp(min=1)
        return dict(kind=kind, frontend=_frontend(), pcm=pcm, counts=counts.to(_device()))
    if kind == "subsampling":
        mel = _normal(seed, (case["utterances"], case["frames"], BINS), torch.float32)
        stride = pk.pipeline.seg_stride_for(pk.subsampling.output_frames(case["frames"]))
        return dict(kind=kind, stage=_subsampling(case["precision"]), mel=mel, stride=stride,
                    frames=torch.full((case["utterances"],), case["frames"], dtype=torch.int32, device=_device()),
                    out=torch.empty((case["utterances"] * stride, WIDTH), dtype=torch.float16, device=_device()))
    rows = case["rows"]
    if kind == "int4_linear":
        codes, scales = _int4_weights(case["n"], case["k"])
        return dict(kind=kind, x=_normal(seed, (rows, case["k"])), codes=codes, scales=scales,
                    out=torch.empty((rows, case["n"]), dtype=torch.float16, device=_device()))
    if kind == "ff_block":
        return dict(kind=kind, **_ff_state(_ff_weights(), _normal(seed, (rows, WIDTH))))
    stride = pk.pipeline.seg_stride_for(rows)
    x = torch.zeros((stride, WIDTH), dtype=torch.float16, device=_device())
    x[:rows] = _normal(seed, (rows, WIDTH))
    new = lambda n, dtype: torch.empty((stride, n), dtype=dtype, device=_device())
    return dict(kind=kind, w=_attention_weights(), x=x, rows=rows, stride=stride, q8=new(WIDTH, torch.int8),
                scales=torch.empty(stride, dtype=torch.float32, device=_device()), qkv=new(3 * WIDTH, torch.float16),
                att=new(WIDTH, torch.float16), out=new(WIDTH, torch.float16),
                status=torch.zeros(1, dtype=torch.int32, device=_device()))


def _token_table(tokens, frames):
    """Token ids of a batch as one table, -1 behind each utterance's end."""
    rows = pk.subsampling.output_frames(frames) * pk.pipeline.MAX_SYMBOLS_PER_FRAME
    table = np.full((len(tokens), rows), -1, np.int32)
    for u, ids in enumerate(tokens):
        table[u, :len(ids)] = ids
    return table


def run(s):
    kind = s["kind"]
    if kind == "transcribe":
        return _token_table(s["engine"].transcribe_batch(s["mel"], s["lengths"]), max(s["lengths"]))
    if kind == "stream":
        return [_token_table(t, s["frames"]) for t in s["engine"].transcribe_stream(s["batches"])]
    if kind == "encode":
        return s["engine"].encode_chunk(s["mel"], 0, s["rows"])
    if kind == "frontend":
        return s["frontend"].compute(s["pcm"], s["counts"])
    if kind == "subsampling":
        return s["stage"].run(s["mel"], s["stride"], mel_frames=s["frames"], out=s["out"])
    if kind == "int4_linear":
        return ops.gemm(s["x"], s["codes"], kind=L.KIND_F16_W4G128, out=s["out"], b_group_scales=s["scales"])
    w = s["w"]
    if kind == "ff_block":
        _ff_expand(s)
        ops.gemm(s["hidden"], w["w2"][0], kind=L.KIND_S8, row_scale=1.0 / 32.0, col_scales=w["w2"][1], residual=s["x"],
                 alpha=0.5, keep_in=s["keep"], out=s["out"], status=s["status"])
        return s["out"], s["keep"]
    ops.layer_norm(s["x"], *w["ln"], mode=L.LN_S8_ROW, valid_rows=s["rows"], out=s["q8"], scales=s["scales"])
    qkv = s["qkv"]
    ops.gemm(s["q8"], w["qkv"][0], kind=L.KIND_S8, row_scales=s["scales"], col_scales=w["qkv"][1], out=qkv,
             status=s["status"])
    ops.local_attention_tcgen05(qkv[:, :WIDTH], qkv[:, WIDTH:2 * WIDTH], qkv[:, 2 * WIDTH:], w["pos"], w["u"], w["v"],
                                valid_rows=s["rows"], out=s["att"], status=s["status"])
    ops.gemm(s["att"], w["out"][0], kind=L.KIND_F16_W4G128, b_group_scales=w["out"][1], residual=s["x"], out=s["out"],
             status=s["status"])
    return s["out"]


# ---- what a pass cannot do without
def _attention_flops(rows):
    return 6.0 * 257 * WIDTH * rows              # Q.P, Q.K and P.V over a 257-key window


def _block_flops(rows):
    ff = 2 * 2.0 * rows * WIDTH * FF * (1 + LIVE)
    return ff + 2.0 * rows * WIDTH * WIDTH * (3 + 1 + 2 + 1) + _attention_flops(rows)


BLOCK_WEIGHT_BYTES = 4 * WIDTH * FF + WIDTH * WIDTH * (3 + 0.5 + 2 + 1)
SUB_WEIGHT_BYTES = 2.0 * (2 * 256 * 256 + 4096 * WIDTH)


def _subsampling_flops(frames):
    rows = frames / 8.0
    convs = 2.0 * 9 * 256 * (frames / 2 * 64 + frames / 4 * 32 + rows * 16)
    return convs + 2.0 * 256 * 256 * (frames / 4 * 32 + rows * 16) + 2.0 * rows * 4096 * WIDTH


def _encode_flops(frames):
    rows = frames / 8.0
    return _subsampling_flops(frames) + LAYERS * _block_flops(rows) + 2.0 * rows * WIDTH * HIDDEN


def _decode(frames, layers):
    """Flops and weight bytes: a few tokens per encoder frame with random weights (at most ten)."""
    lstm = (2 * layers - 1) * 4 * HIDDEN * HIDDEN          # layer 0's input half is a table row
    per_token = 2.0 * (lstm + HIDDEN * HIDDEN + TOKEN_ROWS * HIDDEN)
    return frames / 8.0 * 4 * per_token, 2.0 * (lstm + HIDDEN * HIDDEN + 2 * TOKEN_ROWS * HIDDEN)


def work(case):
    kind = case["kind"]
    if kind in ("transcribe", "stream"):
        lengths = _lengths(case) if kind == "transcribe" else [case["frames"]] * (case["utterances"] * case["batches"])
        frames = sum(lengths)
        flops, weights = _decode(frames, 2 if case.get("engine") == "long" else 1)
        bytes_ = weights + LAYERS * BLOCK_WEIGHT_BYTES + SUB_WEIGHT_BYTES + 4.0 * BINS * frames + 4 * frames / 8.0 * 4
        return dict(bytes=bytes_, flops=flops + _encode_flops(frames))
    if kind == "encode":
        frames = case["frames"]
        return dict(bytes=LAYERS * BLOCK_WEIGHT_BYTES + SUB_WEIGHT_BYTES + 4.0 * BINS * frames + 2.0 * HIDDEN * frames / 8,
                    flops=_encode_flops(frames))
    if kind == "frontend":
        frames = case["utterances"] * (case["samples"] / HOP)
        return dict(bytes=case["utterances"] * case["samples"] * 4.0 + frames * BINS * 4.0,
                    flops=frames * (5 * 512 * 9 + 3 * 512 + 6 * BINS))
    if kind == "subsampling":
        frames = case["utterances"] * case["frames"]
        return dict(bytes=frames * BINS * 4.0 + frames / 8.0 * WIDTH * 2 + SUB_WEIGHT_BYTES / (2 if case["precision"] == "fp8" else 1),
                    flops=_subsampling_flops(frames))
    rows = case["rows"]
    if kind == "int4_linear":
        n, k = case["n"], case["k"]
        return dict(bytes=2.0 * rows * (n + k) + n * k * (0.5 + 2 / 128), flops=2.0 * rows * n * k)
    if kind == "ff_block":
        return dict(bytes=2.0 * rows * WIDTH * 2 + 2.0 * WIDTH * FF, flops=2.0 * rows * WIDTH * FF * (1 + LIVE))
    return dict(bytes=2.0 * rows * WIDTH * 2 + WIDTH * WIDTH * 3.5 + 2.0 * 257 * WIDTH,
                flops=8.0 * rows * WIDTH * WIDTH + _attention_flops(rows))


def tolerance(case):
    kind = case["kind"]
    if kind in ("transcribe", "stream"):
        return "exact"                           # token ids
    if kind == "encode":
        # 24 blocks with E4M3 / INT8 quantisation points and tile thresholds in each: a last-bit
        # difference turns into 6 % steps of single activations; the reference's own gate is 3e-2
        return dict(rel=3e-2, max=0.9)
    if kind == "frontend":
        return dict(rel=1e-4, max=1e-2)          # fp32 FFT; the logarithm of near-silent bins amplifies its rounding
    if kind == "subsampling":
        return dict(rel=1e-2 if case["precision"] == "fp8" else 2e-3)
    if kind == "int4_linear":
        return dict(rel=1e-3)                    # fp16 result of an fp32 sum
    if kind == "ff_block":
        return dict(rel=2e-3, max=0.1, differ=0.01)   # fp16 result; INT8 codes of the hidden activations; tile flags
    return dict(rel=2e-3, max=0.1)               # fp16 result; INT8 codes of the normalised rows
