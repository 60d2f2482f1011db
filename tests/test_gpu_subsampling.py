"""GPU parity: batched convolution subsampling vs the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import ops as O
from tests.util import dev, host, nrmse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp16", "fp8"])
@pytest.mark.parametrize("frames_list", [[400, 400], [203, 77, 8, 1]])
def test_subsampling_matches_oracle(pk, cuda, frames_list, precision):
    w = pk.synth.subsampling_weights(2)
    sub = pk.subsampling.Subsampling(w, cuda, precision=precision)
    # the E4M3 variant (the reference's path from 1024 output frames on) agrees with its oracle to the
    # tolerance of a quantised stage: a byte that rounds the other way is a 6 % step of that activation
    max_abs, max_nrmse = (2e-2, 2e-3) if precision == "fp16" else (4e-2, 1e-2)
    cap = max(frames_list)
    mels = [pk.synth.mel_input(30 + i, f) for i, f in enumerate(frames_list)]
    batch = np.zeros((len(mels), cap, 128), np.float32)
    for i, m in enumerate(mels):
        batch[i, :m.shape[0]] = m
    seg_stride = (pk.subsampling.output_frames(cap) + 127) // 128 * 128
    mf = torch.tensor(frames_list, dtype=torch.int32, device=cuda)
    out = host(sub.run(dev(batch), seg_stride, mel_frames=mf))
    torch.cuda.synchronize()
    assert int(sub.status.item()) == 0
    for i, m in enumerate(mels):
        want = O.subsampling(m, w, fp8=precision == "fp8")
        got = out[i * seg_stride:i * seg_stride + want.shape[0]]
        assert want.shape[0] == pk.subsampling.output_frames(frames_list[i])
        # reference gate for this stage: max abs <= 2.0 and nRMSE <= 0.002
        # (src/cuda/subsampling.rs:375); ours is far inside it
        assert np.max(np.abs(got - want)) <= max_abs
        assert nrmse(got, want) <= max_nrmse


@pytest.mark.parametrize("precision", ["fp16", "fp8"])
@pytest.mark.parametrize("frames_list", [[2501, 97, 2], [6000] * 3])
def test_frames_per_cta_do_not_change_a_bit(pk, cuda, frames_list, precision):
    """The first kernel walks 1 to 8 output frames per CTA depending on the batch: an utterance in a
    batch (7 and 8 frames per CTA here) gives the bits of the utterance alone (1 to 6)."""
    sub = pk.subsampling.Subsampling(pk.synth.subsampling_weights(2), cuda, precision=precision)
    cap = max(frames_list)
    batch = torch.zeros((len(frames_list), cap, 128), dtype=torch.float32, device=cuda)
    for i, f in enumerate(frames_list):
        batch[i, :f] = dev(pk.synth.mel_input(60 + i, f))
    stride = pk.pipeline.seg_stride_for(pk.subsampling.output_frames(cap))
    together = sub.run(batch, stride, mel_frames=torch.tensor(frames_list, dtype=torch.int32, device=cuda)).clone()
    for i, f in enumerate(frames_list):
        alone = sub.run(batch[i:i + 1, :f].contiguous(), stride)
        rows = pk.subsampling.output_frames(f)
        assert torch.equal(alone[:rows], together[i * stride:i * stride + rows]) and bool(alone[:rows].any())


@pytest.mark.parametrize("precision", ["fp16", "fp8"])
def test_nan_mel_values_end_at_the_first_relu(pk, cuda, precision):
    """max(NaN, 0) = 0: a NaN mel value removes the first-layer features it reaches and nothing else."""
    w = pk.synth.subsampling_weights(2)
    sub = pk.subsampling.Subsampling(w, cuda, precision=precision)
    mel = pk.synth.mel_input(8, 203)
    for f, t in ((0, 0), (0, 127), (57, 64), (58, 33), (202, 5)):
        mel[f, t] = np.nan
    mel[120] = np.nan
    got = host(sub.run(dev(mel[None]), 128))[:26]
    want = O.subsampling(mel, w, fp8=precision == "fp8")
    assert np.isfinite(got).all() and np.isfinite(want).all()
    max_abs, max_nrmse = (2e-2, 2e-3) if precision == "fp16" else (4e-2, 1e-2)      # as without NaN
    assert np.max(np.abs(got - want)) <= max_abs and nrmse(got, want) <= max_nrmse


@pytest.mark.parametrize("frames,rows", [(1, (0, 2)), (2, (0,))])
def test_taps_outside_the_utterance_are_not_multiplied(pk, cuda, frames, rows):
    """Taps of the first convolution that lie in front of or behind every frame: infinite weights there change
    nothing (multiplied with a zero they would give NaN)."""
    w = pk.synth.subsampling_weights(2)
    mel = dev(pk.synth.mel_input(9, frames)[None])
    want = pk.subsampling.Subsampling(w, cuda).run(mel, 128).clone()
    taps = w["conv0_w"] = w["conv0_w"].copy()
    taps.reshape(256, 3, 3)[:, rows, :] = np.inf
    got = pk.subsampling.Subsampling(w, cuda).run(mel, 128)
    assert torch.equal(got, want) and bool(got[:1].any())


@pytest.mark.parametrize("precision", ["fp16", "fp8"])
@pytest.mark.parametrize("frames_list", [[3100, 1024, 1025], [8, 3100, 0, 2049], [1, 1, 1024]])
def test_packed_rows_are_the_rows_of_the_uniform_layout(pk, cuda, precision, frames_list):
    """row_base: every utterance in whole 128-row tiles, at its own place, padding rows included; utterances at
    the distance of a larger buffer."""
    sub = pk.subsampling.Subsampling(pk.synth.subsampling_weights(2), cuda, precision=precision)
    n, cap, frames = len(frames_list), 3300, max(frames_list)
    mel = torch.randn((n, cap, 128), generator=torch.Generator(device=cuda).manual_seed(n), device=cuda)
    mf = torch.tensor(frames_list, dtype=torch.int32, device=cuda)
    seg = pk.pipeline.seg_stride_for(pk.subsampling.output_frames(frames))
    want = sub.run(mel[:, :frames].contiguous(), seg, mel_frames=mf).clone()
    rows = [pk.pipeline.seg_stride_for(pk.subsampling.output_frames(f)) for f in frames_list]
    base = np.concatenate([[0], np.cumsum(rows)[:-1]])
    out = torch.full((sum(rows), 1024), float("nan"), dtype=torch.float16, device=cuda)
    sub.run_rows(mel, frames, seg, mf, out, row_base=torch.tensor(base, dtype=torch.int32, device=cuda), rows=sum(rows))
    assert int(sub.status.item()) == 0
    for u in range(n):
        assert torch.equal(out[base[u]:base[u] + rows[u]], want[u * seg:u * seg + rows[u]])
    uniform = sub.run_rows(mel, frames, seg, mf, torch.empty_like(want))
    assert torch.equal(uniform, want) and bool(want.any())


def _first_stage(sub, frames, stride):
    """What the first kernel left in the workspace after a run of one utterance: fp16 rows, or E4M3 codes and scales."""
    def up256(n):
        return (n + 255) // 256 * 256

    f2 = ((frames + 1) // 2 + 1) // 2
    f3 = (f2 + 1) // 2
    rows = f2 * 32
    if sub.q is None:
        return sub._ws[:rows * 512].view(torch.float16).view(rows, 256).clone()
    at = 2 * up256(rows * 512) + 2 * up256(f3 * 16 * 512) + up256(stride * 8192) + 256
    codes = sub._ws[at:at + rows * 256].view(rows, 256).clone()
    at += up256(rows * 256)
    return codes, sub._ws[at:at + rows * 4].view(torch.float32).clone()


@pytest.mark.parametrize("frames", [1, 2, 3, 5, 8, 129, 1030, 4001])
def test_e4m3_variant_codes_the_rows_of_the_fp16_variant(pk, cuda, frames):
    """Both variants take the same fp32 sums in the same order and round them to fp16; the E4M3 variant then codes the
    rows: codes and scales are those of the quantiser on the fp16 variant's rows, bit for bit."""
    w = pk.synth.subsampling_weights(3)
    mel = dev(pk.synth.mel_input(90 + frames, frames)[None] * 3.0)
    stride = pk.pipeline.seg_stride_for(pk.subsampling.output_frames(frames))
    stages = []
    for precision in ("fp16", "fp8"):
        sub = pk.subsampling.Subsampling(w, cuda, precision=precision)
        sub.run(mel, stride)
        torch.cuda.synchronize()
        assert int(sub.status.item()) == 0
        stages.append(_first_stage(sub, frames, stride))
    codes, scales = pk.ops.pack_weight_rows(stages[0], pk.lib.PACK_E4M3)
    assert bool(stages[0].any()) and bool(torch.isfinite(stages[0]).all())
    assert torch.equal(stages[1][0], codes.view(torch.uint8)) and torch.equal(stages[1][1], scales)


@pytest.mark.parametrize("frames", [1, 2, 3, 5, 8, 129, 1030])
def test_e4m3_variant_at_the_edges(pk, cuda, frames):
    """The E4M3 variant against the oracle at the shortest utterances and around the ends of a CTA's range, with finite
    taps and with taps of -inf: where such a tap lies inside, the sum ends at the ReLU; outside it is not
    multiplied and the sum is that of the other taps."""
    w = pk.synth.subsampling_weights(3)
    mel = pk.synth.mel_input(90 + frames, frames) * 3.0
    rows = pk.subsampling.output_frames(frames)
    stride = pk.pipeline.seg_stride_for(rows)
    odd = {k: v.copy() for k, v in w.items()}
    odd["conv0_w"][5, 0] = -np.inf                   # frame tap 0, feature tap 0: outside at frame 0 and at feature 0
    odd["conv0_w"][9, 7] = -np.inf                   # frame tap 2: outside at an odd utterance's last frame
    odd["dw1_w"][[5, 9]] = 4.0                       # their features weigh in every row
    for weights, x in ((w, mel), (odd, np.abs(mel) + 1.0)):
        sub = pk.subsampling.Subsampling(weights, cuda, precision="fp8")
        got = host(sub.run(dev(x[None]), stride))[:rows]
        assert int(sub.status.item()) == 0
        want = O.subsampling(x, weights, fp8=True)
        assert np.isfinite(got).all() and np.isfinite(want).all()
        assert nrmse(got, want) <= 1e-2              # as in test_subsampling_matches_oracle
