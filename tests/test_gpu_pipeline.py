"""GPU parity: the whole path (subsampling -> blocks -> projection -> TDT decode) through the
public pipeline API vs the CPU oracle, on a reduced model (2 blocks, short utterances)."""
import numpy as np
import pytest
import torch

from oracle import decoder as D, ops as O, pipeline as P
from tests.util import nrmse

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine(pk, cuda):
    eng = pk.pipeline.PipelineEngine(cuda, layers=2, decoder_layers=2, seed=9, max_utterances=3,
                                     mel_frames=1000, randomize_norms=True)
    return eng


def _weights(pk, eng):
    sub_w = pk.synth.subsampling_weights(9)
    layers = [O.prepare_layer(pk.synth.layer_weights(9, l, randomize_norms=True)) for l in range(2)]
    dec_w = pk.synth.decoder_weights(9, 2)
    return sub_w, layers, dec_w


def test_transcribe_batch_matches_oracle(pk, cuda, engine):
    eng = engine
    frames = [1000, 1000, 1000]
    mels = np.stack([pk.synth.mel_input(100 + u, 1000) for u in range(3)])
    mel_host = torch.from_numpy(mels).pin_memory()
    # tile thresholds stay 0 here: the free-running stack is compared as a continuous
    # operator (per-block parity WITH thresholds is covered in test_gpu_encoder.py)
    tokens = eng.transcribe_batch(mel_host)
    assert eng.status() == 0
    sub_w, layers, dec_w = _weights(pk, eng)
    taus = [(eng.enc.layers[l].ff1.tau, eng.enc.layers[l].ff2.tau) for l in range(2)]
    for u in range(3):
        want_tokens, want_enc, amb = P.transcribe(mels[u], sub_w, layers, taus, dec_w)
        # encoder output of the free-running 2-block stack: reference's stack gate
        blk = slice(u * eng.seg_stride, u * eng.seg_stride + eng.frames_out)
        got_proj = eng.enc_proj[blk].float().cpu().numpy()
        want_proj = P.project(want_enc, dec_w)
        assert nrmse(got_proj, want_proj) <= 3e-2
        # token ids: exact on the SAME encoder projection (the GPU's), up to the first
        # decision inside fp32 summation noise
        same_tokens, _, amb2 = D.tdt_greedy(got_proj, dec_w, eng.frames_out)
        n = len(same_tokens) if amb2 is None else amb2
        assert n > 10
        assert np.array_equal(tokens[u][:n], same_tokens[:n])
        if amb2 is None:
            assert len(tokens[u]) == len(same_tokens)


def test_resident_path_is_deterministic_and_ragged_lengths(pk, cuda, engine):
    eng = engine
    frames = [1000, 617, 40]
    mels = np.zeros((3, 1000, 128), np.float32)
    for u, f in enumerate(frames):
        mels[u, :f] = pk.synth.mel_input(200 + u, f)
    mel_host = torch.from_numpy(mels).pin_memory()
    eng.set_lengths(frames)
    eng.mel_dev.copy_(mel_host)
    eng.calibrate(3)                       # 70 % zero tiles from here on
    assert all(l.ff1.tau > 0 and l.ff2.tau > 0 for l in eng.enc.layers)
    a = eng.transcribe_batch(mel_host, frames)
    b = eng.transcribe_batch(mel_host, frames)
    assert all(np.array_equal(x, y) for x, y in zip(a, b))
    # a shorter utterance in a batch decodes like the same utterance alone
    solo = eng.transcribe_batch(torch.from_numpy(np.stack([mels[1]] * 3)).pin_memory(), [617, 617, 617])
    assert np.array_equal(solo[0], a[1])
    # a request without lengths means "all frames": nothing is inherited from the request before
    full = eng.transcribe_batch(mel_host)
    assert tuple(eng.out_frames_host.tolist()) == (eng.frames_out,) * 3
    again = eng.transcribe_batch(mel_host, [1000, 1000, 1000])
    assert all(np.array_equal(x, y) for x, y in zip(full, again))
    # and the schedule changes no token: one group for everything, or two encode groups whose
    # decodes run under the next group's encode (the engine above: one encode pass, a decoder
    # cluster per utterance)
    assert eng.encode_groups == 1 and eng.decode_groups == 3
    for enc_groups, dec_groups in ((1, 1), (2, 2), (2, 3)):
        other = pk.pipeline.PipelineEngine(cuda, layers=2, decoder_layers=2, seed=9, max_utterances=3, mel_frames=1000,
                                           randomize_norms=True, encode_groups=enc_groups, decode_groups=dec_groups)
        for l, lw in enumerate(eng.enc.layers):
            other.enc.set_tau(l, lw.ff1.tau, lw.ff2.tau)
        got = other.transcribe_batch(mel_host, frames)
        assert other.status() == 0 and all(np.array_equal(x, y) for x, y in zip(got, a))
        assert len(other.last_groups) == dec_groups and len(other.last_encode_groups) == enc_groups


def test_streamed_batches_return_what_single_requests_return(pk, cuda, engine):
    """transcribe_stream (batch i + 1 encoded beside the decode of batch i, two alternating sets
    of request buffers) yields, in order, exactly the tokens of one transcribe_batch per batch."""
    eng = engine
    rng = np.random.default_rng(5)
    batches, want = [], []
    for i in range(5):
        n = 1 + i % 3
        frames = [int(f) for f in rng.integers(40, 1001, size=n)]
        mels = np.zeros((n, 1000, 128), np.float32)
        for u, f in enumerate(frames):
            mels[u, :f] = pk.synth.mel_input(300 + 10 * i + u, f)
        batches.append((torch.from_numpy(mels).pin_memory(), frames))
    for mel, frames in batches:
        want.append(eng.transcribe_batch(mel, frames))
    for depth, groups in ((2, 2), (3, 1)):
        got = list(eng.transcribe_stream(iter(batches), decode_groups=groups, depth=depth))
        assert len(got) == len(want) and eng.status() == 0
        for g, w in zip(got, want):
            assert len(g) == len(w) and all(np.array_equal(x, y) for x, y in zip(g, w))
    assert any(len(t) > 0 for batch in got for t in batch)


@pytest.mark.parametrize("frames", [[3100, 1024, 1025], [8, 3100, 2049], [40, 40, 40], [0, 2100, 1], [3100, 3100, 1]])
def test_rows_fitted_to_the_request_give_the_same_bits(pk, cuda, frames):
    """Rows laid out for the request's lengths (a smaller distance between utterances, or a packed batch without
    padding tiles; utterances that end on and just behind a tile edge) against the engine's full capacity."""
    eng = pk.pipeline.PipelineEngine(cuda, layers=2, decoder_layers=1, seed=9, max_utterances=3, mel_frames=3100)
    for l in range(2):
        eng.enc.set_tau(l, 0.4, 0.4)
    eng.mel_dev.normal_(generator=torch.Generator(device=cuda).manual_seed(3))
    eng.set_lengths(frames)
    got = []
    for fitted in (False, True):
        eng.enc_proj.fill_(float("nan"))
        eng.run_resident(3, fitted=fitted)
        torch.cuda.synchronize()
        seg = eng._geometry(frames)[1] if fitted else eng.seg_stride
        rows = [eng.enc_proj[u * seg:u * seg + pk.subsampling.output_frames(f)].cpu() for u, f in enumerate(frames)]
        got.append((rows, eng.tokens.cpu().clone(), eng.counts.cpu().clone(), seg))
    assert eng.status() == 0
    for a, b in zip(got[0][0], got[1][0]):
        assert torch.isfinite(b).all() and torch.equal(a, b)
    assert torch.equal(got[0][2], got[1][2])
    for u in range(3):
        assert torch.equal(got[0][1][u, :got[0][2][u]], got[1][1][u, :got[0][2][u]])
    packed = eng._geometry(frames)[2]
    assert (packed is None) == (len({pk.pipeline.seg_stride_for(pk.subsampling.output_frames(f)) for f in frames}) == 1)


def test_a_refused_request_changes_no_later_result(pk, cuda):
    """Requests that the engine is too small for are refused before anything is queued; ragged requests after
    them (sent twice: the second finds its lengths recorded) decode like those of an engine that saw none."""
    engines = [pk.pipeline.PipelineEngine(cuda, layers=1, decoder_layers=1, seed=9, max_utterances=3, mel_frames=3100)
               for _ in range(2)]
    mel = torch.randn((4, 3100, 128), generator=torch.Generator().manual_seed(7)).pin_memory()
    frames = [3100, 1025, 40]
    want = engines[0].transcribe_batch(mel[:3], frames)
    assert engines[1]._geometry(frames)[2] is not None and any(len(t) > 0 for t in want)
    for lengths in ([3100] * 4, frames + [1]):
        with pytest.raises(ValueError):
            engines[1].transcribe_batch(mel, lengths)
        for _ in range(2):
            got = engines[1].transcribe_batch(mel[:3], frames)
            assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("precision", ["fp16", "fp8"])
def test_requests_allocate_no_device_memory_of_their_own(pk, cuda, precision):
    """The stages' workspaces hold the engine's capacity from the start: a request longer than all before it,
    or of more utterances, allocates nothing, nor does a chunk of a long utterance."""
    eng = pk.pipeline.PipelineEngine(cuda, layers=1, decoder_layers=1, seed=9, max_utterances=3, mel_frames=1200,
                                     subsampling_precision=precision)
    mel = torch.randn((3, 1200, 128), generator=torch.Generator().manual_seed(7)).pin_memory()
    held = eng.sub._ws.data_ptr(), eng.sub._ws.numel()
    for n, frames in ((1, 40), (1, 900), (2, 400), (3, 1200)):
        eng.transcribe_batch(mel[:n, :frames])
        assert (eng.sub._ws.data_ptr(), eng.sub._ws.numel()) == held
    eng.encode_chunk(mel[0, :640], 2, 70)
    assert (eng.sub._ws.data_ptr(), eng.sub._ws.numel()) == held


class _Unsized:
    """Iterable whose length is not known, like a loader over a stream."""

    def __init__(self, items):
        self.items = items

    def __iter__(self):
        return iter(self.items)

    def __len__(self):
        raise TypeError("no length")


def test_a_stream_of_unknown_length_is_accepted(pk, cuda, engine):
    mel = torch.randn((2, 400, 128), generator=torch.Generator().manual_seed(2)).pin_memory()
    want = engine.transcribe_batch(mel)
    for got in engine.transcribe_stream(_Unsized([mel, mel]), depth=2):
        assert all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("decode_groups,depth", [(1, 2), (2, 2), (1, 4)])
def test_last_batch_of_a_known_number_takes_the_free_clusters(pk, cuda, engine, decode_groups, depth):
    """A list knows its last batch, an iterator does not: the last batch is decoded on the clusters that the
    batches in flight do not hold, with the same tokens, more batches than buffer sets and ragged lengths."""
    eng, rng = engine, np.random.default_rng(6)
    batches = []
    for i, n in enumerate((3, 1, 2, 3, 2, 3)):
        frames = [int(f) for f in rng.integers(40, 1001, size=n)]
        mels = np.zeros((n, 1000, 128), np.float32)
        for u, f in enumerate(frames):
            mels[u, :f] = pk.synth.mel_input(400 + 10 * i + u, f)
        batches.append((torch.from_numpy(mels).pin_memory(), frames))
    want = [eng.transcribe_batch(mel, frames) for mel, frames in batches]
    assert eng.decode_groups == 3 and any(len(t) > 0 for t in want[-1])
    groups = []
    for source in (batches, iter(batches)):
        got = list(eng.transcribe_stream(source, decode_groups=decode_groups, depth=depth))
        assert eng.status() == 0 and len(got) == len(want)
        for g, w in zip(got, want):
            assert len(g) == len(w) and all(np.array_equal(x, y) for x, y in zip(g, w))
        groups.append(len(eng.last_groups))
    busy = (depth - 1) * decode_groups if depth == 2 else 3          # (at depth 4: batches of at least one cluster each)
    assert groups[1] == decode_groups and groups[0] == max(decode_groups, 3 - busy)
