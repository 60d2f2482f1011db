"""Request lengths on the host side of the pipeline engine (no GPU: an engine's length buffers on the CPU)."""
import pytest
import torch


def _engine(pk, utterances=8, mel_frames=6000):
    cls = pk.pipeline.PipelineEngine
    eng = cls.__new__(cls)
    eng.max_utterances, eng.mel_frames, eng.encode_groups = utterances, mel_frames, 1
    eng.frames_out = pk.subsampling.output_frames(mel_frames)
    eng.seg_stride = pk.pipeline.seg_stride_for(eng.frames_out)
    ints = lambda n, v=0: torch.full((n,), v, dtype=torch.int32)
    eng.mel_frames_dev, eng.out_frames_dev = ints(utterances, mel_frames), ints(utterances, eng.frames_out)
    eng.out_frames_host = eng.out_frames_dev.clone()
    eng.longest_out_frames = eng.frames_out
    eng.place = ints(2 * (utterances + utterances * eng.seg_stride // 128))
    eng._lengths = (mel_frames,) * utterances
    return eng


def _state(eng):
    return [eng._lengths, eng.longest_out_frames] + [t.tolist() for t in (eng.mel_frames_dev, eng.out_frames_dev,
                                                                          eng.out_frames_host, eng.place)]


def test_a_refused_request_leaves_the_engine_as_it_was(pk):
    eng, fresh = _engine(pk), _engine(pk)
    for e in (eng, fresh):
        e.set_lengths([700, 6000, 1])
    before = _state(eng)
    refused = [lambda: eng.set_lengths([6000] * 9), lambda: eng.set_lengths([400, 6001]),
               lambda: eng.transcribe_batch(torch.zeros(9, 6000, 128)),
               lambda: eng.transcribe_batch(torch.zeros(2, 6000, 128), [6000] * 9),
               lambda: eng.transcribe_batch(torch.zeros(2, 6000, 128), [6001, 1])]
    for call in refused:
        for _ in range(2):
            with pytest.raises(ValueError):
                call()
            assert _state(eng) == before
    for lengths in ([5999] * 8, [400], [400, 5000, 0, 6000, 1, 2049, 1025, 1024]):
        for e in (eng, fresh):
            e.set_lengths(lengths)
        assert _state(eng) == _state(fresh) and eng._lengths[:len(lengths)] == tuple(lengths)


@pytest.mark.parametrize("negative", [-1, -8, -2000, -20000])
def test_a_negative_length_is_an_empty_utterance(pk, negative):
    eng, fresh = _engine(pk), _engine(pk)
    eng.set_lengths([3000, negative, 6000, 40])
    fresh.set_lengths([3000, 0, 6000, 40])
    assert _state(eng) == _state(fresh)
    assert eng._geometry(eng._lengths[:4]) == fresh._geometry(fresh._lengths[:4])
