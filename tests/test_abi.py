"""The C-ABI library loads and exports every symbol include/pk100.h declares
(no compute calls here: this runs without a GPU)."""
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def declared_symbols():
    text = (ROOT / "include" / "pk100.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(?:int|long long|void|const char\s*\*)\s*(pk100_\w+)\s*\(", text)))


def test_header_declares_entry_points():
    names = declared_symbols()
    assert "pk100_gemm" in names and "pk100_layer_norm" in names and len(names) >= 10


def test_library_exports_every_declared_symbol(pk):
    for name in declared_symbols():
        assert hasattr(pk.lib.lib, name), f"libpk100.so does not export {name}"


def test_binding_table_matches_header(pk):
    void_setters = ["pk100_set_gemm_cta_pairs", "pk100_set_gemm_cta_cap", "pk100_set_dependent_launch", "pk100_tensor_map_cache_stats"]
    assert sorted(list(pk.lib.SIGNATURES) + void_setters) == declared_symbols()


def test_argument_errors_need_no_gpu(pk):
    L = pk.lib
    # null pointers / bad shapes are rejected on the host before any launch
    assert L.lib.pk100_layer_norm(None, None, None, None, None, None, 0, 0.0, 8, 8, 8, None, 1e-5) == L.ERR_NULL
    assert L.lib.pk100_quantize_fp8_fixed(None, None, None, 16, 1.0) == L.ERR_NULL
    args = L.GemmArgs()
    assert L.lib.pk100_gemm(None, args) == L.ERR_NULL


def test_packed_entry_points_check_their_arguments_on_the_host(pk):
    """Pointers here are numbers that no launch ever sees."""
    L, enc, sub = pk.lib, pk.encoder, pk.subsampling
    layers, ws, out = (enc.LayerWeights * 1)(), enc.Workspace(), enc.vp()
    def run(n_layers=1, a=4096, b=8192, rows=256, tiles=256, work=ws):
        return L.lib.pk100_run_layers_packed(None, layers, n_layers, a, b, work, rows, tiles, out)
    assert run(a=None) == run(b=None) == run(tiles=None) == run(work=None) == L.ERR_NULL
    assert run(rows=200) == run(rows=-128) == run(n_layers=-1) == L.ERR_SHAPE
    assert run(tiles=260) == run(a=4104) == run(b=8200) == L.ERR_ALIGN
    assert run() == L.ERR_NULL                                  # an empty workspace
    w, q = sub.SubsamplingWeightsC(), sub.SubsamplingFp8C()
    def rows_of(mel_stride=100, utterances=2, frames=100, seg=128, base=None, rows=256, fp8=None, weights=w, mel=256):
        return L.lib.pk100_run_subsampling_rows(None, weights, fp8, mel, mel_stride, utterances, frames, None, 256, 256, seg, base,
                                                rows, None)
    assert rows_of(mel_stride=99) == rows_of(utterances=-1) == rows_of(rows=255) == L.ERR_SHAPE
    assert rows_of(base=256, rows=0) == rows_of(base=256, rows=200) == rows_of(base=256, rows=384) == L.ERR_SHAPE
    assert rows_of(fp8=q) == rows_of(mel=None) == rows_of() == L.ERR_NULL      # empty weights
