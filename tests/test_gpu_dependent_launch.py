"""Products and attention of the per-block chain behind a kernel that runs longer than their own waits may."""
import ctypes as C

import pytest
import torch

from tests.util import dev16
from tests.test_gpu_attention import _case

pytestmark = pytest.mark.gpu


class Rows(C.Structure):
    """Mirror of `pk100_rows` (csrc/pk100_internal.h)."""
    _fields_ = [("tiles", C.c_void_p), ("seg_stride", C.c_int), ("valid_rows", C.c_int), ("seg_valid", C.c_void_p)]


def test_waits_begin_behind_the_kernel_in_front(pk, cuda):
    """The sequencers' launches (weights and geometry settled) request weights while the kernel in front still runs.
    That kernel may take any time; only then do the bounded waits of 2 s begin.  Two products whose K is longer
    than their operand ring, and the attention, behind a product on one CTA that takes more than that."""
    L = pk.lib
    chained = L.lib["_Z18pk100_gemm_chainedPvPK15pk100_gemm_argsb"]
    chained.argtypes, chained.restype = [C.c_void_p, C.POINTER(L.GemmArgs), C.c_bool], C.c_int
    attend = L.lib["_Z26pk100_local_attention_rowsPvPKviS1_iS1_iS1_S1_S1_S_iiRK10pk100_rowsbPi"]
    vp, i = C.c_void_p, C.c_int
    attend.argtypes, attend.restype = [vp, vp, i, vp, i, vp, i, vp, vp, vp, vp, i, i, C.POINTER(Rows), C.c_bool, vp], i
    g = torch.Generator().manual_seed(3)
    x = torch.randn((128, 4096), generator=g).half().to(cuda)
    w = (torch.randn((1024, 4096), generator=g) * 0.05).half().to(cuda)
    codes, scales = pk.ops.pack_weight_rows(w, L.PACK_S4_G128)
    q, k, v, pos, u, bv = (dev16(t) for t in _case(7, 128))
    forms = [dict(kind=L.KIND_F16, b=w), dict(kind=L.KIND_F16_W4G128, b=codes, b_group_scales=scales)]
    want = [torch.empty((128, 1024), dtype=torch.float16, device=cuda) for _ in range(3)]
    for form, out in zip(forms, want):
        pk.ops.gemm(x, form["b"], kind=form["kind"], out=out, n=1024, b_group_scales=form.get("b_group_scales"))
    pk.ops.local_attention_tcgen05(q, k, v, pos, u, bv, out=want[2])
    got = [torch.zeros_like(t) for t in want]
    status = torch.zeros(4, dtype=torch.int32, device=cuda)
    front = [torch.zeros(s, dtype=torch.float16, device=cuda) for s in ((8192, 49152), (65536, 49152), (8192, 65536))]
    stream = torch.cuda.current_stream()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    start.record()
    pk.ops.gemm(front[0], front[1], kind=L.KIND_F16, out=front[2], max_ctas=1, status=status[3:])
    for n, (form, out) in enumerate(zip(forms, got)):
        group = form.get("b_group_scales")
        args = L.GemmArgs(kind=form["kind"], m=128, n=1024, k=4096, a=x.data_ptr(), lda=4096, b=form["b"].data_ptr(),
                          ldb=4096, row_scale=1.0, alpha=1.0, out=out.data_ptr(), ld_out=1024, out_scale=1.0,
                          status=status[n:].data_ptr(), b_group_scales=None if group is None else group.data_ptr())
        assert chained(stream.cuda_stream, C.byref(args), True) == 0
    rows = Rows(None, 128, 128, None)
    assert attend(stream.cuda_stream, q.data_ptr(), 1024, k.data_ptr(), 1024, v.data_ptr(), 1024, pos.data_ptr(), u.data_ptr(),
                  bv.data_ptr(), got[2].data_ptr(), 1024, 128, C.byref(rows), True, status[2:].data_ptr()) == 0
    end.record()
    torch.cuda.synchronize()
    assert start.elapsed_time(end) > 2200.0
    assert status.tolist() == [0, 0, 0, 0]
    for a, b in zip(got, want):
        assert torch.equal(a, b) and bool(a.any())
