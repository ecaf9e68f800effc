"""What the Python layer hands on to the library: missing tensors are the library's error. Needs a GPU."""
import pytest
import torch

from flashrt_b200 import moe

pytestmark = pytest.mark.gpu
Q2_0 = moe.Q2_0_TYPE


def test_missing_tensors_are_refused_by_the_library():
    T, K, n, ff = 2, 2, 128, 128
    z = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    x, gate, wts = torch.zeros(T, n, device="cuda"), torch.zeros(T, device="cuda"), torch.zeros(T, K, device="cuda")
    ids = torch.zeros(T, K, dtype=torch.int32, device="cuda")
    ptr, hit_n, yh = torch.zeros(T, K, dtype=torch.int64, device="cuda"), torch.zeros(T, dtype=torch.int32, device="cuda"), torch.zeros(T, K, n, device="cuda")
    layer = (z.data_ptr(), moe.expert_stride(n, ff), 4, None, n, ff)
    calls = [
        lambda: moe.moe_layer(None, *layer[1:], x, torch.zeros(T, 4, device="cuda"), gate, K),
        lambda: moe.moe_layer(*layer, x, None, gate, K),
        lambda: moe.moe_decode(*layer, x, ids, None, gate),
        lambda: moe.moe_decode(*layer, None, ids, wts, gate, out=x, ws=moe.workspace(moe.moe_decode_workspace_bytes(T, K, n, ff))),
        lambda: moe.moe_decode_static(*layer, x, ids, None, gate, x),
        lambda: moe.moe_decode_static(*layer, x, ids, wts, gate, None),
        lambda: moe.moe_hits(None, hit_n, K, x, n, ff, yh, T=T),
        lambda: moe.moe_hits(ptr, None, K, x, n, ff, yh, T=T),
        lambda: moe.moe_hits(ptr, hit_n, K, x, n, ff, None, T=T),
        lambda: moe.moe_combine(yh, None, None, None, None),
        lambda: moe.gemv.swiglu_q8_1(x, None),
        lambda: moe.gemv.moe_q(Q2_0, z, None, None, ids, n, 4, 576, False),
        lambda: moe.gemv.moe_q2_0(z, None, None, ids, n, 4, 576, False),
        lambda: moe.gemv.matvec(Q2_0, None, x, 4),
        lambda: moe.gemm.moe_prepare(Q2_0, 4, None, False, ids, n, z),
        lambda: moe.chain_rmsnorm_unit(x, None, out=torch.empty_like(x)),
    ]
    for call in calls:
        with pytest.raises(moe.FrxError, match="null|misaligned"):
            call()
