"""moe_hits (per-token lists of expert pointers) and the prefill-sized grouped expert product
(moe_q2::run) on the GPU against the CPU oracle. Needs a GPU."""
import numpy as np
import pytest
import torch

from flashrt_b200 import moe, synth
from helpers import Experts, cuda, rel_max

pytestmark = pytest.mark.gpu


def hits_call(ex, x, slot_of, hit_n):
    T, K = slot_of.shape
    ptrs = torch.tensor((ex.base + slot_of.astype(np.int64) * ex.stride).reshape(-1), dtype=torch.int64, device="cuda")
    yh = torch.full((T, K, ex.n), float("nan"), device="cuda")
    scratch = moe.workspace(moe.moe_hits_scratch_bytes(K, ex.n, ex.ff, T))
    moe.moe_hits(ptrs, cuda(hit_n), K, cuda(x), ex.n, ex.ff, yh, scratch=scratch, T=T)
    moe.workspace_status(scratch)
    return yh.cpu().numpy()


def test_hits_single_token_with_pad_entry(port):
    # tests/test_moe_hits.cpp:62-122: 10 entries over 16 slots, the last a pad entry that must not be written
    n, ff, K = 2560, 640, 10
    ex = Experts(port, n, ff, 16, shared=False, seed=7)
    x = synth.activations(1, n)
    slot_of = np.array([[3, 11, 0, 7, 15, 5, 9, 2, 13, 3]])
    yh = hits_call(ex, x, slot_of, np.array([9], np.int32))
    assert np.all(np.isnan(yh[0, 9]))
    xq, xd = port.quantize_q8(x)
    for k in range(9):
        assert rel_max(yh[0, k], port.expert_ffn(ex.planar[slot_of[0, k]], n, ff, xq[0], xd[0])) < 1e-5


def test_hits_window_bit_identical_to_single_token_calls(port):
    # tests/test_moe_hits.cpp:125-165
    n, ff, K, T = 2560, 640, 10, 3
    ex = Experts(port, n, ff, 16, shared=False, seed=7)
    x = synth.activations(T, n)
    slot_of = np.array([[3, 11, 0, 7, 15, 5, 9, 2, 13, 3], [11, 3, 6, 7, 1, 5, 9, 12, 14, 8], [0, 11, 4, 10, 15, 2, 6, 3, 13, 1]])
    hit_n = np.array([9, 10, 7], np.int32)
    yw = hits_call(ex, x, slot_of, hit_n)
    for t in range(T):
        y1 = hits_call(ex, x[t:t + 1], slot_of[t:t + 1], hit_n[t:t + 1])
        assert np.array_equal(yw[t, :hit_n[t]], y1[0, :hit_n[t]])
        assert np.all(np.isnan(yw[t, hit_n[t]:]))


def test_hits_rejects_large_windows():
    with pytest.raises(moe.FrxError, match="unsupported window"):
        moe.moe_hits(torch.zeros(200 * 10, dtype=torch.int64, device="cuda"), torch.zeros(200, dtype=torch.int32, device="cuda"), 10,
                     torch.zeros(200, 256, device="cuda"), 256, 128, torch.zeros(200, 10, 256, device="cuda"), T=200)


@pytest.mark.parametrize("form", ["stream", "umma"])
@pytest.mark.parametrize("T,E,K,zipf", [(96, 16, 4, False), (300, 24, 6, True), (1, 8, 2, False), (1200, 12, 3, True)])
def test_prefill_per_slot_outputs(port, T, E, K, zipf, form):
    # moe_q2::run contract: yd[t*K + k] = expert ids[t][k] applied to x_t
    n, ff = 256, 128
    ex = Experts(port, n, ff, E, shared=False)
    x = synth.activations(T, n, through_bf16=True)
    lg = synth.zipf_logits(T, E) if zipf else synth.router_logits(T, E)
    ids, wts, _ = port.route(lg, K)
    ws = moe.workspace(moe.moe_q2.workspace_bytes(T, K, n, ff, E))
    yd = moe.moe_q2.run(ex.base, ex.stride, E, n, ff, cuda(x), cuda(ids), ws=ws, form=form)
    moe.workspace_status(ws)
    yd = yd.cpu().numpy()
    _, ref_ys, _ = port.moe_layer(ex.routed_planar(), ex.blob_bytes, None, n, ff, x, ids, wts, None, n_threads=8, want_slots=True)
    assert max(rel_max(yd[s], ref_ys[s]) for s in range(T * K)) < 1e-5


def test_prefill_config_shape_sample(port):
    # layer shape of the benchmark's prefill config, fewer experts and tokens; a sample of slots;
    # the tensor-memory form (chosen by size) and the streaming form must agree to the bit
    n, ff, E, K, T = 2048, 512, 32, 10, 256
    ex = Experts(port, n, ff, E, shared=False, direct=True)
    x = synth.activations(T, n, through_bf16=True)
    ids, wts, _ = port.route(synth.zipf_logits(T, E), K)
    yd = moe.moe_q2.run(ex.base, ex.stride, E, n, ff, cuda(x), cuda(ids)).cpu().numpy()
    assert np.array_equal(yd, moe.moe_q2.run(ex.base, ex.stride, E, n, ff, cuda(x), cuda(ids), form="stream").cpu().numpy())
    xq, xd = port.quantize_q8(x)
    for s in range(0, T * K, 97):
        t, k = divmod(s, K)
        assert rel_max(yd[s], port.expert_ffn(ex.planar[ids[t, k]], n, ff, xq[t], xd[t])) < 1e-5


@pytest.mark.parametrize("T,E,K", [(1, 3, 1), (127, 5, 3), (129, 4096, 2), (1024, 2, 1), (1025, 300, 3), (2500, 48, 4)])
def test_grouping_edges(port, T, E, K):
    # chunks of 1024 slots in parts of 128, items of 8, token blocks of 48: one more, one less, all slots on one expert; both
    # forms group for themselves, and every slot's row must be its own expert's
    n, ff = 128, 128
    planar = synth.planar_experts_random(np.random.default_rng(E), min(E, 24), n, ff)
    stride = moe.expert_stride(n, ff)
    some = moe.tile_experts(cuda(planar.reshape(-1)), n, ff, len(planar)).view(len(planar), stride)
    tiled = some[torch.arange(E, device="cuda") % len(planar)].contiguous()
    rng = np.random.default_rng(T)
    ids = rng.integers(0, E, size=(T, K)).astype(np.int32)
    ids[: T // 2] = E - 1                                                # half the slots on one expert
    x = synth.activations(T, n)
    ws = moe.workspace(moe.moe_q2.workspace_bytes(T, K, n, ff, E))
    yd = {}
    for form in ("stream", "umma"):
        yd[form] = moe.moe_q2.run(tiled.data_ptr(), stride, E, n, ff, cuda(x), cuda(ids), ws=ws, form=form)
        moe.workspace_status(ws)
    assert torch.equal(yd["stream"], yd["umma"])
    xq, xd = port.quantize_q8(x)
    got = yd["stream"].cpu().numpy()
    for s in sorted({0, T * K - 1, *rng.integers(0, T * K, size=24).tolist()}):
        t, k = divmod(s, K)
        assert rel_max(got[s], port.expert_ffn(planar[ids[t, k] % len(planar)], n, ff, xq[t], xd[t])) < 1e-5


@pytest.mark.parametrize("n,ff", [(512, 256), (384, 640), (2560, 128)])
def test_warps_that_only_build_items_give_the_same_bits(port, n, ff):
    # the large block of the streaming kernels leaves the item buffers to four warps of its own; here a block goes
    # through more than twice as many items as it has buffers, against blocks whose warps do both
    from flashrt_b200.lib import check, lib
    T, E, K = 900, 256, 6                # 21 tokens per expert: about 900 items of up to eight
    ex = Experts(port, n, ff, E, shared=False, direct=True)
    x = cuda(synth.activations(T, n))
    ids = cuda(np.argsort(synth.zipf_logits(T, E), axis=1)[:, :K].astype(np.int32))
    got = moe.moe_q2.run(ex.base, ex.stride, E, n, ff, x, ids)
    try:
        check(lib.frx_debug_set_consumer_warps(8))
        want = moe.moe_q2.run(ex.base, ex.stride, E, n, ff, x, ids)
    finally:
        check(lib.frx_debug_set_consumer_warps(12))
    assert torch.equal(got, want)


def test_prefill_with_more_slots_on_an_expert_than_a_square_root_of_int32(port):
    # 1.4 million slots of one expert: 87,500 units of 16 in 29,167 token blocks, whose product is above 2^31
    n, ff, T = 128, 128, 1_400_000
    ex = Experts(port, n, ff, 1, shared=False)
    rows = synth.activations(997, n)
    x = cuda(rows).repeat(T // len(rows) + 1, 1)[:T]
    ids = torch.zeros(T, 1, dtype=torch.int32, device="cuda")
    ws = moe.workspace(moe.moe_q2.workspace_bytes(T, 1, n, ff, 1))
    yd = moe.moe_q2.run(ex.base, ex.stride, 1, n, ff, x, ids, ws=ws, form="umma")
    moe.workspace_status(ws)
    xq, xd = port.quantize_q8(rows)
    want = cuda(np.stack([port.expert_ffn(ex.planar[0], n, ff, q, d) for q, d in zip(xq, xd)]))
    assert rel_max(yd[:len(rows)].cpu().numpy(), want.cpu().numpy()) < 1e-5
    # the same token gives the same bits wherever it lies
    whole = T // len(rows) * len(rows)
    assert torch.equal(yd[:whole].view(-1, len(rows), n), yd[:len(rows)].expand(whole // len(rows), -1, -1))
    assert torch.equal(yd[whole:], yd[:T - whole])


@pytest.mark.parametrize("block64", [False, True])
@pytest.mark.parametrize("S", [1, 3, 63, 64, 65, 4097])
def test_hidden_quantizer_where_rows_end_inside_a_warp(port, S, block64):
    # rows of four 32-blocks, eight to a warp: an odd number of rows leaves the last warp of the hidden-row quantizer half full
    n, ff = 256, 128
    ex = Experts(port, n, ff, 1, shared=False)
    x, ids = cuda(synth.activations(S, n)), torch.zeros(S, 1, dtype=torch.int32, device="cuda")
    ws = moe.workspace(moe.moe_q2.workspace_bytes(S, 1, n, ff, 1))
    got, want = (moe.moe_q2.run_ex(ex.base, ex.stride, 1, n, ff, x, ids, block64=block64, ws=ws, form=f) for f in ("umma", "stream"))
    moe.workspace_status(ws)
    assert torch.equal(got, want)


def hidden_codes(pairs, block):
    """The quantizer of hidden rows restated: fp32 silu(g) * u with a correctly rounded exponential, d = amax / 127, id = 1 / d,
    codes to the nearest integer, halves away from zero; missing numbers have code 0 and no part in the maximum."""
    f32 = np.float32
    g, u = pairs[..., 0], pairs[..., 1]
    with np.errstate(all="ignore"):
        h = (g / (f32(1) + np.exp(-g.astype(np.float64)).astype(f32)) * u).reshape(len(g), -1, block)
        d = np.fmax.reduce(np.abs(h), axis=-1, keepdims=True, initial=f32(0)) / f32(127)
        c = h * np.where(d != 0, f32(1) / d, f32(0))
        t = np.trunc(c)
        code = np.nan_to_num(np.where(np.abs(c - t) >= 0.5, t + np.copysign(f32(1), c), t)).reshape(g.shape)
        scale = np.repeat(d[..., 0].astype(np.float16).astype(f32), block // 32, axis=-1)
    assert h.dtype == d.dtype == c.dtype == f32
    return code, scale, np.broadcast_to(d, h.shape).reshape(g.shape)


def hidden_rows(kind, R, ff, rng):
    """(gate x, up x) pairs [R][ff][2]: the values that decide which of the quantizer's values are formed how."""
    g, u = rng.normal(0, 3, (R, ff)), rng.normal(0, 1, (R, ff))
    some = rng.random((R, ff)) < 0.3
    sign = rng.choice([-1.0, 1.0], (R, ff))
    if kind == "steep":                    # gates to beyond both ends of the exponential's range
        g *= 40
    elif kind == "rounding":               # codes next to, and on, the halves: silu(g) = g from 17 on
        g, u = np.where(rng.random((R, ff)) < 0.1, 127.0, rng.integers(17, 127, (R, ff)) + 0.5), sign * (1 + rng.integers(-2, 3, (R, ff)) * 2.0 ** -23)
    elif kind == "last of the exponential":
        g, u = rng.uniform(-95, -70, (R, ff)), sign * 10 ** rng.uniform(8, 12, (R, ff))
    elif kind == "tiny gates":             # silu(g) below the normal numbers, brought back by u
        tiny = np.where(rng.random((R, ff)) < 0.5, rng.integers(1, 64, (R, ff)) * 2.0 ** -149, 10 ** rng.uniform(-44.5, -37, (R, ff)))
        g, u = np.where(some, sign * tiny, g), np.where(some, 10 ** rng.uniform(13, 38, (R, ff)), u * 1e-6)
    elif kind == "small":                  # block maxima around 1e-25 and down to where d is no normal number
        g, u = g * 1e-13, u * 10 ** rng.uniform(-26, -11, (R, 1))
    elif kind == "large":                  # around 1e25 and beyond the floats
        g, u = np.abs(g) * 1e12, u * 10 ** rng.uniform(11, 27, (R, 1))
    elif kind == "zeros":                  # whole blocks, whole rows, and blocks with a single value
        g[:, :ff // 2] = 0
        g[R // 2:] = sign[R // 2:] * 0.0
        u[: R // 4, ff // 2:] = 0
        g[R // 2:, 5::64] = 2.0
    elif kind == "equal":                  # every value may be the largest
        g[:], u = 3.0, sign
    elif kind == "not finite":             # one in every third block
        g = np.abs(g) + 0.1                # (an infinite up x times a positive gate)
        for i, j in zip(*np.nonzero(rng.random((R, ff // 32)) < 0.33)):
            (g if rng.random() < 0.5 else u)[i, 32 * j + rng.integers(32)] = rng.choice([np.inf, -np.inf, np.nan])
    else:
        assert kind == "ordinary"
    return np.stack([g, u], axis=-1).astype(np.float32)


@pytest.mark.parametrize("block", [32, 64])
@pytest.mark.parametrize("kind", ["ordinary", "steep", "rounding", "last of the exponential", "tiny gates", "small", "large", "zeros", "equal", "not finite"])
def test_hidden_quantizer_codes(kind, block):
    from flashrt_b200.lib import check, lib
    R, ff = 4001, 384
    pairs = hidden_rows(kind, R, ff, np.random.default_rng(5))
    pieces = torch.full((R + 3, ff // 64, 128), 0x55, dtype=torch.uint8, device="cuda")
    scales = torch.full((R + 3, ff // 32), -7.0, device="cuda")
    x, n_rows = cuda(np.concatenate([pairs, pairs[:3]])), torch.tensor([R], dtype=torch.int32, device="cuda")
    check(lib.frx_debug_quantize_hidden(x.data_ptr(), n_rows.data_ptr(), R + 3, ff, pieces.data_ptr(), scales.data_ptr(), int(block == 64),
                                        torch.cuda.current_stream().cuda_stream))
    assert (pieces[R:] == 0x55).all() and (scales[R:] == -7).all()   # rows that are not there
    # bytes [s][piece][t / 2][t % 2][q][i] -> elements [s][q][t][i]
    b = pieces[:R].cpu().view(torch.float8_e4m3fn).float().view(R, ff // 64, 2, 2, 2, 2, 2, 4).sum(dim=3)
    got = b.permute(0, 1, 2, 5, 3, 4, 6).reshape(R, ff).numpy()
    want, scale, d = hidden_codes(pairs, block)
    assert np.array_equal(scales[:R].cpu().numpy(), scale)
    sure = d >= 2.0 ** -126   # below, 1 / d may be none, and the scale is 0 as fp16
    assert sure.any() and np.array_equal(got[sure], want[sure])
    if kind not in ("not finite", "large"):
        assert (np.abs(want[sure]).max(initial=0) == 127) and (kind == "zeros" or (want[sure] != 0).mean() > 0.1)
    if kind in ("ordinary", "steep", "rounding"):   # an exponential that is off by 2^-18 would show
        off = pairs.copy()
        off[..., 1] *= np.random.default_rng(6).choice(np.float32([1 - 2.0 ** -18, 1 + 2.0 ** -18]), off.shape[:2])
        assert (hidden_codes(off, block)[0] != want).sum() > 10


@pytest.mark.parametrize("block64", [False, True])
@pytest.mark.parametrize("spread", [0.02, 8.0, 6e4, "special"])
def test_hidden_quantizer_over_the_range_of_the_swiglu(port, spread, block64):
    # the whole product against the form that computes the exact SwiGLU for every value, gate values from a few units to beyond the
    # exponential's range. Scales pass through fp16, so rows of large values come out as missing numbers and rows of small ones as zeros
    # (all of them in "special"): what this shows for those is that they do so in both forms. test_hidden_quantizer_codes has the codes.
    n, ff, E, S = 256, 384, 2, 333
    rng = np.random.default_rng(11)
    planar = np.zeros((E, moe.expert_bytes(n, ff)), np.uint8)
    off = 0
    for rows, cols in ((ff, n), (ff, n), (n, ff)):
        nblk = rows * cols // 64
        planar[:, off:off + nblk * 16] = rng.integers(0, 256, (E, nblk * 16))
        scale = rng.normal(0, 0.02 if spread == "special" or cols == ff else spread, (E, nblk)).clip(-6e4, 6e4).astype(np.float16)
        if spread == "special" and cols == n:
            scale[:, rng.integers(0, nblk, 40)] = rng.choice(np.array([np.inf, -np.inf, np.nan, 6e4, 6e-8], np.float16), 40)
            scale[0, :nblk // 4] = 0
        planar[:, off + nblk * 16:off + nblk * 18] = scale.view(np.uint8)
        off += nblk * 18
    tiled = moe.tile_experts(cuda(planar.reshape(-1)), n, ff, E)
    x = synth.activations(S, n) * rng.choice(np.array([1e-30, 1e-3, 1.0, 3e4], np.float32), (S, 1))
    ids = cuda(rng.integers(0, E, (S, 1)).astype(np.int32))
    got, want = (moe.moe_q2.run_ex(tiled.data_ptr(), moe.expert_stride(n, ff), E, n, ff, cuda(x), ids, block64=block64, form=f) for f in ("umma", "stream"))
    assert torch.allclose(got, want, rtol=0, atol=0, equal_nan=True)


@pytest.mark.parametrize("n,ff,E,K,per_expert,umma", [(2048, 512, 1, 1, 64, False), (2560, 640, 2, 2, 200, False), (512, 256, 8, 4, 32, False), (512, 256, 64, 8, 31, False),
                                                      (512, 256, 64, 8, 48, True), (2048, 512, 64, 8, 64, True), (384, 640, 16, 4, 300, True), (4096, 1024, 1, 1, 40, True)])
def test_prefill_takes_the_form_that_fills_the_gpu(port, n, ff, E, K, per_expert, umma):
    # few experts leave most SMs without a tile of the tensor-memory form; a shape that the streaming form has no room for takes
    # the other one from 32 tokens per expert on
    from flashrt_b200.lib import lib
    T = per_expert * E // K
    assert lib.frx_moe_prefill_form(T, K, n, ff, E, E) == (2 if umma else 1)
    assert lib.frx_moe_prefill_form(4 * T, K, n, ff, 4 * E, E) == (2 if umma else 1)      # a quarter of the experts is here
    ex = Experts(port, n, ff, E, shared=False, direct=True)
    x, ids = cuda(synth.activations(T, n)), torch.randint(0, E, (T, K), dtype=torch.int32, device="cuda")
    got = moe.moe_q2.run(ex.base, ex.stride, E, n, ff, x, ids)
    assert torch.equal(got, moe.moe_q2.run(ex.base, ex.stride, E, n, ff, x, ids, form="umma" if umma else "stream"))
