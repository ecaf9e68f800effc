"""Router top-k and the Q8 activation quantizer on the GPU against the oracle: ids, counts and
int8 codes bit-exact; weights within 1e-6 of the oracle and 1e-5 of a double reference. Needs a GPU."""
import numpy as np
import pytest
import torch

from flashrt_b200 import moe, synth
from helpers import cuda

pytestmark = pytest.mark.gpu


def test_route_tie_heavy_full_size():
    # the reference's own router test (tests/test_route_topk.cpp): 16,384 tokens, 512 experts,
    # top-10, logits rounded to 0.25 so exact ties are common
    T, E, K = 16384, 512, 10
    lg = synth.tie_heavy_logits(T, E)
    counts = torch.zeros(E, dtype=torch.int32, device="cuda")
    tail = torch.zeros(E, dtype=torch.int32, device="cuda")
    ids, wts = moe.moe_route_topk(cuda(lg), K, counts=counts, tail_counts=tail, tail_from=T - 100)
    ids, wts = ids.cpu().numpy(), wts.cpu().numpy()
    order = np.argsort(-lg, axis=1, kind="stable")[:, :K]
    assert np.array_equal(ids, order)
    assert np.array_equal(counts.cpu().numpy(), np.bincount(order.reshape(-1), minlength=E))
    assert np.array_equal(tail.cpu().numpy(), np.bincount(order[T - 100:].reshape(-1), minlength=E))
    l64 = lg.astype(np.float64)
    p = np.exp(l64 - l64.max(1, keepdims=True))
    p /= p.sum(1, keepdims=True)
    sel = np.take_along_axis(p, order, 1)
    assert np.abs(wts - sel / sel.sum(1, keepdims=True)).max() < 1e-5


@pytest.mark.parametrize("T,E,K", [(1, 512, 10), (64, 512, 10), (777, 512, 10), (33, 128, 8), (40, 1000, 32), (9, 8, 3), (5, 40, 32)])
def test_route_matches_oracle(port, T, E, K):
    lg = synth.router_logits(T, E)
    ids, wts = moe.moe_route_topk(cuda(lg), K)
    oid, ow, _ = port.route(lg, K)
    assert np.array_equal(ids.cpu().numpy(), oid)
    assert np.abs(wts.cpu().numpy() - ow).max() < 1e-6


def test_route_zipf_and_signed_zero(port):
    lg = synth.zipf_logits(512, 512)
    ids, wts = moe.moe_route_topk(cuda(lg), 10)
    oid, ow, _ = port.route(lg, 10)
    assert np.array_equal(ids.cpu().numpy(), oid)
    assert np.abs(wts.cpu().numpy() - ow).max() < 1e-6
    z = np.zeros((2, 64), np.float32)
    z[0, ::2] = -0.0                     # -0.0 and +0.0 tie: lower index first
    z[1, 5] = -np.inf
    ids, _ = moe.moe_route_topk(cuda(z), 4)
    assert np.array_equal(ids.cpu().numpy(), np.array([[0, 1, 2, 3], [0, 1, 2, 3]]))


def test_route_rejects_unsupported_shapes():
    lg = torch.zeros(4, 2048, device="cuda")
    with pytest.raises(moe.FrxError, match="unsupported shape"):
        moe.moe_route_topk(lg, 10)


def test_quantize_q8_bit_exact(port):
    rng = np.random.default_rng(7)
    x = rng.standard_normal((37, 2048), dtype=np.float32)
    x[1] *= 1e-6
    x[2] *= 3e4
    x[3, 64:96] = 0.0
    x[4, :32] = np.arange(-16, 16, dtype=np.float32) + 0.5          # amax 15.5
    x[5, :32] = 0
    x[5, 0], x[5, 1], x[5, 2], x[5, 3] = 127.0, 2.5, -2.5, 0.5       # d = 1: exact halves round away from zero
    x[6, :32] = 1e-30                                               # scale underflows in fp16
    q, d = moe.quantize_q8(cuda(x))
    oq, od = port.quantize_q8(x)
    assert np.array_equal(q.cpu().numpy(), oq)
    assert np.array_equal(d.cpu().numpy(), od)
    assert list(oq[5, :4]) == [127, 3, -3, 1]
    # the same rows from a buffer that is only 4-byte aligned (the one-value-per-lane form of the kernel)
    buf = torch.empty(x.size + 1, device="cuda")
    shifted = buf[1:].view(x.shape)
    shifted.copy_(cuda(x))
    assert shifted.data_ptr() % 16 == 4
    q2, d2 = moe.quantize_q8(shifted)
    assert torch.equal(q2, q) and torch.equal(d2, d)


def test_quantize_q8_empty_and_bad_shape():
    q, d = moe.quantize_q8(torch.zeros(0, 256, device="cuda"))
    assert q.shape == (0, 256)
    with pytest.raises(moe.FrxError):
        moe.quantize_q8(torch.zeros(2, 48, device="cuda"))


@pytest.mark.parametrize("T,E,n,gate", [(1, 512, 2048, True), (64, 512, 2048, True), (7, 33, 512, False), (200, 128, 1024, True)])
def test_router_projection(T, E, n, gate):
    # logits = W_r x (bf16 weights, fp32 activations and sums) and the shared expert's gate logit
    # in the same launch; tolerance against a float64 sum: fp32 accumulation over n terms
    from oracle import oracle
    rng = np.random.default_rng(3)
    w = torch.from_numpy(rng.standard_normal((E, n), dtype=np.float32) * 0.05).to(torch.bfloat16)
    wg = torch.from_numpy(rng.standard_normal(n, dtype=np.float32) * 0.05).to(torch.bfloat16) if gate else None
    x = rng.standard_normal((T, n), dtype=np.float32)
    logits, g = moe.router_logits(w.cuda(), wg.cuda() if gate else None, cuda(x))
    want = oracle.router_logits(w.view(torch.int16).numpy().view(np.uint16), x)
    scale = np.abs(want).max()
    assert np.abs(logits.cpu().numpy() - want).max() < 2e-6 * scale * np.sqrt(n / 256)
    if gate:
        wantg = oracle.router_logits(wg.view(torch.int16).numpy().view(np.uint16)[None, :], x)[:, 0]
        assert np.abs(g.cpu().numpy() - wantg).max() < 2e-6 * max(scale, np.abs(wantg).max()) * np.sqrt(n / 256)
    # feeding the router: the ids of the GPU logits are the ids of their own values
    ids, _ = moe.moe_route_topk(logits, min(8, E))
    top = np.argsort(-logits.cpu().numpy(), axis=1, kind="stable")[:, :min(8, E)]
    assert np.array_equal(ids.cpu().numpy(), top)


@pytest.mark.parametrize("T,E", [(15, 512), (16, 40), (17, 512), (33, 512), (40, 15), (41, 512), (64, 512), (137, 511), (293, 512), (321, 16),
                                 (2369, 7), (2433, 3), (9473, 7), (2400, 8), (6001, 16), (501, 130), (700, 99)])
def test_router_projection_same_bits_for_any_tile(T, E):
    # every tile adds in the same order (eight slices of n one after the other), so a token's logits do not
    # depend on how many tokens the call has; tails of rows and tokens included
    n = 768
    g = torch.Generator(device="cuda").manual_seed(T)
    w = torch.randn(E, n, generator=g, device="cuda").to(torch.bfloat16)
    wg = torch.randn(n, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(T, n, generator=g, device="cuda")
    logits, gate = moe.router_logits(w, wg, x)
    for t in {0, T // 2, T - 2, T - 1}:
        one, g1 = moe.router_logits(w, wg, x[t:t + 1].contiguous())
        assert torch.equal(one[0], logits[t]) and torch.equal(g1[0], gate[t])


@pytest.mark.parametrize("T,E,n", [(1, 1, 256), (9, 15, 512), (33, 17, 256), (130, 511, 2560), (300, 513, 2048), (600, 512, 768), (2500, 7, 256), (9480, 15, 256),
                                   (501, 130, 768), (700, 99, 2560)])
def test_router_projection_keeps_every_bit_of_the_activations(T, E, n):
    # activations with full 24-bit mantissas over the exponent range (the kernel multiplies them in three pieces of eight bits): rows from
    # 1e-36 to 1e30, an infinity and a missing number, against float64. Products are exact; how an MMA rounds its sums is not specified, so
    # the bounds are measurements: relative 2-norms of 1.1e-7 to 1.6e-7, and 3.3e-7 for rows of 1e-36 (multiply-adds one after the
    # other), times four. Activations of two pieces, 16 bits, are off by 1e-5. For a single logit, n / 8 + 7 roundings of 2^-24 of the
    # magnitudes, as the multiply-adds may have, or of half the smallest number.
    g = torch.Generator(device="cuda").manual_seed(n + T)
    w = torch.randn(E, n, generator=g, device="cuda").to(torch.bfloat16)
    wg = torch.randn(n, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(T, n, generator=g, device="cuda") * torch.tensor([1.0, 1e-36, 1e30, 1e-20], device="cuda")[torch.arange(T, device="cuda") % 4][:, None]
    if T > 8:
        x[T - 1, n // 3], x[T - 2, n - 1], x[T - 3, 0] = float("inf"), float("-inf"), float("nan")
    logits, gate = moe.router_logits(w, wg, x)
    wd = torch.cat([w, wg[None]]).double().T
    ref, mag = x.double() @ wd, x.double().abs() @ wd.abs()
    got = torch.cat([logits, gate.view(T, 1)], dim=1).double()
    fin = torch.isfinite(ref)
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(got[~fin & ~torch.isnan(ref)], ref[~fin & ~torch.isnan(ref)])
    assert bool(((got - ref).abs()[fin] <= ((n // 8 + 7) * (mag * 2.0 ** -24 + 2.0 ** -150))[fin]).all())
    rows = torch.isfinite(x).all(dim=1)
    cut = (x.view(torch.int32) & ~0xff).view(torch.float32).double() @ wd
    for i in range(min(T, 4)):
        sel = rows & (torch.arange(T, device="cuda") % 4 == i)
        bound = 1.4e-6 if i == 1 else 6.4e-7
        assert (got - ref)[sel].norm() <= bound * ref[sel].norm()
        assert T < 30 or (cut - ref)[sel].norm() > 4 * bound * ref[sel].norm()


# tokens, experts and n that reach each of the five tiles on 148 SMs, with tails of rows and tokens (the gate is one row more)
ROUTER_TILES = [(5, 99, 512), (501, 510, 512), (501, 130, 768), (301, 513, 2048), (2500, 7, 256)]


def test_router_projection_sizes_of_the_tests_reach_every_tile():
    from flashrt_b200.lib import lib
    assert [lib.frx_router_logits_tile(T, E + 1, n, 0) for T, E, n in ROUTER_TILES] == [1608, 3216, 4816, 4832, 1632]
    assert [lib.frx_router_logits_tile(T, E + 1, n, 0) for T, E, n in ((501, 130, 768), (700, 99, 768), (700, 99, 2560))] == [4816] * 3
    assert lib.frx_router_logits_tile(0, 5, 256, 0) == lib.frx_router_logits_tile(1, 5, 257, 0) == lib.frx_router_logits_tile(1, 0, 256, 0) == 0


@pytest.mark.parametrize("T,E,n", ROUTER_TILES)
def test_router_projection_with_infinite_weights(T, E, n):
    # activations of eight significant bits, as a bf16 residual stream has them: an infinite weight gives an infinite logit as in a
    # multiply-add, a missing number or an infinity times zero a missing number, and no other logit changes
    g = torch.Generator(device="cuda").manual_seed(T + E)
    w = torch.randn(E + 1, n, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(T, n, generator=g, device="cuda").to(torch.bfloat16).float()
    x[T // 2, n // 4] = 0.0
    x[T - 1, 3] = float("inf")
    clean = torch.cat([a.reshape(T, -1) for a in moe.router_logits(w[:E].contiguous(), w[E], x)], dim=1)
    w[1, n // 4], w[E - 1, n - 1], w[E - 2, 0], w[E, n // 2] = float("inf"), float("-inf"), float("nan"), float("-inf")
    got = torch.cat([a.reshape(T, -1) for a in moe.router_logits(w[:E].contiguous(), w[E], x)], dim=1)
    ref = x.double() @ w.double().T
    fin = torch.isfinite(ref)
    assert not fin[:, [1, E - 1, E - 2, E]].any() and torch.isinf(ref[:, 1]).sum() >= T - 2 and torch.isnan(ref[T // 2, 1])
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(got[torch.isinf(ref)].double(), ref[torch.isinf(ref)])
    assert torch.equal(got[fin], clean[fin])


@pytest.mark.parametrize("T,E,n", ROUTER_TILES)
def test_router_projection_one_activation_comes_through_whole(T, E, n):
    # a token with one activation, of 24 significant bits and any exponent down to the smallest subnormal number, and rows of one weight,
    # +1 or -1, at a place of their own: the logit is that activation, to the bit, or zero
    g = torch.Generator(device="cuda").manual_seed(T + n)
    places = torch.randint(0, n, (T,), generator=g, device="cuda")
    bits = torch.randint(0, 255 << 23, (T,), generator=g, device="cuda", dtype=torch.int32)   # all finite magnitudes
    bits[::3] = torch.randint(1, 40 << 23, bits[::3].shape, generator=g, device="cuda", dtype=torch.int32)   # below 2^-87
    bits[:3] = torch.tensor([1, (1 << 23) - 1, (255 << 23) - 1], device="cuda")
    v = (bits | torch.randint(0, 2, (T,), generator=g, device="cuda", dtype=torch.int32) << 31).view(torch.float32)
    x = torch.zeros(T, n, device="cuda").scatter_(1, places[:, None], v[:, None])
    rows = torch.randint(0, n, (E + 1,), generator=g, device="cuda")
    rows[::2] = places[torch.arange(0, E + 1, 2, device="cuda") % T]   # so that some meet
    sign = torch.randint(0, 2, (E + 1,), generator=g, device="cuda").float() * 2 - 1
    w = torch.zeros(E + 1, n, device="cuda").scatter_(1, rows[:, None], sign[:, None]).to(torch.bfloat16)
    got = torch.cat([a.reshape(T, -1) for a in moe.router_logits(w[:E].contiguous(), w[E], x)], dim=1)
    want = torch.where(places[:, None] == rows[None, :], v[:, None] * sign[None, :], torch.zeros((), device="cuda"))
    assert (want != 0).sum() >= min(T, E) // 2 and torch.equal(got, want)


@pytest.mark.parametrize("exponent", [-109, -112, -118, -124, -130])
@pytest.mark.parametrize("T,E,n", ROUTER_TILES)
def test_router_projection_of_small_activations(T, E, n, exponent):
    # below 2^-110 a third piece of eight bits would be below bf16's smallest number. fp32 products and sums in eight slices one after the
    # other: n / 8 + 7 additions of at most 2^-24 of the magnitudes, or of half the smallest subnormal number
    g = torch.Generator(device="cuda").manual_seed(T + E + exponent)
    w = torch.randn(E + 1, n, generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn(T, n, generator=g, device="cuda")
    x[1::2] *= 2.0 ** exponent
    x[0, 1:] *= 2.0 ** exponent   # small ones beside an ordinary one
    got = torch.cat([a.reshape(T, -1) for a in moe.router_logits(w[:E].contiguous(), w[E], x)], dim=1).double()
    ref, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert ((got - ref).abs() <= (n // 8 + 7) * (mag * 2.0 ** -24 + 2.0 ** -150)).all()
    small = (got - ref)[1::2].norm() / ref[1::2].norm()
    assert small < 2e-6 + 2.0 ** (-148 - exponent)   # (three pieces alone: 2^(-135 - exponent) and more)


@pytest.mark.parametrize("T,E,n", [(1, 64, 512), (37, 512, 2048), (293, 130, 2560), (2500, 7, 256)])
def test_router_projection_of_activations_that_are_rewritten_in_place(T, E, n):
    # the kernel in front writes x, lets the projection start early, and the next step writes the same addresses again; directly and replayed
    g = torch.Generator(device="cuda").manual_seed(T)
    w = torch.randn(E, n, generator=g, device="cuda").to(torch.bfloat16)
    src = torch.randn(12, T, n, generator=g, device="cuda")
    zero, x = torch.zeros(T, n, device="cuda"), torch.empty(T, n, device="cuda")
    want = [moe.router_logits(w, w[0], moe.chain_rmsnorm_unit(s, zero)) for s in src]
    torch.cuda.synchronize()

    def steps():
        return [moe.router_logits(w, w[0], moe.chain_rmsnorm_unit(s, zero, out=x)) for s in src]

    for _ in range(3):
        got = steps()
        assert all(torch.equal(a, b) for p, q in zip(got, want) for a, b in zip(p, q))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = steps()
    src.copy_(src.flip(0))
    for _ in range(2):
        graph.replay()
    assert all(torch.equal(a, b) for p, q in zip(got, reversed(want)) for a, b in zip(p, q))


@pytest.mark.parametrize("n", [1, 31, 33, 512, 2048, 4095, 4096, 4097, 9000])
def test_chain_rmsnorm_order_of_additions(n):
    rng = np.random.default_rng(n)
    x, y = rng.standard_normal((3, n), dtype=np.float32), rng.standard_normal((3, n), dtype=np.float32)
    r = x + y
    sq = np.zeros((3, -(-n // 32) * 32))
    sq[:, :n] = r.astype(np.float64) ** 2
    lanes = np.zeros((3, 32))
    for row in sq.reshape(3, -1, 32).transpose(1, 0, 2):
        lanes = lanes + row
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[:, np.arange(32) ^ o]
    inv = (1.0 / np.sqrt(lanes[:, :1] / n + 1e-6)).astype(np.float32)
    assert np.array_equal(moe.chain_rmsnorm_unit(cuda(x), cuda(y)).cpu().numpy(), r * inv)


@pytest.mark.parametrize("n,T", [(640, 149), (1024, 297), (2048, 593), (512, 2), (128, 4096)])
def test_chain_rmsnorm_forms_give_the_same_bits(n, T):
    # T is one token more than the block form takes at this length (none at 512 and 128): rows of the long call against calls
    # of one token, which take the block form from 640 on
    rng = np.random.default_rng(n)
    x, y = cuda(rng.standard_normal((T, n), dtype=np.float32)), cuda(rng.standard_normal((T, n), dtype=np.float32))
    got = moe.chain_rmsnorm_unit(x, y)
    for t in {0, 1, T // 2, T - 1}:
        assert torch.equal(moe.chain_rmsnorm_unit(x[t:t + 1].contiguous(), y[t:t + 1].contiguous())[0], got[t])
    ref = (x + y).double()
    ref = ref / (ref.square().mean(dim=1, keepdim=True) + 1e-6).sqrt()
    assert float((got.double() - ref).abs().max() / ref.square().mean().sqrt()) < 1e-5   # rows of +-5: three roundings of 2^-24 each
