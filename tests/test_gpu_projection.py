"""The steps either side of the expert kernels, and the boundary's remaining forms, on the GPU against the CPU oracle:
the router-logits projection (streaming and tcgen05), router + pack as one launch, the residual add, the dense tcgen05
projections (linear_q*_wmma), FP32 activations, and a C++ host that issues the reference's call block through the shim."""
import re
import subprocess

import numpy as np
import pytest
import torch

from helpers import bf16_tensor, bits_of, capture_calls, max_abs_over_rms, random_weights, upload

pytestmark = pytest.mark.gpu


def logits_f64(oracle, x_bits, w, bias):
    return oracle.bf16_to_f32(x_bits).astype(np.float64) @ w.astype(np.float64).T + bias.astype(np.float64)


@pytest.mark.parametrize("M,N,K,w_bf16", [(16, 513, 4096, False), (1, 65, 1024, True), (37, 513, 4096, True), (64, 129, 512, False)])
def test_router_logits_streaming(cuda, oracle, M, N, K, w_bf16):
    """logits = x W^T + bias against a float64 evaluation: within 1e-5 of the largest logit (FP32 sums of exact products)."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(M * 1000 + N)
    xb = oracle.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    bias = (rng.standard_normal(N) * 0.5).astype(np.float32)
    if w_bf16:
        wb = oracle.f32_to_bf16(w)
        w = oracle.bf16_to_f32(wb)
        w_dev = bf16_tensor(wb, cuda)
    else:
        w_dev = torch.from_numpy(w).to(cuda)
    x = bf16_tensor(xb, cuda)
    ld = N + 3
    out = torch.full((M, ld), float("nan"), dtype=torch.float32, device=cuda)
    Kn.router_logits(x, w_dev, torch.from_numpy(bias).to(cuda), out)
    want = logits_f64(oracle, xb, w, bias)
    got = out.cpu().numpy()
    assert np.all(np.isnan(got[:, N:])), "columns past N must stay untouched"
    assert np.max(np.abs(got[:, :N] - want)) <= 1e-5 * np.max(np.abs(want))
    if w_bf16:  # the reference's launcher (kernels/linear.hpp:22-27): no bias, ld = N, F32 or BF16 out
        y32 = torch.empty((M, N), dtype=torch.float32, device=cuda)
        ybf = torch.empty((M, N), dtype=torch.bfloat16, device=cuda)
        Kn.linear_bf16w(x, w_dev, y32, M, N, K, Kn.Act.BF16, Kn.Act.F32)
        Kn.linear_bf16w(x, w_dev, ybf, M, N, K, Kn.Act.BF16)
        plain = logits_f64(oracle, xb, w, np.zeros(N, np.float32))
        assert np.max(np.abs(y32.cpu().numpy() - plain)) <= 1e-5 * np.max(np.abs(plain))
        assert torch.equal(ybf, y32.to(torch.bfloat16))


@pytest.mark.parametrize("w_bf16", [False, True])
@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (8, 15, 40), (9, 16, 2048), (16, 17, 4104), (33, 130, 4096), (127, 513, 1000)])
def test_router_logits_streaming_edges(cuda, oracle, M, N, K, w_bf16):
    """Groups of 8 and 16 tokens full, one over or partly filled, rows past a tile of 16, contractions that end inside a run of 32 or leave
    warps without one.  Exact products added in chains of at most 128 (K <= 4104: a warp's runs, 16 products an MMA, 64 parts): within
    2^-17 sum|terms| of 64 bits.  Infinities keep their sign, NaN stays, and a row does not notice its batch."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(M + 31 * N + K)
    xb = oracle.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    if w_bf16:
        w = oracle.bf16_to_f32(oracle.f32_to_bf16(w))
    w_dev = torch.from_numpy(w).to(cuda)
    w_dev = w_dev.to(torch.bfloat16) if w_bf16 else w_dev
    bias = torch.from_numpy(rng.standard_normal(N).astype(np.float32)).to(cuda)
    x, out = bf16_tensor(xb, cuda), torch.empty((M, N), dtype=torch.float32, device=cuda)
    Kn.router_logits(x, w_dev, bias, out)
    xf, b = oracle.bf16_to_f32(xb).astype(np.float64), bias.cpu().numpy().astype(np.float64)
    want = xf @ w.astype(np.float64).T + b
    assert np.all(np.abs(out.cpu().numpy() - want) <= 2.0 ** -17 * (np.abs(xf) @ np.abs(w).T.astype(np.float64) + np.abs(b)))
    one = torch.empty((1, N), dtype=torch.float32, device=cuda)
    Kn.router_logits(x[M - 1:].clone(), w_dev, bias, one)
    assert torch.equal(one[0], out[M - 1])
    x2, w2 = x.clone(), w_dev.clone()
    x2[0, K - 1] = float("-inf")
    w2[N - 1, K - 2] = float("inf")
    out2 = torch.empty_like(out)
    Kn.router_logits(x2, w2, bias, out2)
    with np.errstate(invalid="ignore"):
        want2 = x2.double().cpu().numpy() @ w2.double().cpu().numpy().T
    got2 = out2.cpu().numpy()
    bad = ~np.isfinite(want2)
    assert np.array_equal(got2[bad], want2[bad], equal_nan=True) and np.array_equal(got2[~bad], out.cpu().numpy()[~bad])


@pytest.mark.parametrize("w_bf16", [False, True])
@pytest.mark.parametrize("M,N,K", [(17, 513, 4096), (24, 600, 8), (63, 530, 4128), (64, 513, 8192), (65, 514, 1000), (129, 520, 12296), (37, 65, 4096)])
def test_router_logits_streaming_eights(cuda, M, N, K, w_bf16):
    """Above sixteen tokens and a machine full of CTAs, a CTA keeps its weights for eight eights of tokens: groups full, partly filled and one over,
    an odd number of eights, contractions of one pass of a warp's registers, several, and none.  A token's sums do not depend on its group: every row has the
    bits of the call for that token by itself."""
    from strixite_b200 import kernels as Kn
    gen = torch.Generator(device="cpu").manual_seed(M + N + K)
    x = torch.randn(M, K, generator=gen).to(cuda).to(torch.bfloat16)
    w = (torch.randn(N, K, generator=gen) * 0.02).to(cuda).to(torch.bfloat16 if w_bf16 else torch.float32)
    bias = torch.randn(N, generator=gen).to(cuda)
    out = torch.full((M, N + 2), float("nan"), device=cuda)
    Kn.router_logits(x, w, bias, out)
    one = torch.empty((M, N), device=cuda)
    for m in range(M):
        Kn.router_logits(x[m:m + 1], w, bias, one[m:m + 1])
    assert torch.equal(out[:, :N], one) and bool(torch.isnan(out[:, N:]).all())


@pytest.mark.parametrize("M,N,K", [(1, 17, 64), (16, 513, 4096), (37, 33, 1000)])
def test_router_logits_streaming_third_plane(cuda, oracle, M, N, K):
    """FP32 weights whose last bits are all that is left of a logit: pairs 1 + 2^-8 + k 2^-23 and -(1 + 2^-8) against the same activation, a
    small whole number, so that every sum is exact in FP32 whatever its order.  The logits are the 64-bit ones, bit for bit; cut to two
    BF16 planes (16 bits) the weights give zeros."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(M + N)
    w = np.empty((N, K), dtype=np.float32)
    w[:, 0::2] = 1 + 2.0 ** -8 + rng.integers(1, 128, (N, K // 2)) * 2.0 ** -23
    w[:, 1::2] = -(1 + 2.0 ** -8)
    x = np.repeat(rng.integers(-3, 4, (M, K // 2)), 2, axis=1).astype(np.float32)
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert not np.any(x.astype(np.float64) @ (w.view(np.uint32) & 0xFFFFFF00).view(np.float32).astype(np.float64).T)
    out = torch.empty((M, N), dtype=torch.float32, device=cuda)
    Kn.router_logits(torch.from_numpy(x).to(cuda).to(torch.bfloat16), torch.from_numpy(w).to(cuda), None, out)
    assert np.any(want) and np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("form", ["dense", "router"])
def test_non_finite_rows(cuda, oracle, form):
    """NaN and infinities in some tokens' activations and, for the router, weights: the results are what 64 bits give, and the other
    tokens keep their bits.  Nor does a token of NaN hold the call up: forming every one of its results again, one thread each, took 20 times
    the call's time; looking at its activations once is a small part of it.  (x 5: the clock and the first launch.)"""
    from strixite_b200 import kernels as Kn
    M, N, K = 8, 4096, 4096
    rng = np.random.default_rng(5)
    x = torch.randn((M, K), device=cuda).to(torch.bfloat16)
    if form == "dense":
        wq = oracle.quantize(np.abs(rng.standard_normal((N, K)).astype(np.float32)), 64, 8)
        wq.q[3, 7], wq.minv[3, 0] = 0, 0  # a weight of zero against an infinity
        wd, w64 = upload(wq, cuda), torch.from_numpy(oracle.affine_weights(wq)).to(cuda)
        call = lambda xs, out: Kn.linear_qw(xs, wd, out, M, Kn.Act.BF16, out_act=Kn.Act.F32)
    else:
        wd = torch.randn((N, K), device=cuda) * 0.02
        wd[3, 7] = 0.0
        wd[5, 9], wd[6, 9] = float("-inf"), float("nan")
        w64 = wd.double()
        call = lambda xs, out: Kn.router_logits(xs, wd, None, out)
    bad = x.clone()
    bad[1, 4000], bad[2, 7], bad[4, 7], bad[4, 8] = float("nan"), float("inf"), float("inf"), float("-inf")
    y, yb = (torch.empty((M, N), dtype=torch.float32, device=cuda) for _ in range(2))
    call(x, y)
    call(bad, yb)
    want = torch.stack([(row * w64).sum(dim=1) for row in bad.double()])
    odd = ~torch.isfinite(want)
    assert torch.equal(torch.isnan(yb), torch.isnan(want)) and torch.equal(yb[odd].nan_to_num(), want[odd].float().nan_to_num())
    assert torch.equal(yb[[0, 3, 5, 6, 7]].nan_to_num(), y[[0, 3, 5, 6, 7]].nan_to_num())

    def us(xs):
        e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        best = float("inf")
        for _ in range(5):
            e[0].record()
            for _ in range(10):
                call(xs, y)
            e[1].record()
            torch.cuda.synchronize()
            best = min(best, e[0].elapsed_time(e[1]) * 100)
        return best
    plain, all_nan = us(x), us(torch.full_like(x, float("nan")))
    assert all_nan <= 5 * plain, (plain, all_nan)


@pytest.mark.parametrize("M,N,K,planes,w_bf16", [(4096, 513, 4096, 3, False), (300, 513, 1024, 2, False), (1000, 129, 512, 1, True),
                                                   (128, 64, 256, 3, False)])
def test_router_logits_tcgen05(cuda, oracle, M, N, K, planes, w_bf16):
    """The tensor-core projection: three planes reproduce the FP32 weight exactly, two planes keep 16 bits of it, one plane
    is a BF16 weight.  What is left is the tensor cores' FP32 accumulation, which is not IEEE summation (the reference says
    the same of its matrix units, kernels/wmma.hpp:10-11): measured 1.3e-5 of the largest logit over K = 4096 x 3 planes,
    held to 3e-5 here (the streaming form, plain FP32 FMAs, is held to 1e-5)."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(M + N + planes)
    xb = oracle.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w = (rng.standard_normal((N, K)) * 0.02).astype(np.float32)
    bias = (rng.standard_normal(N) * 0.5).astype(np.float32)
    x = bf16_tensor(xb, cuda)
    if w_bf16:
        wb = oracle.f32_to_bf16(w)
        w = oracle.bf16_to_f32(wb)
        w_dev = bf16_tensor(wb, cuda)
    else:
        w_dev = torch.from_numpy(w).to(cuda)
    rp = Kn.router_prepare(w_dev, planes)
    out = torch.full((M, N + 1), float("nan"), dtype=torch.float32, device=cuda)
    Kn.router_logits_wmma(x, rp, torch.from_numpy(bias).to(cuda), out)
    torch.cuda.synchronize()
    Kn.check_dense_status("router_logits_wmma")
    want = logits_f64(oracle, xb, w, bias)
    got = out.cpu().numpy()
    assert np.all(np.isnan(got[:, N:]))
    tol = 3e-5 if planes != 2 else 6e-5
    assert np.max(np.abs(got[:, :N] - want)) <= tol * np.max(np.abs(want)), np.max(np.abs(got[:, :N] - want)) / np.max(np.abs(want))
    if w_bf16 and planes == 1:  # the unprepared BF16 weight as its own plane
        out2 = torch.empty((M, N), dtype=torch.float32, device=cuda)
        Kn.router_logits_wmma(x, Kn.RouterPlanes(w_dev.view(torch.int16), 1, N, K), None, out2)
        plain = logits_f64(oracle, xb, w, np.zeros(N, np.float32))
        assert np.max(np.abs(out2.cpu().numpy() - plain)) <= 1e-5 * np.max(np.abs(plain))


@pytest.mark.parametrize("M,E,k,shards", [(16, 512, 10, 1), (64, 512, 10, 1), (7, 64, 4, 1), (200, 1000, 10, 1), (16, 512, 10, 4)])
def test_route_small_equals_router_then_pack(cuda, M, E, k, shards):
    """sxb_moe_route_small writes the same ids, coef and workspace, word for word, as moe_router + moe_group_routes[_ep]."""
    from strixite_b200 import kernels as Kn
    g = torch.Generator(device="cpu").manual_seed(M * 31 + E)
    logits = torch.randn((M, E + 1), generator=g).to(cuda)
    logits[0, :4] = 0.5  # ties
    E_local = E // shards
    e_lo = E_local * (shards - 1)
    nbytes = Kn.moe_route_workspace_bytes(M, k, E_local)
    outs = []
    for fused in (False, True):
        ids = torch.full((M, k), -7, dtype=torch.int32, device=cuda)
        coef = torch.zeros((M, k), dtype=torch.float32, device=cuda)
        ws = torch.zeros(nbytes // 4, dtype=torch.int32, device=cuda)
        e1, e2 = torch.zeros(4, dtype=torch.int32, device=cuda), torch.zeros(4, dtype=torch.int32, device=cuda)
        if fused:
            Kn.moe_route_small(logits, E + 1, M, E, k, e_lo if shards > 1 else 0, E_local, ids, coef, ws, nbytes, e1, e2)
        else:
            Kn.moe_router(logits, E + 1, M, E, k, None, 1, 0, ids, coef, Kn.Act.F32, e1)
            if shards > 1:
                Kn.moe_group_routes_ep(ids, M, k, E, e_lo, E_local, ws, nbytes, e2)
            else:
                Kn.moe_group_routes(ids, M, k, E, ws, nbytes, e2)
        torch.cuda.synchronize()
        outs.append((ids.cpu(), coef.cpu(), ws.cpu(), e1.cpu(), e2.cpu()))
    for a, b in zip(*outs):
        assert torch.equal(a, b)


def test_route_small_reports_a_bad_logit(cuda):
    from strixite_b200 import kernels as Kn
    logits = torch.zeros((4, 65), device=cuda)
    logits[2, 9] = float("inf")
    ids = torch.zeros((4, 4), dtype=torch.int32, device=cuda)
    coef = torch.zeros((4, 4), device=cuda)
    nbytes = Kn.moe_route_workspace_bytes(4, 4, 64)
    ws = torch.zeros(nbytes // 4, dtype=torch.int32, device=cuda)
    e1, e2 = torch.zeros(4, dtype=torch.int32, device=cuda), torch.zeros(4, dtype=torch.int32, device=cuda)
    Kn.moe_route_small(logits, 65, 4, 64, 4, 0, 64, ids, coef, ws, nbytes, e1, e2)
    torch.cuda.synchronize()
    assert e1.tolist()[:3] == [1, 2, 9] and ids[2].tolist() == [-1] * 4
    assert e2.tolist()[0] == 1  # the pack sees the token's ids of -1 as out of range


@pytest.mark.parametrize("M,N,K,planes", [(1, 1, 64, 3), (129, 17, 128, 2), (150, 513, 256, 3), (640, 255, 192, 1), (777, 513, 512, 3), (1200, 513, 128, 3),
                                           (4096, 513, 64, 3), (60001, 16, 64, 2), (40000, 300, 64, 1)])
def test_router_logits_tcgen05_tiles(cuda, M, N, K, planes):
    """Tiles of every width that the launch picks, ragged last tiles on both sides, several tiles a CTA (both accumulators, several turns).
    FP32 sums of exact products: K P of them, each off by 2^-23 of the largest partial sum at most; two planes hold 16 bits of a weight."""
    from strixite_b200 import kernels as Kn
    g = torch.Generator(device="cpu").manual_seed(M + N)
    x = torch.randn((M, K), generator=g).to(torch.bfloat16).to(cuda)
    w = (torch.randn((N, K), generator=g) * 0.02).to(cuda)
    if planes == 1:
        w = w.to(torch.bfloat16)
    bias = torch.randn(N, generator=g).to(cuda)
    out = torch.full((M, N + 3), float("nan"), device=cuda)
    Kn.router_logits_wmma(x, Kn.router_prepare(w, planes), bias, out)
    torch.cuda.synchronize()
    Kn.check_dense_status("router_logits_wmma")
    want = x.double() @ w.double().T + bias.double()
    size = x.double().abs() @ w.double().abs().T + bias.double().abs()
    bound = size * (K * planes * 2.0 ** -23 + (2.0 ** -16 if planes == 2 else 0)) + 1e-7
    assert torch.isnan(out[:, N:]).all() and ((out[:, :N].double() - want).abs() <= bound).all()


@pytest.mark.parametrize("M,K,bits", [(19000, 64 * 17, 8), (19000, 64 * 17, 4), (10001, 64 * 32, 8), (33, 64 * 40, 4), (32, 64, 8)])
def test_staged_tiles_cut_by_k(cuda, M, K, bits):
    """Tile-blocked activations of a dense projection, word for word, where the launch cuts k into ranges: one block past a range, two
    whole ranges, and few rows."""
    from strixite_b200 import kernels as Kn
    x = torch.randn((M, K), generator=torch.Generator(device="cpu").manual_seed(K)).to(torch.bfloat16).to(cuda)
    xs = torch.full((M, K), -1, dtype=torch.int16, device=cuda)
    Kn.stage_f16_tiles(x, None, 0, M, 1, 1, K, bits, xs)
    v = x.to(torch.float16).view(M, K // 64, 8, 8)  # [row, 64-k block, 16-byte chunk, element]
    if bits == 4:
        v = v[..., [0, 4, 1, 5, 2, 6, 3, 7]]
    chunk = torch.arange(8, device=cuda)[None, :] ^ (torch.arange(M, device=cuda)[:, None] & 7)  # chunk c of row r lies at place c ^ r % 8
    v = torch.gather(v, 2, chunk[:, None, :, None].expand(M, K // 64, 8, 8))
    assert torch.equal(xs.view(K // 64, M, 64), v.permute(1, 0, 2, 3).reshape(K // 64, M, 64).contiguous().view(torch.int16))


@pytest.mark.parametrize("ydt", [torch.float32, torch.bfloat16])
def test_residual_add(cuda, ydt):
    from strixite_b200 import kernels as Kn
    g = torch.Generator(device="cpu").manual_seed(3)
    x = torch.randn((33, 1024), generator=g).to(torch.bfloat16).to(cuda)
    y = torch.randn((33, 1024), generator=g).to(ydt).to(cuda)
    out = torch.empty_like(x)
    Kn.residual_add(x, y, out)
    assert torch.equal(out, (x.float() + y.float()).to(torch.bfloat16))
    Kn.residual_add(x, y, x)  # in place
    assert torch.equal(x, out)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_hc_inject(cuda, oracle, dt):
    """kernels/hc.hpp:52-54 against the oracle's injection (the one inside moe_shared_add_inject, with s = 0 and a gate that
    does not matter), bit for bit."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(9)
    T, d, H = 7, 320, 4
    y = rng.standard_normal((T, d)).astype(np.float32)
    x = rng.standard_normal((T, H * d)).astype(np.float32)
    w_in = (rng.random((T, H)) * 2).astype(np.float32)
    if dt == torch.bfloat16:
        yb, xb = oracle.f32_to_bf16(y), oracle.f32_to_bf16(x)
        _, want = oracle.moe_shared_add_inject(yb, np.zeros_like(yb), np.zeros(T, np.float32), 0, xb, w_in)
        xd, yd = bf16_tensor(xb, cuda), bf16_tensor(yb, cuda)
    else:
        _, want = oracle.moe_shared_add_inject(y, np.zeros_like(y), np.zeros(T, np.float32), 0, x, w_in)
        xd, yd = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
    Kn.hc_inject(xd, torch.from_numpy(w_in).to(cuda), yd, T, H, d, Kn.Act.F32 if dt == torch.float32 else Kn.Act.BF16)
    got = xd.cpu().numpy() if dt == torch.float32 else bits_of(xd)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("bits,G,M,N,K", [(8, 64, 300, 2048, 1024), (4, 128, 129, 512, 2048), (8, 64, 5, 256, 256)])
def test_dense_tcgen05_projections(cuda, oracle, bits, G, M, N, K):
    """linear_q*_wmma: y = x W^T with the matrix-unit numerics, against oracle.linear_q(w_f16); then the fused SwiGLU form
    feeding a down projection in the tile-blocked layout (the prefill shared expert's launch sequence)."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(bits * 100 + M)
    wq = oracle.quantize(random_weights(rng, N, K), G, bits)
    xb = oracle.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w, x = upload(wq, cuda), bf16_tensor(xb, cuda)
    want = oracle.linear_q(xb, wq, out_act=oracle.F32, w_f16=True)
    y32 = torch.empty((M, N), dtype=torch.float32, device=cuda)
    ybf = torch.empty((M, N), dtype=torch.bfloat16, device=cuda)
    Kn.linear_qw_wmma(x, w, y32, M, Kn.Act.BF16, Kn.Act.F32)
    Kn.linear_qw_wmma(x, w, ybf, M, Kn.Act.BF16, Kn.Act.BF16)
    torch.cuda.synchronize()
    Kn.check_dense_status("linear_wmma")
    assert max_abs_over_rms(y32.cpu().numpy(), want) <= 2e-5
    assert torch.equal(ybf, y32.to(torch.bfloat16))
    # staged input gives the same bits
    xs = torch.empty((M, K), dtype=torch.float16, device=cuda)
    Kn.stage_f16_tiles(x, None, 0, M, 1, 1, K, bits, xs)
    y2 = torch.empty_like(y32)
    Kn.linear_qw_wmma(xs, w, y2, M, Kn.Act.F16_TILED, Kn.Act.F32)
    assert torch.equal(y2, y32)
    # [gate | up] -> h (tile-blocked) -> down
    I = N // 2
    dq = oracle.quantize(random_weights(rng, 256, I), 64, 8)
    dn = upload(dq, cuda)
    h = torch.empty((M, I), dtype=torch.bfloat16, device=cuda)
    Kn.linear_qw_wmma_swiglu(xs, w, h, M, Kn.Act.F16_TILED, h_f16=4)
    s32 = torch.empty((M, 256), dtype=torch.float32, device=cuda)
    Kn.linear_qw_wmma(h, dn, s32, M, Kn.Act.F16_TILED, Kn.Act.F32)
    torch.cuda.synchronize()
    Kn.check_dense_status("linear_wmma_swiglu")
    zero = np.zeros((M, 1), dtype=np.int32)
    hs = oracle.experts_gather(xb, wq, 1, zero, swiglu_mode=2, w_f16=True)[:, 0]
    want_s = oracle.linear_q(hs, dq, out_act=oracle.F32, w_f16=True)
    assert max_abs_over_rms(s32.cpu().numpy(), want_s) <= 1e-2


@pytest.mark.parametrize("bits,G,M,N,K", [(8, 64, 300, 400, 256), (4, 128, 300, 400, 2048), (4, 32, 193, 144, 2048)])
def test_dense_tcgen05_partial_row_blocks(cuda, oracle, bits, G, M, N, K):
    """Tile-blocked activations into a weight whose row count is not a multiple of the 128-row work item, with token counts
    that leave a partly filled last tile - on both shapes of the kernel for tile-blocked activations (K below and from 2048).
    A store for a row past N would land in the next token's output row, so the comparison sees it."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(bits + M + N)
    wq = oracle.quantize(random_weights(rng, N, K), G, bits)
    xb = oracle.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w, x = upload(wq, cuda), bf16_tensor(xb, cuda)
    xs = torch.empty((M, K), dtype=torch.float16, device=cuda)
    Kn.stage_f16_tiles(x, None, 0, M, 1, 1, K, bits, xs)
    y32 = torch.full((M + 1, N), 7.0, dtype=torch.float32, device=cuda)
    ybf = torch.empty((M, N), dtype=torch.bfloat16, device=cuda)
    Kn.linear_qw_wmma(xs, w, y32, M, Kn.Act.F16_TILED, Kn.Act.F32)
    Kn.linear_qw_wmma(xs, w, ybf, M, Kn.Act.F16_TILED, Kn.Act.BF16)
    torch.cuda.synchronize()
    Kn.check_dense_status("partial row blocks")
    want = oracle.linear_q(xb, wq, out_act=oracle.F32, w_f16=True)
    assert max_abs_over_rms(y32[:M].cpu().numpy(), want) <= 2e-5
    assert torch.all(y32[M] == 7.0)  # nothing past the last token's row
    assert torch.equal(ybf, y32[:M].to(torch.bfloat16))


@pytest.mark.parametrize("bits,G", [(4, 32), (4, 64), (4, 128), (8, 32), (8, 64), (8, 128)])
@pytest.mark.parametrize("K", [128, 384, 1152])
def test_dense_tcgen05_scale_alignment(cuda, oracle, bits, G, K):
    """Contractions of 1, 3 and 9 steps of 128 - fewer than the producers' sets, and no multiple of them - with scales and mins that start
    on any 2-byte boundary: the vector loads' groups and those read one by one give the same bits."""
    from dataclasses import replace
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(bits + G + K)
    M, N = 140, 200
    wq = oracle.quantize(random_weights(rng, N, K), G, bits)
    xb = oracle.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w, x = upload(wq, cuda), bf16_tensor(xb, cuda)
    want = oracle.linear_q(xb, wq, out_act=oracle.F32, w_f16=True)
    ys = []
    for off in (0, 1, 2):
        moved = [torch.cat([v.new_zeros(8 + off), v.reshape(-1)])[8 + off:] for v in (w.scale, w.minv)]
        y = torch.empty((M, N), dtype=torch.float32, device=cuda)
        Kn.linear_qw_wmma(x, replace(w, scale=moved[0], minv=moved[1]), y, M, Kn.Act.BF16, Kn.Act.F32)
        ys.append(y)
    torch.cuda.synchronize()
    Kn.check_dense_status("scale alignment")
    assert max_abs_over_rms(ys[0].cpu().numpy(), want) <= 2e-5
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])


@pytest.mark.parametrize("way", ["staged", "captured"])
@pytest.mark.parametrize("bits,G,M,N,K", [(4, 128, 64, 4104, 2048), (8, 64, 127, 4104, 512), (4, 64, 129, 24, 256), (8, 128, 1001, 136, 256)])
def test_dense_tcgen05_rows_in_eights(cuda, oracle, monkeypatch, way, bits, G, M, N, K):
    """Weights whose row count is a multiple of 8 and not of 16, on both kernels: the last row block ends inside a 16-row piece of
    tensor memory; nothing is stored past the last row."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(M + N)
    wq = oracle.quantize(random_weights(rng, N, K), G, bits)
    xb = oracle.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w, x = upload(wq, cuda), bf16_tensor(xb, cuda)
    y32 = torch.full((M + 1, N), 7.0, dtype=torch.float32, device=cuda)
    ybf = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device=cuda)
    if way == "captured":
        capture_calls(monkeypatch)
    Kn.linear_qw_wmma(x, w, y32, M, Kn.Act.BF16, Kn.Act.F32)
    Kn.linear_qw_wmma(x, w, ybf, M, Kn.Act.BF16, Kn.Act.BF16)
    torch.cuda.synchronize()
    Kn.check_dense_status("rows in eights")
    assert max_abs_over_rms(y32[:M].cpu().numpy(), oracle.linear_q(xb, wq, out_act=oracle.F32, w_f16=True)) <= 2e-5
    assert torch.all(y32[M] == 7.0) and torch.all(ybf[M] == 7.0) and torch.equal(ybf[:M], y32[:M].to(torch.bfloat16))


@pytest.mark.parametrize("spread", [0, 6, 7, 9, 12])
@pytest.mark.parametrize("bits,G,K", [(4, 128, 1024), (8, 64, 1024), (4, 32, 384), (8, 128, 640)])
def test_dense_tcgen05_spread_scales(cuda, oracle, bits, G, K, spread):
    """Rows whose groups' scales lie up to 2^spread apart, against activations that meet the small groups only (large weight
    columns and small activations, as activation-scaling quantizers make them).  Row blocks of every kind: all rows spread, one
    row of a block, rows of small weights throughout, a constant group, an all-zero group.  The dots are no further from 64 bits than
    with every weight rounded once to F16 at its natural magnitude (2e-6: FP32 sums)."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(bits + K + spread)
    N, M = 400, 40
    W = random_weights(rng, N, K)
    W[:128, K // 2:] *= 2.0 ** spread
    W[130, K // 2:] *= 2.0 ** spread
    W[256:384] *= 2.0 ** -spread
    W[256:384, K // 2:] *= 2.0 ** spread
    W[3, :G], W[4, :G], W[131, :G] = 0.0, 0.01, 0.0
    wq = oracle.quantize(W, G, bits)
    x = rng.standard_normal((M, K)).astype(np.float32)
    x[:, K // 2:] = 0.0
    xb = oracle.f32_to_bf16(x)
    y = torch.empty((M, N), dtype=torch.float32, device=cuda)
    Kn.linear_qw_wmma(bf16_tensor(xb, cuda), upload(wq, cuda), y, M, Kn.Act.BF16, Kn.Act.F32)
    torch.cuda.synchronize()
    Kn.check_dense_status("spread scales")
    exact = oracle.bf16_to_f32(xb).astype(np.float64) @ oracle.affine_weights(wq).T
    natural = oracle.linear_q(xb, wq, out_act=oracle.F32, w_f16=True)
    got = y.cpu().numpy()
    for lo, hi in ((0, 128), (128, 256), (256, 384), (384, 400)):
        size = np.linalg.norm(exact[:, lo:hi])
        off, off_natural = (np.linalg.norm(v[:, lo:hi] - exact[:, lo:hi]) / size for v in (got, natural))
        assert off <= 1.05 * off_natural + 2e-6, (lo, hi, off, off_natural)


@pytest.mark.parametrize("bits,G", [(4, 128), (8, 64)])
def test_fp32_activations(cuda, oracle, bits, G):
    """Act::F32 into the dense, per-slot and grouped entry points (kernels/linear_q4.hpp:26-30): FP32 in, FP32 out,
    against the oracle's FP32 mode."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(bits)
    E, N, K, M, A = 6, 64, 256, 9, 3
    wq = oracle.quantize(random_weights(rng, E * N, K), G, bits)
    w = upload(wq, cuda)
    xf = rng.standard_normal((M, K)).astype(np.float32)
    x = torch.from_numpy(xf).to(cuda)
    ids_np = np.stack([rng.permutation(E)[:A] for _ in range(M)]).astype(np.int32)
    ids = torch.from_numpy(ids_np).to(cuda)
    err = torch.zeros(4, dtype=torch.int32, device=cuda)
    tol = 2e-5
    # dense: the stacked matrix as one [E*N, K] weight
    y = torch.empty((M, E * N), dtype=torch.float32, device=cuda)
    Kn.linear_qw(x, w, y, M, Kn.Act.F32)
    assert max_abs_over_rms(y.cpu().numpy(), oracle.linear_q(xf, wq)) <= tol
    # per-slot gather, SwiGLU gather, combine
    g = torch.empty((M, A, N), dtype=torch.float32, device=cuda)
    Kn.linear_qw_experts_gather(x, w, E, ids, M, A, g, Kn.Act.F32, err)
    assert max_abs_over_rms(g.cpu().numpy(), oracle.experts_gather(xf, wq, E, ids_np)) <= tol
    hh = torch.empty((M, A, N // 2), dtype=torch.float32, device=cuda)
    Kn.linear_qw_experts_gather_swiglu(x, w, E, ids, M, A, hh, Kn.Act.F32, err)
    assert max_abs_over_rms(hh.cpu().numpy(), oracle.experts_gather(xf, wq, E, ids_np, swiglu_mode=1)) <= tol
    dq = oracle.quantize(random_weights(rng, E * 32, N), 32, bits)
    dn = upload(dq, cuda)
    coef_np = rng.random((M, A)).astype(np.float32)
    coef = torch.from_numpy(coef_np).to(cuda)
    yc = torch.empty((M, 32), dtype=torch.float32, device=cuda)
    Kn.linear_qw_experts_combine(g, dn, E, ids, coef, M, A, yc, Kn.Act.F32, err)
    want_c = oracle.experts_combine(g.cpu().numpy(), dq, E, ids_np, coef_np)
    assert max_abs_over_rms(yc.cpu().numpy(), want_c) <= tol
    # grouped forms (any math: FP32 activations always take the plain path)
    nbytes = Kn.moe_route_workspace_bytes(M, A, E)
    ws = torch.empty(nbytes // 4, dtype=torch.int32, device=cuda)
    Kn.moe_group_routes(ids, M, A, E, ws, nbytes, err)
    hg = torch.empty_like(hh)
    Kn.linear_qw_experts_gather_grouped_swiglu(x, w, E, ws, nbytes, M, A, hg, Kn.Act.F32, Kn.MoeMath.WmmaF16)
    assert torch.equal(hg, hh)
    partial = torch.empty((M * A, 32), dtype=torch.float32, device=cuda)
    yg = torch.empty_like(yc)
    Kn.linear_qw_experts_combine_grouped(g, dn, E, ids, coef, ws, nbytes, partial, M, A, yg, Kn.Act.F32, Kn.MoeMath.F32)
    torch.cuda.synchronize()
    assert int(err[0]) == 0
    assert max_abs_over_rms(yg.cpu().numpy(), want_c) <= tol


def test_cxx_host_runs_the_call_block(cuda, oracle, tmp_path):
    """tests/cpp/call_block.cpp, linked against libstrix_b200.so, issues the reference's call block through the C++ shim;
    its ids, coef and y equal the Python launcher sequence's bit for bit."""
    from helpers_cpp import build_call_block
    from strixite_b200 import kernels as Kn
    exe = build_call_block(tmp_path)
    rng = np.random.default_rng(11)
    M, E, A, d, I, G = 12, 8, 2, 256, 128, 64
    xb = oracle.f32_to_bf16(rng.standard_normal((M, d)).astype(np.float32))
    logits = rng.standard_normal((M, E)).astype(np.float32)
    gu = oracle.quantize(random_weights(rng, E * 2 * I, d), G, 4)
    dn = oracle.quantize(random_weights(rng, E * d, I), G, 4)
    with open(tmp_path / "in.bin", "wb") as f:
        f.write(np.array([M, E, A, d, I, G, G], dtype=np.int64).tobytes())
        for a in (xb, logits, gu.q, gu.scale, gu.minv, dn.q, dn.scale, dn.minv):
            f.write(np.ascontiguousarray(a).tobytes())
    subprocess.run([str(exe), str(tmp_path / "in.bin"), str(tmp_path / "out.bin")], check=True, timeout=120)
    raw = (tmp_path / "out.bin").read_bytes()
    ids_c = np.frombuffer(raw[: M * A * 4], dtype=np.int32).reshape(M, A)
    coef_c = np.frombuffer(raw[M * A * 4: 2 * M * A * 4], dtype=np.float32).reshape(M, A)
    y_c = np.frombuffer(raw[2 * M * A * 4:], dtype=np.uint16).reshape(M, d)
    # the same launchers from Python
    x, lg = bf16_tensor(xb, cuda), torch.from_numpy(logits).to(cuda)
    wg, wd = upload(gu, cuda), upload(dn, cuda)
    ids = torch.empty((M, A), dtype=torch.int32, device=cuda)
    coef = torch.empty((M, A), dtype=torch.float32, device=cuda)
    err = torch.zeros(8, dtype=torch.int32, device=cuda)
    nbytes = Kn.moe_route_workspace_bytes(M, A, E)
    ws = torch.empty(nbytes // 4, dtype=torch.int32, device=cuda)
    h = torch.empty((M * A, I), dtype=torch.bfloat16, device=cuda)
    partial = torch.empty((M * A, d), dtype=torch.float32, device=cuda)
    y = torch.empty((M, d), dtype=torch.bfloat16, device=cuda)
    Kn.moe_router(lg, E, M, E, A, None, 1, 0, ids, coef, Kn.Act.F32, err)
    Kn.moe_group_routes(ids, M, A, E, ws, nbytes, err[4:])
    Kn.linear_qw_experts_gather_grouped_swiglu(x, wg, E, ws, nbytes, M, A, h, Kn.Act.BF16, Kn.MoeMath.F32)
    Kn.linear_qw_experts_combine_grouped(h, wd, E, ids, coef, ws, nbytes, partial, M, A, y, Kn.Act.BF16, Kn.MoeMath.F32)
    torch.cuda.synchronize()
    assert np.array_equal(ids_c, ids.cpu().numpy())
    assert np.array_equal(coef_c.view(np.uint32), coef.cpu().numpy().view(np.uint32))
    assert np.array_equal(y_c, bits_of(y))
    # and the oracle agrees with both
    ref = oracle.moe_layer(xb, np.concatenate([logits, np.zeros((M, 1), np.float32)], axis=1), oracle.LayerWeights(gu, dn), E, A)
    assert np.array_equal(ref["ids"], ids_c)


@pytest.mark.parametrize("tiled", [False, True])
def test_a_wait_that_runs_out_ends_the_kernel_with_a_status(cuda, oracle, lib, tiled):
    """The tcgen05 kernels (tiled: the one for tile-blocked activations) bound every device-side wait.  With the limit set to 2 ms and CTA 0 told to leave one fill of its
    weight-code ring out (nothing is issued for it, so nothing can fault), the producers' wait for those codes runs out:
    the kernel returns, the status words name the work item and the role, tensor memory is released - a normal launch on
    the same context right after gives the right answer."""
    from strixite_b200 import kernels as Kn
    rng = np.random.default_rng(5)
    M, N, K = 200, 512, 1024
    wq = oracle.quantize(random_weights(rng, N, K), 64, 8)
    xb = oracle.f32_to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w, x = upload(wq, cuda), bf16_tensor(xb, cuda)
    y = torch.empty((M, N), dtype=torch.float32, device=cuda)
    act = Kn.Act.BF16
    if tiled:
        xs = torch.empty((M, K), dtype=torch.float16, device=cuda)
        Kn.stage_f16_tiles(x, None, 0, M, 1, 1, K, 8, xs)
        x, act = xs, Kn.Act.F16_TILED
    Kn.linear_qw_wmma(x, w, y, M, act, Kn.Act.F32)  # warm: module loaded, attributes set
    torch.cuda.synchronize()
    Kn.check_dense_status("warm-up")
    try:
        Kn.set_wait_limit(2_000_000)
        assert lib.sxb_test_skip_ring_slot(3) == 0
        Kn.linear_qw_wmma(x, w, y, M, act, Kn.Act.F32)
        torch.cuda.synchronize()
    finally:
        lib.sxb_test_skip_ring_slot(-1)
        Kn.set_wait_limit(2_000_000_000)
    # which role's limit fires first is a matter of microseconds (every role of the stalled CTA is waiting): any of them
    with pytest.raises(Kn.Error, match=r"a tcgen05 kernel gave up a wait at work item 0 \((a weight producer|an MMA warp|the epilogue|the activation copy|the weight-code copy)"):
        Kn.check_dense_status("skipped fill")
    Kn.check_dense_status("cleared by the read")  # the words are cleared by the failing check
    y2 = torch.empty_like(y)
    Kn.linear_qw_wmma(x, w, y2, M, act, Kn.Act.F32)
    torch.cuda.synchronize()
    Kn.check_dense_status("after")
    want = oracle.linear_q(xb, wq, out_act=oracle.F32, w_f16=True)
    assert max_abs_over_rms(y2.cpu().numpy(), want) <= 2e-5


@pytest.mark.parametrize("M,N,K,planes,slot", [(150, 513, 512, 3, 0), (150, 513, 512, 3, 6), (40000, 300, 64, 1, 1), (1200, 513, 2048, 2, 9)])
def test_router_gemm_gives_up_a_wait(cuda, lib, M, N, K, planes, slot):
    """The router-logits GEMM with CTA 0 told to leave one stage fill out: in its first item, behind a full turn of the stages and in its second item.
    The kernel returns, the status names the role, the next call has the bits of the call before."""
    from strixite_b200 import kernels as Kn
    g = torch.Generator(device="cpu").manual_seed(M)
    x, w = torch.randn((M, K), generator=g).to(torch.bfloat16).to(cuda), (torch.randn((N, K), generator=g) * 0.02).to(cuda)
    planes_ = Kn.router_prepare(w.to(torch.bfloat16) if planes == 1 else w, planes)
    out = [torch.full((M, N), float("nan"), device=cuda) for _ in range(3)]
    Kn.router_logits_wmma(x, planes_, None, out[0])
    Kn.check_dense_status("warm-up")
    try:
        Kn.set_wait_limit(2_000_000)
        assert lib.sxb_test_skip_ring_slot(slot) == 0
        Kn.router_logits_wmma(x, planes_, None, out[1])
        torch.cuda.synchronize()
    finally:
        lib.sxb_test_skip_ring_slot(-1)
        Kn.set_wait_limit(2_000_000_000)
    with pytest.raises(Kn.Error, match=r"skipped fill: a tcgen05 kernel gave up a wait at work item \d+ \((an MMA warp|the epilogue|the activation copy)"):
        Kn.check_dense_status("skipped fill")
    Kn.router_logits_wmma(x, planes_, None, out[2])
    Kn.check_dense_status("after")
    assert torch.equal(out[2], out[0]) and not bool(torch.isnan(out[2]).any())


# (slot, item that it belongs to): in the first turn of the ring of codes, behind a full turn, and in a later item, so that the item warp stands at a place for scales.
# Eight groups (four places for scales), thirty-two (two), forty (the producers load scales themselves).
@pytest.mark.parametrize("bits,N,K,slot", [(4, 32768, 1024, 3), (4, 32768, 1024, 11), (4, 32768, 1024, 45), (4, 32768, 4096, 5), (4, 32768, 4096, 130), (8, 32768, 512, 22),
                                           (8, 32768, 2048, 60), (4, 32768, 5120, 13), (4, 32768, 5120, 130)])
def test_a_wait_that_runs_out_in_a_later_item(cuda, lib, bits, N, K, slot):
    """The kernel for tile-blocked activations with several items a CTA and CTA 0 told to leave one fill of its ring of codes out.  The kernel returns, the status names item and
    role, the next call has the bits of the call before."""
    from strixite_b200 import kernels as Kn
    M, g = 512, torch.Generator(device="cuda").manual_seed(slot)
    w = Kn.quantize(torch.randn((N, K), generator=g, device=cuda) * 0.05, 128 if bits == 4 else 64, bits)
    x = torch.randn((M, K), generator=g, device=cuda).to(torch.bfloat16)
    xs, out = torch.empty((M, K), dtype=torch.float16, device=cuda), [torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=cuda) for _ in range(3)]
    Kn.stage_f16_tiles(x, None, 0, M, 1, 1, K, bits, xs)
    Kn.linear_qw_wmma(xs, w, out[0], M, Kn.Act.F16_TILED)
    Kn.check_dense_status("warm-up")
    try:
        Kn.set_wait_limit(2_000_000)
        assert lib.sxb_test_skip_ring_slot(slot) == 0
        Kn.linear_qw_wmma(xs, w, out[1], M, Kn.Act.F16_TILED)
        torch.cuda.synchronize()
    finally:
        lib.sxb_test_skip_ring_slot(-1)
        Kn.set_wait_limit(2_000_000_000)
    # items of CTA 0, of which any role's wait may run out first: the skipped step's, one before it and up to four ahead
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    item = sms * (slot // (K // 128))
    with pytest.raises(Kn.Error, match=r"skipped fill: a tcgen05 kernel gave up a wait at work item \d+ \((a weight producer|an MMA warp|the epilogue|the activation copy|the weight-code copy|a warp waiting for the description|the work-item)") as e:
        Kn.check_dense_status("skipped fill")
    at = int(re.search(r"work item (\d+)", str(e.value)).group(1))
    assert at in range(max(item - sms, 0), item + 5 * sms, sms), (at, item)
    Kn.linear_qw_wmma(xs, w, out[2], M, Kn.Act.F16_TILED)
    Kn.check_dense_status("after")
    assert torch.equal(out[2].view(torch.int16), out[0].view(torch.int16)) and not bool(torch.isnan(out[2]).any())


@pytest.mark.parametrize("bits,G,M,N,K", [(8, 64, 777, 4096, 1024), (4, 128, 300, 2048, 4096), (4, 32, 150, 4096, 1024), (8, 64, 200, 2560, 1536), (8, 128, 129, 4112, 4096), (4, 128, 1001, 1040, 768)])
def test_dense_tiles_of_fewer_rows(cuda, bits, G, M, N, K):
    """Tiles of 64 to 112 rows, the last one ragged, with scales in shared memory (and, at six groups, without): FP32, BF16 and gate/up rows, bit for bit the general kernel's,
    which a captured call runs on."""
    from strixite_b200 import kernels as Kn
    g = torch.Generator(device="cuda").manual_seed(M)
    w = Kn.quantize(torch.randn((N, K), generator=g, device=cuda) * 0.05, G, bits)
    x = torch.randn((M, K), generator=g, device=cuda).to(torch.bfloat16)
    forms = [(torch.float32, N, lambda y: Kn.linear_qw_wmma(x, w, y, M, Kn.Act.BF16, Kn.Act.F32)), (torch.bfloat16, N, lambda y: Kn.linear_qw_wmma(x, w, y, M, Kn.Act.BF16))]
    forms += [(torch.bfloat16, N // 2, lambda y: Kn.linear_qw_wmma_swiglu(x, w, y, M, Kn.Act.BF16))]
    for dtype, cols, call in forms:
        y = [torch.full((M + 1, cols), 77.0, dtype=dtype, device=cuda) for _ in range(2)]
        call(y[0])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call(y[1])
        graph.replay()
        torch.cuda.synchronize()
        Kn.check_dense_status("tiles of fewer rows")
        assert torch.equal(y[0].view(torch.uint8), y[1].view(torch.uint8)) and not bool(torch.isnan(y[0]).any())


def test_dense_tcgen05_captured(cuda, oracle, lib, monkeypatch):
    """The dense forms, spread scales and a wait that runs out, on the kernel that captured calls take (no scratch)."""
    graphs = capture_calls(monkeypatch)
    test_dense_tcgen05_projections(cuda, oracle, 8, 64, 300, 2048, 1024)
    test_dense_tcgen05_projections(cuda, oracle, 4, 128, 129, 512, 2048)
    for spread in (0, 7, 12):
        test_dense_tcgen05_spread_scales(cuda, oracle, 4, 128, 1024, spread)
        test_dense_tcgen05_spread_scales(cuda, oracle, 8, 64, 1024, spread)
    test_a_wait_that_runs_out_ends_the_kernel_with_a_status(cuda, oracle, lib, False)
    assert graphs
