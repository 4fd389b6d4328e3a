"""The hyper-connection mix either side of the MoE block (kernels/hc.hpp:36-54) against the float64 oracle, through the
C ABI: hc_mix_down, hc_mix_up (chunk-major weight) and the device-side chunk-major re-layout."""
import numpy as np
import pytest
import torch

from helpers import bf16_tensor, bits_of, max_abs_over_rms, random_weights, upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,G", [(4, 64), (8, 128), (4, 32)])
def test_to_chunk_major_on_the_device(cuda, oracle, bits, G):
    """sxb_to_chunk_major equals the host re-layout, which test_oracle pins to the reference's own to_chunk_major."""
    from strixite_b200 import kernels as K
    rng = np.random.default_rng(bits + G)
    wq = oracle.quantize(random_weights(rng, 1300, 320), G if 320 % G == 0 else 64, bits)
    cm = K.to_chunk_major(upload(wq, cuda))
    want = oracle.to_chunk_major(wq)
    assert np.array_equal(cm.q.cpu().numpy().reshape(-1), want.q.reshape(-1))
    assert np.array_equal(cm.scale.cpu().numpy().view(np.uint16).reshape(-1), want.scale.reshape(-1))
    assert np.array_equal(cm.minv.cpu().numpy().view(np.uint16).reshape(-1), want.minv.reshape(-1))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,G,T,d,r,inject", [(4, 64, 1, 256, 64, True), (8, 128, 5, 512, 96, True), (4, 128, 16, 1024, 320, True),
                                                  (8, 64, 37, 256, 32, False), (4, 32, 300, 128, 64, True)])
def test_hc_mix(cuda, oracle, dt, bits, G, T, d, r, inject):
    """hc_mix_down then hc_mix_up, each against the oracle on the same inputs: h, w_in and inv within FP32 summation noise of the
    float64 values, u within it (F32 streams) or within one BF16 rounding of it (BF16 streams)."""
    from strixite_b200 import kernels as K
    H, eps = 4, 1e-6
    rng = np.random.default_rng(T * 7 + d + bits)
    R = r + (H if inject else 0)
    wd = oracle.quantize(random_weights(rng, R, H * d, std=0.05), G, bits)
    wu = oracle.quantize(random_weights(rng, H * d, r, std=0.2), 32 if r % G else G, bits)
    norm_w = (rng.standard_normal(H * d) * 0.1).astype(np.float32)
    x = (rng.standard_normal((T, H * d)) * np.repeat(rng.random((T, H)) * 3 + 0.2, d, axis=1)).astype(np.float32)  # streams of different RMS
    if dt == torch.bfloat16:
        xb = oracle.f32_to_bf16(x)
        x = oracle.bf16_to_f32(xb)
        xd, act = bf16_tensor(xb, cuda), K.Act.BF16
    else:
        xd, act = torch.from_numpy(x).to(cuda), K.Act.F32
    h = torch.full((T, r), float("nan"), dtype=torch.float32, device=cuda)
    w_in = torch.full((T, H), float("nan"), dtype=torch.float32, device=cuda) if inject else None
    inv = torch.full((T, H), float("nan"), dtype=torch.float32, device=cuda)
    K.hc_mix_down(xd, upload(wd, cuda), T, H, d, r, inject, eps, h, w_in, inv, act)
    h_ref, w_in_ref, inv_ref = oracle.hc_mix_down(x, wd, H, d, r, inject, eps)
    assert max_abs_over_rms(inv.cpu().numpy(), inv_ref) <= 1e-5
    assert max_abs_over_rms(h.cpu().numpy(), h_ref) <= 1e-4
    if inject:
        assert max_abs_over_rms(w_in.cpu().numpy(), w_in_ref) <= 1e-4
    # the up half on the GPU's own h and inv (so that its error is its own)
    u = torch.empty((T, d), dtype=dt, device=cuda)
    K.hc_mix_up(h, K.to_chunk_major(upload(wu, cuda)), xd, torch.from_numpy(norm_w).to(cuda), inv, T, H, d, u, act)
    torch.cuda.synchronize()
    u_ref = oracle.hc_mix_up(h.cpu().numpy(), wu, x, norm_w, inv.cpu().numpy(), H, d)
    if dt == torch.float32:
        assert max_abs_over_rms(u.cpu().numpy(), u_ref) <= 1e-4
    else:
        got = oracle.bf16_to_f32(bits_of(u)).astype(np.float64)
        assert np.all(np.abs(got - u_ref) <= 2.0 ** -8 * np.abs(u_ref) + 1e-5 * np.sqrt(np.mean(u_ref ** 2)))  # one BF16 rounding


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,G,T,d,r", [(8, 64, 8, 64, 32), (4, 32, 9, 192, 1024), (8, 32, 17, 320, 352), (4, 64, 33, 64, 64), (8, 64, 49, 2560, 320)])
def test_hc_mix_edges(cuda, oracle, dt, bits, G, T, d, r):
    """The edges of the tensor-core tiles: rows past a tile of 16, groups of 8 / 16 / 32 tokens that are full, one over, or partly filled, warps
    without a chunk (d = 64), the longest rank, an h that 16-byte loads may not read; and a token's results do not depend on its batch.
    FP32 sums of exact products: a dot of n terms, added in any order, is within n 2^-24 sum|terms| of 64 bits; the sums below are
    chains of at most 256 (MMAs of a warp, groups, warps, CTAs), so 2^-16 sum|terms| with the activation functions' few ulp."""
    from strixite_b200 import kernels as K
    H, eps = 4, 1e-6
    rng = np.random.default_rng(T * 3 + d + r)
    R = r + H
    wd = oracle.quantize(random_weights(rng, R, H * d, std=0.05), G, bits)
    wu = oracle.quantize(random_weights(rng, H * d, r, std=0.2), 32 if r % G else G, bits)
    norm_w = (rng.standard_normal(H * d) * 0.1).astype(np.float32)
    x = (rng.standard_normal((T, H * d)) * np.repeat(rng.random((T, H)) * 3 + 0.2, d, axis=1)).astype(np.float32)
    act = K.Act.F32
    xd = torch.from_numpy(x).to(cuda)
    if dt == torch.bfloat16:
        xd, act = xd.to(torch.bfloat16), K.Act.BF16
        x = xd.float().cpu().numpy()
    wdd, wud, nw = upload(wd, cuda), K.to_chunk_major(upload(wu, cuda)), torch.from_numpy(norm_w).to(cuda)

    def mix(xt):
        n = xt.shape[0]
        h = torch.full((n * r + 1,), float("nan"), dtype=torch.float32, device=cuda)[1:].view(n, r)  # 4-byte aligned
        w_in, inv = (torch.full((n, H), float("nan"), dtype=torch.float32, device=cuda) for _ in range(2))
        u = torch.empty((n, d), dtype=dt, device=cuda)
        K.hc_mix_down(xt, wdd, n, H, d, r, True, eps, h, w_in, inv, act)
        K.hc_mix_up(h, wud, xt, nw, inv, n, H, d, u, act)
        return h, w_in, inv, u

    h, w_in, inv, u = mix(xd)
    h_ref, w_in_ref, inv_ref = oracle.hc_mix_down(x, wd, H, d, r, True, eps)
    assert np.max(np.abs(inv.cpu().numpy() / inv_ref - 1)) <= 2.0 ** -20
    terms = np.abs(x.reshape(T, H, d) * inv_ref[:, :, None]).reshape(T, H * d) @ np.abs(oracle.affine_weights(wd)).T / H
    assert np.all(np.abs(h.cpu().numpy() - h_ref) <= 2.0 ** -16 * terms[:, :r])
    assert np.all(np.abs(w_in.cpu().numpy() - w_in_ref) <= 2.0 ** -16 * terms[:, r:] + 2.0 ** -20)
    hn = h.cpu().numpy()
    u_ref = oracle.hc_mix_up(hn, wu, x, norm_w, inv.cpu().numpy(), H, d)
    z_terms = np.abs(hn) @ np.abs(oracle.affine_weights(wu)).T  # sigmoid' <= 1/4
    scale = np.abs(x * np.repeat(inv.cpu().numpy(), d, axis=1) * (1 + norm_w))
    bound = ((2.0 ** -18 * z_terms + 2.0 ** -20) * scale).reshape(T, H, d).sum(axis=1) / H + (2.0 ** -8 * np.abs(u_ref) if dt == torch.bfloat16 else 0)
    assert np.all(np.abs(u.float().cpu().numpy() - u_ref) <= bound)
    for t in (0, T - 1):
        one = mix(xd[t:t + 1])
        assert all(torch.equal(a[0], b[t]) for a, b in zip(one, (h, w_in, inv, u)))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,zero,far", [(8, 0, 20), (8, 3, 40), (8, 255, 28), (4, 0, 28), (4, 2, 20), (4, 15, 40)])
def test_hc_mix_large_value_against_zero_weights(cuda, oracle, dt, bits, zero, far):
    """An activation, and an h, 2^far times the others meets weights that are exactly zero (code `zero`, min -zero * scale): the dots are
    those of the small values, and none of their bits may go.  Bounds as in test_hc_mix_edges."""
    from strixite_b200 import kernels as K
    H, eps, T, d, r, G, at = 4, 1e-6, 17, 256, 64, 32, 37
    rng = np.random.default_rng(bits + zero + far)

    def weight(rows, cols, std):
        w = oracle.quantize(random_weights(rng, rows, cols, std=std), G, bits)
        s = np.float32(2.0 ** -9)
        w.scale[:, at // G], w.minv[:, at // G] = oracle.f32_to_bf16(s[None])[0], oracle.f32_to_bf16((-zero * s)[None])[0]
        if bits == 8:
            w.q[:, at] = zero
        else:
            low = w.q[:, at // 2] & 0x0F if at % 2 else zero
            w.q[:, at // 2] = low | ((zero if at % 2 else w.q[:, at // 2] >> 4) << 4)
        assert np.all(oracle.affine_weights(w)[:, at] == 0)
        return w

    wd, wu = weight(r + H, H * d, 0.05), weight(H * d, r, 0.2)
    x = rng.standard_normal((T, H * d)).astype(np.float32)
    x[::2, at] = 2.0 ** far
    xd, act = torch.from_numpy(x).to(cuda), K.Act.F32
    if dt == torch.bfloat16:
        xd, act = xd.to(torch.bfloat16), K.Act.BF16
        x = xd.float().cpu().numpy()
    h, w_in, inv = (torch.full((T, n), float("nan"), dtype=torch.float32, device=cuda) for n in (r, H, H))
    K.hc_mix_down(xd, upload(wd, cuda), T, H, d, r, True, eps, h, w_in, inv, act)
    h_ref, w_in_ref, inv_ref = oracle.hc_mix_down(x, wd, H, d, r, True, eps)
    terms = np.abs(x.reshape(T, H, d) * inv_ref[:, :, None]).reshape(T, H * d) @ np.abs(oracle.affine_weights(wd)).T / H
    assert np.all(np.abs(h.cpu().numpy() - h_ref) <= 2.0 ** -16 * terms[:, :r])
    assert np.all(np.abs(w_in.cpu().numpy() - w_in_ref) <= 2.0 ** -16 * terms[:, r:] + 2.0 ** -20)
    hn = rng.standard_normal((T, r)).astype(np.float32)
    hn[::2, at] = 2.0 ** far
    norm_w = (rng.standard_normal(H * d) * 0.1).astype(np.float32)
    inv1 = torch.ones((T, H), dtype=torch.float32, device=cuda)
    u = torch.empty((T, d), dtype=dt, device=cuda)
    xs = rng.standard_normal((T, H * d)).astype(np.float32)
    xsd = torch.from_numpy(xs).to(cuda).to(dt)
    xs = xsd.float().cpu().numpy()
    K.hc_mix_up(torch.from_numpy(hn).to(cuda), K.to_chunk_major(upload(wu, cuda)), xsd, torch.from_numpy(norm_w).to(cuda), inv1, T, H, d, u, act)
    u_ref = oracle.hc_mix_up(hn, wu, xs, norm_w, np.ones((T, H), dtype=np.float32), H, d)
    z_terms = np.abs(hn).astype(np.float64) @ np.abs(oracle.affine_weights(wu)).T
    bound = ((2.0 ** -18 * z_terms + 2.0 ** -20) * np.abs(xs * (1 + norm_w))).reshape(T, H, d).sum(axis=1) / H
    bound += 2.0 ** -8 * np.abs(u_ref) if dt == torch.bfloat16 else 0
    assert np.all(np.abs(u.float().cpu().numpy() - u_ref) <= bound)


@pytest.mark.parametrize("bits,T,d,r", [(8, 1, 64, 64), (8, 17, 256, 320), (4, 33, 128, 96)])
def test_hc_mix_third_plane(cuda, oracle, bits, T, d, r):
    """FP32 streams, and an FP32 h, whose last bits are all that is left of a dot: pairs 1 + 2^-8 + k 2^-23 and -(1 + 2^-8) against equal
    weights, 1 to 12 times a power of two.  With two BF16 planes (16 bits) of the pairs, every dot is zero.  Bound: the products of an MMA are
    added at its largest one's exponent, at most 3, 24 bits deep; two MMAs of 16 for each of three planes, 96 2^-21 = 5e-5 where a run of 32
    keeps 16 x 64 x 6 2^-23 = 7e-4 in the mean: an eighth of the dot."""
    from strixite_b200 import kernels as K
    H, eps, G = 4, 1e-6, 32
    rng = np.random.default_rng(T + d + r)

    def pairs(rows, cols):
        v = np.empty((rows, cols), dtype=np.float32)
        v[:, 0::2] = 1 + 2.0 ** -8 + rng.integers(1, 128, (rows, cols // 2)) * 2.0 ** -23
        v[:, 1::2] = -(1 + 2.0 ** -8)
        return v

    def weight(rows, cols, scale):
        w = oracle.quantize(random_weights(rng, rows, cols), G, bits)
        codes = np.repeat(rng.integers(4, 16, (rows, cols // 2)), 2, axis=1).astype(np.uint8)
        w.q[:] = codes if bits == 8 else codes[:, 0::2] | (codes[:, 1::2] << 4)
        w.scale[:], w.minv[:] = oracle.f32_to_bf16(np.float32([scale]))[0], oracle.f32_to_bf16(np.float32([-3 * scale]))[0]
        return w

    def cut(v):
        return (v.view(np.uint32) & 0xFFFFFF00).view(np.float32)

    wd, wu, x, hn = weight(r + H, H * d, 2.0 ** -4), weight(H * d, r, 2.0 ** 7), pairs(T, H * d), pairs(T, r)
    assert not np.any(cut(x).astype(np.float64) @ oracle.affine_weights(wd).T) and not np.any(cut(hn).astype(np.float64) @ oracle.affine_weights(wu).T)
    xd = torch.from_numpy(x).to(cuda)
    h, w_in, inv = (torch.full((T, n), float("nan"), dtype=torch.float32, device=cuda) for n in (r, H, H))
    K.hc_mix_down(xd, upload(wd, cuda), T, H, d, r, True, eps, h, w_in, inv, K.Act.F32)
    h_ref, _, inv_ref = oracle.hc_mix_down(x, wd, H, d, r, True, eps)
    assert np.all(h_ref > 0) and np.all(np.abs(h.cpu().numpy() - h_ref) <= h_ref / 8)
    ones = torch.ones((T, H), dtype=torch.float32, device=cuda)
    xs, nw, u = torch.rand((T, H * d), device=cuda) + 0.5, torch.zeros(H * d, device=cuda), torch.empty((T, d), device=cuda)
    K.hc_mix_up(torch.from_numpy(hn).to(cuda), K.to_chunk_major(upload(wu, cuda)), xs, nw, ones, T, H, d, u, K.Act.F32)
    u_ref = oracle.hc_mix_up(hn, wu, xs.cpu().numpy(), np.zeros(H * d, dtype=np.float32), np.ones((T, H), dtype=np.float32), H, d)
    z = hn.astype(np.float64) @ oracle.affine_weights(wu).T  # sigmoid' <= 1/4
    xn = xs.double().cpu().numpy()
    bound = (xn * (np.abs(z) / 32 + 2.0 ** -20)).reshape(T, H, d).sum(axis=1) / H
    assert np.all(np.abs(u.cpu().numpy() - u_ref) <= bound)
    assert np.all(np.abs(xn.reshape(T, H, d).sum(axis=1) / (2 * H) - u_ref) > bound)  # what dots of zero would give


def test_hc_mix_argument_checks(cuda, oracle):
    from strixite_b200 import kernels as K
    rng = np.random.default_rng(1)
    H, d, r, T = 4, 64, 32, 3
    wd = upload(oracle.quantize(random_weights(rng, r + H, H * d), 64, 4), cuda)
    x = torch.zeros((T, H * d), dtype=torch.bfloat16, device=cuda)
    h, w_in, inv = (torch.zeros((T, n), dtype=torch.float32, device=cuda) for n in (r, H, H))
    with pytest.raises(K.Error, match="w_in must be given exactly when inject"):
        K.hc_mix_down(x, wd, T, H, d, r, True, 1e-6, h, None, inv, K.Act.BF16)
    with pytest.raises(K.Error, match="rows, expected r"):
        K.hc_mix_down(x, wd, T, H, d, r, False, 1e-6, h, None, inv, K.Act.BF16)
    with pytest.raises(K.Error, match="streams, only 4"):
        K.hc_mix_down(x, wd, T, 2, 2 * d, r, True, 1e-6, h, w_in, inv, K.Act.BF16)
    with pytest.raises(K.Error, match="eps must be finite"):
        K.hc_mix_down(x, wd, T, H, d, r, True, 0.0, h, w_in, inv, K.Act.BF16)


def test_concurrent_calls_of_different_shared_memory(cuda, oracle):
    """Threads with a stream each may call the library at the same time.  A kernel's shared-memory limit is one for the whole process, and
    these calls of one kernel need different amounts (an up mix of rank 1024 beside one of rank 32; a dense Q4 projection of a long row
    beside a short one; a router projection of three planes beside one): every call must go through, with the result it has alone.  A
    call's own limit, set before its launch, let one up mix in 300 fail."""
    import ctypes as C
    import threading
    import time
    from strixite_b200 import _lib
    from strixite_b200 import kernels as K
    rng = np.random.default_rng(3)
    lib = _lib.load()
    H, d, T = 4, 64, 25

    def p(t):
        return C.c_void_p(t.data_ptr())

    def up(r, st):
        wu = K.to_chunk_major(upload(oracle.quantize(random_weights(rng, H * d, r, std=0.2), 32, 8), cuda))
        h, inv = torch.randn((T, r), device=cuda), torch.rand((T, H), device=cuda)
        x, nw, u = torch.randn((T, H * d), device=cuda), torch.randn(H * d, device=cuda), torch.empty((T, d), device=cuda)
        args = (p(h), C.byref(wu.c()), p(x), p(nw), p(inv), T, H, d, p(u), int(K.Act.F32), st)
        return u, (wu, h, inv, x, nw), lambda: lib.sxb_hc_mix_up_q8(*args)

    def dense(k, st):
        w = upload(oracle.quantize(random_weights(rng, 64, k), 64, 4), cuda)
        x, y = torch.randn((4, k), device=cuda).to(torch.bfloat16), torch.empty((4, 64), dtype=torch.bfloat16, device=cuda)
        args = (p(x), C.byref(w.c()), p(y), 4, int(K.Act.BF16), int(K.Act.BF16), st)
        return y, (w, x), lambda: lib.sxb_linear_q4(*args)

    def router(planes, st):
        w = K.router_prepare(torch.randn((64, 128), device=cuda), planes)
        x, out = torch.randn((130, 128), device=cuda).to(torch.bfloat16), torch.empty((130, 64), device=cuda)
        args = (p(x), p(w.data), planes, None, 130, 64, 128, p(out), 64, st)
        return out, (w, x), lambda: lib.sxb_router_logits_wmma(*args)

    for make, sizes in ((up, (1024, 32)), (dense, (11008, 256)), (router, (3, 1))):
        streams = [torch.cuda.Stream() for _ in sizes]
        calls = [make(n, C.c_void_p(s.cuda_stream)) for n, s in zip(sizes, streams)]
        want, failed = [], []
        torch.cuda.synchronize()
        for out, _, call in calls:
            assert call() == 0
            torch.cuda.synchronize()
            want.append(out.clone())
            out.zero_()
        torch.cuda.synchronize()
        stop = time.monotonic() + 1.0

        def loop(call, stream):
            while time.monotonic() < stop:
                for _ in range(200):
                    if call() != 0:
                        failed.append(lib.sxb_last_error().decode())
                stream.synchronize()

        threads = [threading.Thread(target=loop, args=(call, s)) for (_, _, call), s in zip(calls, streams)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert not failed, (len(failed), failed[0])
        assert all(torch.equal(out, w) for (out, _, _), w in zip(calls, want))


def _ws(nbytes, device):
    return torch.empty(nbytes, dtype=torch.uint8, device=device)  # the caching allocator hands out 512-byte aligned blocks


# (bits, G, T, d, r, inject): short and long contractions, few and many tokens a stream (the two tcgen05 kernels and both
# tile widths of the second), an up mix of more than one block of 1024 tokens, one token
WMMA_CASES = [(4, 64, 40, 256, 64, True), (8, 128, 200, 512, 320, True), (4, 128, 700, 2560, 320, True), (8, 64, 50, 2560, 64, False),
              (4, 32, 1100, 128, 32, True), (8, 32, 1, 128, 64, True)]


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,G,T,d,r,inject", WMMA_CASES)
def test_hc_mix_wmma(cuda, oracle, dt, bits, G, T, d, r, inject):
    """hc_mix_down_wmma then hc_mix_up_wmma against the oracle with the matrix-unit path's operand roundings (x, h and the
    weights once to F16): what remains is FP32 summation order.  Also within 1e-2 x RMS of the unrounded math."""
    from strixite_b200 import kernels as K
    H, eps = 4, 1e-6
    rng = np.random.default_rng(T * 11 + d + bits)
    R = r + (H if inject else 0)
    wd = oracle.quantize(random_weights(rng, R, H * d, std=0.05), G, bits)
    wu = oracle.quantize(random_weights(rng, H * d, r, std=0.2), 32 if r % G else G, bits)
    norm_w = (rng.standard_normal(H * d) * 0.1).astype(np.float32)
    x = (rng.standard_normal((T, H * d)) * np.repeat(rng.random((T, H)) * 3 + 0.2, d, axis=1)).astype(np.float32)
    if dt == torch.bfloat16:
        xb = oracle.f32_to_bf16(x)
        x = oracle.bf16_to_f32(xb)
        xd, act = bf16_tensor(xb, cuda), K.Act.BF16
    else:
        xd, act = torch.from_numpy(x).to(cuda), K.Act.F32
    h = torch.full((T, r), float("nan"), dtype=torch.float32, device=cuda)
    w_in = torch.full((T, H), float("nan"), dtype=torch.float32, device=cuda) if inject else None
    inv = torch.full((T, H), float("nan"), dtype=torch.float32, device=cuda)
    ws = _ws(K.hc_wmma_workspace_bytes(T, H, d, R, bits, G), cuda)
    K.hc_mix_down_wmma(xd, upload(wd, cuda), T, H, d, r, inject, eps, h, w_in, inv, ws, act)
    K.check_grouped_status(ws, "hc_mix_down_wmma")
    # the grouping workspace the mix wrote without ids (streams as experts) is the pack's own for ids[t * H + s] = s
    S = T * H
    ids = (torch.arange(S, device=cuda) % H).to(torch.int32)
    nbytes = K.moe_route_workspace_bytes(S, 1, H)
    ws_pack, err = torch.zeros(nbytes // 4, dtype=torch.int32, device=cuda), torch.zeros(4, dtype=torch.int32, device=cuda)
    K.moe_group_routes(ids, S, 1, H, ws_pack, nbytes, err)
    got_ws, want_ws, lay = ws[:nbytes].view(torch.int32).cpu().numpy(), ws_pack.cpu().numpy(), K.route_layout(S, 1, H)
    assert np.array_equal(got_ws[:5], want_ws[:5])
    assert np.array_equal(got_ws[lay["offsets"]:lay["offsets"] + H + 2], want_ws[lay["offsets"]:lay["offsets"] + H + 2])
    assert np.array_equal(got_ws[lay["slots"]:lay["slots"] + S], want_ws[lay["slots"]:lay["slots"] + S])
    for rows, n_at in ((8, 0), (128, 3)) + tuple((rows, lay[f"tile{rows}_n"]) for rows in K.TC_TILES):
        n = int(want_ws[n_at])
        assert int(got_ws[n_at]) == n
        for part in ("bucket", "start"):
            at = lay[f"tile{rows}_{part}"]
            assert np.array_equal(got_ws[at:at + n], want_ws[at:at + n])
    h_ref, w_in_ref, inv_ref = oracle.hc_mix_down(x, wd, H, d, r, inject, eps, f16_operands=True)
    h_exact, _, _ = oracle.hc_mix_down(x, wd, H, d, r, inject, eps)
    assert max_abs_over_rms(inv.cpu().numpy(), inv_ref) <= 1e-5
    assert max_abs_over_rms(h.cpu().numpy(), h_ref) <= 2e-4
    assert max_abs_over_rms(h.cpu().numpy(), h_exact) <= 1e-2
    if inject:
        assert max_abs_over_rms(w_in.cpu().numpy(), w_in_ref) <= 2e-4
    # inv_ready: the same result from an inv the caller already holds, which must not be rewritten
    h2 = torch.full_like(h, float("nan"))
    inv_before = inv.clone()
    K.hc_mix_down_wmma(xd, upload(wd, cuda), T, H, d, r, inject, eps, h2, w_in, inv, ws, act, inv_ready=True)
    assert torch.equal(h2, h) and torch.equal(inv, inv_before)
    # the up half on the GPU's own h and inv
    u = torch.empty((T, d), dtype=dt, device=cuda)
    wu_dev = K.to_chunk_major(upload(wu, cuda))
    ws_up = _ws(K.hc_mix_up_wmma_workspace_bytes(T, H, d, r, bits, wu.G), cuda)
    K.hc_mix_up_wmma(h, wu_dev, xd, torch.from_numpy(norm_w).to(cuda), inv, T, H, d, u, ws_up, act)
    K.check_dense_status("hc_mix_up_wmma")
    u_ref = oracle.hc_mix_up(h.cpu().numpy(), wu, x, norm_w, inv.cpu().numpy(), H, d, f16_operands=True)
    u_exact = oracle.hc_mix_up(h.cpu().numpy(), wu, x, norm_w, inv.cpu().numpy(), H, d)
    if dt == torch.float32:
        assert max_abs_over_rms(u.cpu().numpy(), u_ref) <= 2e-4
        assert max_abs_over_rms(u.cpu().numpy(), u_exact) <= 1e-2
    else:
        got = oracle.bf16_to_f32(bits_of(u)).astype(np.float64)
        assert np.all(np.abs(got - u_ref) <= 2.0 ** -8 * np.abs(u_ref) + 2e-4 * np.sqrt(np.mean(u_ref ** 2)))  # one BF16 rounding
    # and the tensor-core mix agrees with the per-token kernels of the same library
    u_pt = torch.empty_like(u)
    K.hc_mix_up(h, wu_dev, xd, torch.from_numpy(norm_w).to(cuda), inv, T, H, d, u_pt, act)
    # (two roundings to BF16 of values a few times the RMS may differ by one unit in the last place each)
    assert max_abs_over_rms(u.float().cpu().numpy(), u_pt.float().cpu().numpy().astype(np.float64)) <= (5e-2 if dt == torch.bfloat16 else 1e-2)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,d", [(1, 64), (37, 2560), (300, 136)])
def test_hc_inject_inv(cuda, oracle, dt, T, d):
    """hc_inject_inv leaves X bit-identical to hc_inject, and inv = 1 / sqrt(mean(stored X_s^2) + eps)."""
    from strixite_b200 import kernels as K
    H, eps = 4, 1e-6
    rng = np.random.default_rng(T + d)
    x = torch.from_numpy(rng.standard_normal((T, H * d)).astype(np.float32)).to(cuda).to(dt)
    y = torch.from_numpy(rng.standard_normal((T, d)).astype(np.float32)).to(cuda).to(dt)
    w_in = torch.from_numpy((rng.random((T, H)) * 2).astype(np.float32)).to(cuda)
    act = K.Act.BF16 if dt == torch.bfloat16 else K.Act.F32
    want = x.clone()
    K.hc_inject(want, w_in, y, T, H, d, act)
    inv = torch.full((T, H), float("nan"), dtype=torch.float32, device=cuda)
    K.hc_inject_inv(x, w_in, y, T, H, d, eps, inv, act)
    torch.cuda.synchronize()
    assert torch.equal(x, want)
    xs = want.double().cpu().numpy().reshape(T, H, d)
    inv_ref = 1.0 / np.sqrt((xs * xs).mean(axis=2) + eps)
    assert max_abs_over_rms(inv.cpu().numpy(), inv_ref) <= 1e-5


def test_hc_mix_wmma_argument_checks(cuda, oracle):
    from strixite_b200 import kernels as K
    rng = np.random.default_rng(2)
    H, d, r, T = 4, 128, 32, 3
    wd = upload(oracle.quantize(random_weights(rng, r + H, H * d), 64, 4), cuda)
    x = torch.zeros((T, H * d), dtype=torch.bfloat16, device=cuda)
    h, w_in, inv = (torch.zeros((T, n), dtype=torch.float32, device=cuda) for n in (r, H, H))
    need = K.hc_wmma_workspace_bytes(T, H, d, r + H, 4, 64)
    with pytest.raises(K.Error, match="workspace of"):
        K.hc_mix_down_wmma(x, wd, T, H, d, r, True, 1e-6, h, w_in, inv, _ws(need - 256, cuda), K.Act.BF16)
    with pytest.raises(K.Error, match="w_in must be given exactly when inject"):
        K.hc_mix_down_wmma(x, wd, T, H, d, r, True, 1e-6, h, None, inv, _ws(need, cuda), K.Act.BF16)
    with pytest.raises(K.Error, match="hc_mix_down_wmma_workspace_bytes: T = 3, H = 4, d = 96"):
        K.hc_wmma_workspace_bytes(T, H, 96, r + H, 4, 32)
    wu = K.to_chunk_major(upload(oracle.quantize(random_weights(rng, H * d, r), 32, 8), cuda))
    u = torch.zeros((T, d), dtype=torch.bfloat16, device=cuda)
    nw = torch.zeros(H * d, dtype=torch.float32, device=cuda)
    with pytest.raises(K.Error, match="workspace of"):
        K.hc_mix_up_wmma(h, wu, x, nw, inv, T, H, d, u, _ws(256, cuda), K.Act.BF16)
    with pytest.raises(K.Error, match="u overlaps"):
        K.hc_mix_up_wmma(h, wu, x, nw, inv, T, H, d, x, _ws(K.hc_mix_up_wmma_workspace_bytes(T, H, d, r, 8, 32), cuda), K.Act.BF16)


@pytest.mark.parametrize("T", [1, 7, 128, 129, 1000])
def test_down_mix_grouping_workspace(cuda, T):
    """The grouping workspace that the tensor-core down mix writes by formula is the pack's for the same slots."""
    from strixite_b200 import kernels as K
    d, r, H, G = 128, 16, 4, 32
    g = torch.Generator(device="cpu").manual_seed(T)
    w = K.quantize((torch.randn((r + H, H * d), generator=g) * 0.1).to(cuda), G, 8)
    x = torch.randn((T, H * d), generator=g).to(torch.bfloat16).to(cuda)
    h, w_in, inv = (torch.empty((T, n), device=cuda) for n in (r, H, H))
    ws = torch.full((K.hc_wmma_workspace_bytes(T, H, d, r + H, 8, G),), 255, dtype=torch.uint8, device=cuda)
    K.hc_mix_down_wmma(x, w, T, H, d, r, True, 1e-6, h, w_in, inv, ws, K.Act.BF16)
    S, nbytes = T * H, K.moe_route_workspace_bytes(T * H, 1, H)
    ref, err = torch.full((nbytes // 4,), -1, dtype=torch.int32, device=cuda), torch.zeros(4, dtype=torch.int32, device=cuda)
    K.moe_group_routes((torch.arange(S, device=cuda) % H).to(torch.int32), S, 1, H, ref, nbytes, err)
    got = ws[:nbytes].view(torch.int32)
    at = K.route_layout(S, 1, H)
    n8, n128 = int(ref[0]), int(ref[3])
    for lo, n in ((0, 8), (at["offsets"], H + 2), (at["slots"], S), (at["tile8_bucket"], n8), (at["tile8_start"], n8), (at["tile128_bucket"], n128), (at["tile128_start"], n128)):
        assert torch.equal(got[lo:lo + n], ref[lo:lo + n]), (lo, n)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,G,T,d,r,spread", [(8, 64, 129, 128, 512, 0), (4, 32, 300, 1280, 416, 0), (8, 128, 700, 256, 384, 9), (4, 64, 65, 384, 192, 9), (8, 32, 1, 128, 32, 0),
                                                 (4, 128, 260, 128, 512, 9), (8, 32, 200, 256, 544, 0), (4, 64, 130, 128, 1024, 9)])
def test_hc_mix_up_wmma_ranks(cuda, oracle, dt, bits, G, T, d, r, spread):
    """The up mix by rank: the kernel that keeps a row block's weights in tensor memory up to 512 (one to four steps, several tokens tiles and row blocks a
    CTA, rows whose groups' scales lie 2^spread apart) and the general one above it."""
    from strixite_b200 import kernels as K
    rng, H = np.random.default_rng(T + r), 4
    w, h = random_weights(rng, H * d, r, std=0.2), (rng.standard_normal((T, r)) * 0.5).astype(np.float32)
    w[:, :G] *= 2.0 ** spread
    h[:, :G] *= 2.0 ** -spread
    wu = oracle.quantize(w, G, bits)
    x, norm_w = rng.standard_normal((T, H * d)).astype(np.float32), (rng.standard_normal(H * d) * 0.1).astype(np.float32)
    inv = (0.5 + rng.random((T, H))).astype(np.float32)
    xd = torch.from_numpy(x).to(cuda).to(dt)
    x = xd.float().cpu().numpy()
    act = K.Act.BF16 if dt == torch.bfloat16 else K.Act.F32
    u = torch.full((T, d), float("nan"), dtype=dt, device=cuda)
    ws = _ws(K.hc_mix_up_wmma_workspace_bytes(T, H, d, r, bits, G), cuda)
    K.hc_mix_up_wmma(torch.from_numpy(h).to(cuda), K.to_chunk_major(upload(wu, cuda)), xd, torch.from_numpy(norm_w).to(cuda), torch.from_numpy(inv).to(cuda), T, H, d, u,
                     ws, act)
    K.check_dense_status("hc_mix_up_wmma")
    ref = oracle.hc_mix_up(h, wu, x, norm_w, inv, H, d, f16_operands=True)
    got = u.float().cpu().numpy().astype(np.float64)
    step = 2.0 ** -8 if dt == torch.bfloat16 else 0.0
    assert np.all(np.abs(got - ref) <= step * np.abs(ref) + 2e-4 * np.sqrt(np.mean(np.square(ref))))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("bits,T,d,r,slot", [(8, 200, 256, 512, 0), (4, 130, 128, 320, 2), (8, 700, 4096, 320, 7), (4, 130, 128, 1024, 3)])
def test_up_mix_gives_up_a_wait(cuda, oracle, lib, dt, bits, T, d, r, slot):
    """Both kernels of the tensor-core up mix (the line is rank 512) with CTA 0 told to leave one fill of its operand ring out: in the first item or in a
    later one, whose predecessors' copies, products and epilogues are under way.  The kernel returns, the status names it, the next call is right."""
    from strixite_b200 import kernels as K
    rng, H, G = np.random.default_rng(T + r), 4, 32
    w, h = random_weights(rng, H * d, r, std=0.2), (rng.standard_normal((T, r)) * 0.5).astype(np.float32)
    wu = oracle.quantize(w, G, bits)
    x, norm_w = rng.standard_normal((T, H * d)).astype(np.float32), (rng.standard_normal(H * d) * 0.1).astype(np.float32)
    inv = (0.5 + rng.random((T, H))).astype(np.float32)
    xd, act = torch.from_numpy(x).to(cuda).to(dt), K.Act.BF16 if dt == torch.bfloat16 else K.Act.F32
    args = [torch.from_numpy(h).to(cuda), K.to_chunk_major(upload(wu, cuda)), xd, torch.from_numpy(norm_w).to(cuda), torch.from_numpy(inv).to(cuda), T, H, d]
    ws, u = _ws(K.hc_mix_up_wmma_workspace_bytes(T, H, d, r, bits, G), cuda), [torch.full((T, d), float("nan"), dtype=dt, device=cuda) for _ in range(3)]
    K.hc_mix_up_wmma(*args, u[0], ws, act)
    K.check_dense_status("warm-up")
    try:
        K.set_wait_limit(2_000_000)
        assert lib.sxb_test_skip_ring_slot(slot) == 0
        K.hc_mix_up_wmma(*args, u[1], ws, act)
        torch.cuda.synchronize()
    finally:
        lib.sxb_test_skip_ring_slot(-1)
        K.set_wait_limit(2_000_000_000)
    with pytest.raises(K.Error, match=r"skipped fill: a tcgen05 kernel gave up a wait at work item \d+ \((a weight producer|an MMA warp|the epilogue|the activation copy|the weight-code copy)"):
        K.check_dense_status("skipped fill")
    K.hc_mix_up_wmma(*args, u[2], ws, act)
    K.check_dense_status("after")
    assert torch.equal(u[2], u[0]) and not bool(torch.isnan(u[2]).any())
