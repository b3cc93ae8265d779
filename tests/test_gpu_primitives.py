"""GPU parity of the primitive-level C ABI (the hd_* functions of o1.c src/cuda/hd_cuda.h)
against the CPU oracle, and against the reference's own CUDA build when oracle/_ref holds it.
Tolerance classes are the reference's (docs/M1_NUMERICAL_CONTRACT.md:48-54): A exact, B pointwise,
C GEMM."""
import ctypes as C

import numpy as np
import pytest
import torch

import parity
from parity import np_ptr, seeded_bf16, torch_to_u16, u16_to_torch, assert_close

pytestmark = pytest.mark.gpu


_KEEP = []


@pytest.fixture(autouse=True)
def _release_device_temporaries():
    yield
    _KEEP.clear()


def dv(a, dev):
    """Host array -> device tensor that stays alive until the test ends (its address is handed to
    asynchronous kernels, so it must not return to the allocator mid-test)."""
    t = u16_to_torch(a, dev) if a.dtype == np.uint16 else torch.from_numpy(a).to(dev)
    _KEEP.append(t)
    return t


def empty_bf16(shape, dev):
    return torch.empty(shape, dtype=torch.bfloat16, device=dev)


def done(pkg, what):
    torch.cuda.synchronize()
    pkg.check_cuda_errbuf(what)


@pytest.mark.parametrize("rows,cols", [(7, 4096), (300, 4096), (1280 * 4, 128), (33, 96), (5, 100), (3, 8192)])
def test_rmsnorm(pkg, orc, dev, rows, cols):
    x, w = seeded_bf16((rows, cols), 1), seeded_bf16(cols, 2, 1.0, 0.1)
    y = empty_bf16((rows, cols), dev)
    pkg.lib.hd_rmsnorm(pkg.ptr(dv(x, dev)), pkg.ptr(dv(w, dev)), pkg.ptr(y), rows, cols, 1e-6)
    done(pkg, "rmsnorm")
    ref = np.empty_like(x)
    orc.orc_rmsnorm(np_ptr(x), np_ptr(w), np_ptr(ref), rows, cols, 1e-6)
    assert_close(torch_to_u16(y), ref, "B", "rmsnorm")
    r = parity.reflib()
    # The reference kernel reduces with a halving tree over min(cols,256) threads (norm.cu:31-35), which
    # only sums every element when that count is a power of two: compare against it for those shapes.
    if r is not None and (cols >= 256 or (cols & (cols - 1)) == 0):
        y2 = empty_bf16((rows, cols), dev)
        r.hd_rmsnorm(pkg.ptr(dv(x, dev)), pkg.ptr(dv(w, dev)), pkg.ptr(y2), rows, cols, 1e-6)
        torch.cuda.synchronize()
        assert_close(y, y2, "B", "rmsnorm vs reference CUDA")


@pytest.mark.parametrize("n", [1, 8, 1000, 4096 * 33 + 5])
def test_pointwise(pkg, orc, dev, n):
    a, b = seeded_bf16(n, 3, 0.0, 3.0), seeded_bf16(n, 4)
    ad, bd, y = dv(a, dev), dv(b, dev), empty_bf16(n, dev)
    ref = np.empty_like(a)
    r = parity.reflib()
    for name, fn, ofn, two in (("silu", pkg.lib.hd_silu, orc.orc_silu, False),
                               ("swiglu", pkg.lib.hd_swiglu, orc.orc_swiglu, True),
                               ("residual_add", pkg.lib.hd_residual_add, orc.orc_residual_add, True)):
        if two:
            fn(pkg.ptr(ad), pkg.ptr(bd), pkg.ptr(y), n)
            ofn(np_ptr(a), np_ptr(b), np_ptr(ref), n)
        else:
            fn(pkg.ptr(ad), pkg.ptr(y), n)
            ofn(np_ptr(a), np_ptr(ref), n)
        done(pkg, name)
        got = torch_to_u16(y)
        if name == "residual_add":
            assert (got == ref).all()               # one fp32 add + RNE: exact
        else:
            assert_close(got, ref, "B", name)
            assert np.abs(got.astype(np.int32) - ref.astype(np.int32)).max() <= 1   # expf ulp only
        if r is not None:
            y2 = empty_bf16(n, dev)
            rfn = getattr(r, "hd_" + name)
            rfn(pkg.ptr(ad), pkg.ptr(bd), pkg.ptr(y2), n) if two else rfn(pkg.ptr(ad), pkg.ptr(y2), n)
            torch.cuda.synchronize()
            assert torch.equal(y.view(torch.int16), y2.view(torch.int16)), f"{name} vs reference CUDA"


LINEAR_SHAPES = [(7, 5, 6, True), (1, 4096, 256, True), (1, 4096, 4096, True), (23, 1024, 4096, False),
                 (300, 4096, 1024, True), (129, 3072, 4096, True), (1037, 4096, 4096, False),
                 (1280, 1024, 3072, False), (257, 4096, 12288, False)]


@pytest.mark.parametrize("M,N,K,bias", LINEAR_SHAPES)
def test_linear(pkg, orc, dev, M, N, K, bias):
    x, w = seeded_bf16((M, K), 5), seeded_bf16((N, K), 6, 0.0, 0.02)
    b = seeded_bf16(N, 7, 0.0, 0.5) if bias else None
    y = empty_bf16((M, N), dev)
    pkg.lib.hd_linear(pkg.ptr(dv(x, dev)), pkg.ptr(dv(w, dev)), pkg.ptr(dv(b, dev)) if bias else None,
                      pkg.ptr(y), M, N, K, 1)
    done(pkg, "linear")
    ref = np.empty((M, N), dtype=np.uint16)
    orc.orc_linear(np_ptr(x), np_ptr(w), np_ptr(b) if bias else None, np_ptr(ref), M, N, K)
    assert_close(torch_to_u16(y), ref, "C", "linear")
    r = parity.reflib()
    if r is not None and M * N * K <= 1037 * 4096 * 4096:
        y2 = empty_bf16((M, N), dev)
        r.hd_linear_reference(pkg.ptr(dv(x, dev)), pkg.ptr(dv(w, dev)), pkg.ptr(dv(b, dev)) if bias else None,
                              pkg.ptr(y2), M, N, K, 1)
        torch.cuda.synchronize()
        assert_close(y, y2, "C", "linear vs reference CUDA kernel")


def test_linear_rejects_untransposed(pkg, dev):
    x = empty_bf16((4, 4), dev)
    pkg.lib.hd_cuda_clear_error()
    pkg.lib.hd_linear(pkg.ptr(x), pkg.ptr(x), None, pkg.ptr(x), 4, 4, 4, 0)
    assert b"transpose_w=0 unsupported" in pkg.lib.hd_cuda_last_error()   # gemm.cu:511-514
    pkg.lib.hd_cuda_clear_error()


@pytest.mark.parametrize("epi", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("bn", [128, 256])
def test_gemm_epilogues(pkg, orc, dev, epi, bn):
    """The fused epilogues keep the reference's rounding points: compare with the unfused oracle chain."""
    if epi == 3 and bn == 128:
        pytest.skip("SwiGLU tiles are 256 wide")
    M, N, K = 300, 512, 768
    x, w, w2 = seeded_bf16((M, K), 8), seeded_bf16((N, K), 9, 0, 0.03), seeded_bf16((N, K), 10, 0, 0.03)
    bias, resid = seeded_bf16(N, 11), seeded_bf16((M, N), 12)
    y = dv(resid, dev).clone() if epi == 4 else empty_bf16((M, N), dev)
    rc = pkg.lib.o1_gemm(pkg.ptr(dv(x, dev)), K, pkg.ptr(dv(w, dev)), pkg.ptr(dv(w2, dev)), pkg.ptr(y), N, M, N,
                         K, epi, pkg.ptr(dv(bias, dev)), pkg.ptr(dv(resid, dev)), N, 0.25, bn)
    assert rc == 0, pkg.last_error()
    done(pkg, "gemm")
    acc = np.empty((M, N), dtype=np.uint16)
    ref = np.empty((M, N), dtype=np.uint16)
    orc.orc_linear(np_ptr(x), np_ptr(w), None, np_ptr(acc), M, N, K)
    if epi == 0:
        ref = acc
    elif epi == 1:
        orc.orc_linear(np_ptr(x), np_ptr(w), np_ptr(bias), np_ptr(ref), M, N, K)
    elif epi == 2:
        orc.orc_residual_add(np_ptr(acc), np_ptr(resid), np_ptr(ref), M * N)
    elif epi == 3:
        up = np.empty((M, N), dtype=np.uint16)
        orc.orc_linear(np_ptr(x), np_ptr(w2), None, np_ptr(up), M, N, K)
        orc.orc_swiglu(np_ptr(acc), np_ptr(up), np_ptr(ref), M * N)
    else:
        accf = parity.bf16_to_f32_np(x).astype(np.float64) @ parity.bf16_to_f32_np(w).astype(np.float64).T
        ref = parity.f32_to_bf16_np((parity.bf16_to_f32_np(resid) + 0.25 * accf).astype(np.float32))
    assert_close(torch_to_u16(y), ref, "C", f"gemm epi {epi}")


def test_gemm_pitched_operands(pkg, orc, dev):
    """x and y as column slices of wider buffers (how the block writes q|k|v side by side)."""
    M, N, K, ldx, ldy = 200, 256, 128, 320, 640
    xb, w = seeded_bf16((M, ldx), 13), seeded_bf16((N, K), 14, 0, 0.05)
    yb = torch.zeros(M, ldy, dtype=torch.bfloat16, device=dev)
    xd = dv(xb, dev)
    rc = pkg.lib.o1_gemm(C.c_void_p(xd.data_ptr() + 64 * 2), ldx, pkg.ptr(dv(w, dev)), None,
                         C.c_void_p(yb.data_ptr() + 128 * 2), ldy, M, N, K, 0, None, None, 0, 0.0, 0)
    assert rc == 0, pkg.last_error()
    done(pkg, "gemm pitched")
    xs = np.ascontiguousarray(xb[:, 64:64 + K])
    ref = np.empty((M, N), dtype=np.uint16)
    orc.orc_linear(np_ptr(xs), np_ptr(w), None, np_ptr(ref), M, N, K)
    got = torch_to_u16(yb)
    assert_close(np.ascontiguousarray(got[:, 128:128 + N]), ref, "C", "pitched gemm")
    assert not got[:, :128].any() and not got[:, 128 + N:].any()


def test_timestep_and_mrope(pkg, orc, dev):
    t = np.array([500.0, 3.0], dtype=np.float32)
    y = torch.empty(2, 256, device=dev)
    pkg.lib.hd_timestep_embed(pkg.ptr(dv(t, dev)), pkg.ptr(y), 2, 256)
    done(pkg, "timestep_embed")
    ref = np.empty((2, 256), dtype=np.float32)
    orc.orc_timestep_embed(np_ptr(t), np_ptr(ref), 2, 256)
    # t*freq reaches 500 rad; one ulp of expf in freq moves the angle by ~3e-5
    assert np.abs(y.cpu().numpy() - ref).max() <= 1e-4
    assert_close(y.cpu().numpy(), ref, "B", "timestep_embed")
    S = 23 + 48
    pos, _ = pkg.seq_t2i(23, 6, 8)
    sec = torch.tensor([24, 20, 20], dtype=torch.int64, device=dev)
    cs, sn = torch.empty(S, 128, device=dev), torch.empty(S, 128, device=dev)
    pkg.lib.hd_mrope_cos_sin(pkg.ptr(pos.to(dev)), 1, S, pkg.ptr(sec), 3, 128, 5e6, 1.0, 1, pkg.ptr(cs), pkg.ptr(sn))
    done(pkg, "mrope")
    rc_, rs_ = np.empty((S, 128), dtype=np.float32), np.empty((S, 128), dtype=np.float32)
    secn = np.array([24, 20, 20], dtype=np.int64)
    orc.orc_mrope_cos_sin(np_ptr(pos.numpy()), 1, S, np_ptr(secn), 3, 128, 5e6, 1.0, 1, np_ptr(rc_), np_ptr(rs_))
    assert np.abs(cs.cpu().numpy() - rc_).max() <= 5e-4 and np.abs(sn.cpu().numpy() - rs_).max() <= 5e-4
    # the compact per-forward table holds the same 64 angles
    tab = torch.empty(S, 128, device=dev)
    assert pkg.lib.o1_mrope_table(pkg.ptr(pos.to(dev)), S, 5e6, pkg.ptr(tab)) == 0
    done(pkg, "mrope_table")
    assert torch.equal(tab[:, :64], cs[:, :64]) and torch.equal(tab[:, 64:], sn[:, :64])
    r = parity.reflib()
    if r is not None:
        c2, s2 = torch.empty(S, 128, device=dev), torch.empty(S, 128, device=dev)
        r.hd_mrope_cos_sin(pkg.ptr(pos.to(dev)), 1, S, pkg.ptr(sec), 3, 128, 5e6, 1.0, 1, pkg.ptr(c2), pkg.ptr(s2))
        torch.cuda.synchronize()
        assert torch.equal(cs, c2) and torch.equal(sn, s2), "mrope table vs reference CUDA (same expressions)"


def test_rotary_and_fused_qk_norm_rope(pkg, orc, dev):
    T, gh, gw, H = 9, 5, 7, 6
    S = T + gh * gw
    pos, _ = pkg.seq_t2i(T, gh, gw)
    secn = np.array([24, 20, 20], dtype=np.int64)
    cs, sn = np.empty((S, 128), dtype=np.float32), np.empty((S, 128), dtype=np.float32)
    orc.orc_mrope_cos_sin(np_ptr(pos.numpy()), 1, S, np_ptr(secn), 3, 128, 5e6, 1.0, 1, np_ptr(cs), np_ptr(sn))
    x = seeded_bf16((H, S, 128), 15)
    y = empty_bf16((H, S, 128), dev)
    pkg.lib.hd_apply_rotary(pkg.ptr(dv(x, dev)), pkg.ptr(dv(cs, dev)), pkg.ptr(dv(sn, dev)), pkg.ptr(y), H, S, 128)
    done(pkg, "rotary")
    ref = np.empty_like(x)
    orc.orc_apply_rotary(np_ptr(x), np_ptr(cs), np_ptr(sn), np_ptr(ref), H, S, 128)
    assert (torch_to_u16(y) == ref).all()          # same table, same three roundings: exact
    # fused: seq-major [S, ld] in place == head_split -> rmsnorm -> rotary of the oracle
    ld = H * 128 + 256
    buf = seeded_bf16((S, ld), 16)
    w = seeded_bf16(128, 17, 1.0, 0.1)
    tab = torch.empty(S, 128, device=dev)
    pkg.lib.o1_mrope_table(pkg.ptr(pos.to(dev)), S, 5e6, pkg.ptr(tab))
    bd = dv(buf, dev)
    assert pkg.lib.o1_qk_norm_rope(pkg.ptr(bd), ld, S, H, pkg.ptr(dv(w, dev)), pkg.ptr(tab), 1e-6) == 0
    done(pkg, "qk_norm_rope")
    xs = np.ascontiguousarray(buf[:, :H * 128])
    hm, nr, ro = (np.empty((H, S, 128), dtype=np.uint16) for _ in range(3))
    orc.orc_head_split(np_ptr(xs), np_ptr(hm), S, H, 128)
    orc.orc_rmsnorm(np_ptr(hm), np_ptr(w), np_ptr(nr), H * S, 128, 1e-6)
    tabn = tab.cpu().numpy()
    cs2 = np.concatenate([tabn[:, :64], tabn[:, :64]], 1).copy()
    sn2 = np.concatenate([tabn[:, 64:], tabn[:, 64:]], 1).copy()
    orc.orc_apply_rotary(np_ptr(nr), np_ptr(cs2), np_ptr(sn2), np_ptr(ro), H, S, 128)
    want = np.empty((S, H * 128), dtype=np.uint16)
    orc.orc_head_merge(np_ptr(ro), np_ptr(want), S, H, 128)
    got = torch_to_u16(bd)
    assert_close(np.ascontiguousarray(got[:, :H * 128]), want, "B", "fused q/k norm + rope")
    assert (got[:, H * 128:] == buf[:, H * 128:]).all()      # columns beyond the heads untouched


def test_exact_copies(pkg, orc, dev):
    S, H, D = 37, 5, 128
    x = seeded_bf16((S, H, D), 18)
    a, b = empty_bf16((H, S, D), dev), empty_bf16((S, H, D), dev)
    pkg.lib.hd_head_split(pkg.ptr(dv(x, dev)), pkg.ptr(a), S, H, D)
    pkg.lib.hd_head_merge(pkg.ptr(a), pkg.ptr(b), S, H, D)
    done(pkg, "head split/merge")
    ref = np.empty((H, S, D), dtype=np.uint16)
    orc.orc_head_split(np_ptr(x), np_ptr(ref), S, H, D)
    assert (torch_to_u16(a) == ref).all() and (torch_to_u16(b) == x).all()
    # gather (OOB -> row 0) and tms substitution (embed.cu:15-58)
    rows, cols = 50, 256
    table = seeded_bf16((rows, cols), 19)
    idx = np.array([3, 0, 49, 50, -1, 7, 151673], dtype=np.int64)
    out = empty_bf16((len(idx), cols), dev)
    pkg.lib.hd_gather_rows(pkg.ptr(dv(table, dev)), pkg.ptr(dv(idx, dev)), pkg.ptr(out), len(idx), cols, rows)
    done(pkg, "gather")
    want = table[np.where((idx < 0) | (idx >= rows), 0, idx)]
    assert (torch_to_u16(out) == want).all()
    temb = seeded_bf16(cols, 20)
    out2 = empty_bf16((len(idx), cols), dev)
    pkg.lib.hd_apply_tms_condition(pkg.ptr(dv(idx, dev)), pkg.ptr(out), pkg.ptr(dv(temb, dev)), pkg.ptr(out2),
                                   len(idx), cols, 151673)
    done(pkg, "tms")
    want2 = want.copy()
    want2[6] = temb
    assert (torch_to_u16(out2) == want2).all()
    # vision rows (vision_kernels.cu:344-401)
    mask = np.array([0, 1, 1, 0, 0, 1, 0], dtype=np.uint8)
    emb = seeded_bf16((3, cols), 21)
    o3, o4 = empty_bf16((7, cols), dev), empty_bf16((7, cols), dev)
    pkg.lib.hd_vision_masked_scatter(pkg.ptr(out), pkg.ptr(dv(mask, dev)), pkg.ptr(dv(emb, dev)), pkg.ptr(o3), 7, cols)
    pkg.lib.hd_vision_deepstack_inject(pkg.ptr(out), pkg.ptr(dv(mask, dev)), pkg.ptr(dv(emb, dev)), pkg.ptr(o4), 7, cols)
    done(pkg, "vision rows")
    w3, w4 = want.copy(), want.copy()
    for k, r_ in enumerate(np.nonzero(mask)[0]):
        w3[r_] = emb[k]
        w4[r_] = parity.f32_to_bf16_np(parity.bf16_to_f32_np(want[r_]) + parity.bf16_to_f32_np(emb[k]))
    assert (torch_to_u16(o3) == w3).all() and (torch_to_u16(o4) == w4).all()


@pytest.mark.parametrize("n", [1, 7, 3072 * 64, 3072 * 64 + 3])
def test_scheduler_kernels(pkg, orc, dev, n):
    z, xc, xu = seeded_bf16(n, 22, 0, 4.0), seeded_bf16(n, 23), seeded_bf16(n, 24)
    sigma, sigma_next, g = 0.8769999742507935, 0.8569999933242798, 5.0
    zd, cd, ud = dv(z, dev), dv(xc, dev), dv(xu, dev)
    mc, mu, mo = (torch.empty(n, device=dev) for _ in range(3))
    zn = empty_bf16(n, dev)
    lib = pkg.lib
    lib.hd_sched_vcond(pkg.ptr(zd), pkg.ptr(cd), sigma, pkg.ptr(mc), n)
    lib.hd_sched_vcond(pkg.ptr(zd), pkg.ptr(ud), sigma, pkg.ptr(mu), n)
    lib.hd_sched_cfg_guided(pkg.ptr(mc), pkg.ptr(mu), g, pkg.ptr(mo), n)
    lib.hd_sched_flow_match_step(pkg.ptr(zd), pkg.ptr(mo), sigma, sigma_next, pkg.ptr(zn), n)
    fused = empty_bf16(n, dev)
    assert lib.o1_sched_cfg_flow_step(pkg.ptr(zd), pkg.ptr(cd), pkg.ptr(ud), sigma, sigma_next, g, pkg.ptr(fused), n) == 0
    done(pkg, "scheduler")
    assert torch.equal(zn.view(torch.int16), fused.view(torch.int16)), "fused step != unfused chain"
    omc, omu, omo = (np.empty(n, dtype=np.float32) for _ in range(3))
    ozn, ofz = np.empty(n, dtype=np.uint16), np.empty(n, dtype=np.uint16)
    orc.orc_sched_vcond(np_ptr(z), np_ptr(xc), sigma, np_ptr(omc), n)
    orc.orc_sched_vcond(np_ptr(z), np_ptr(xu), sigma, np_ptr(omu), n)
    orc.orc_sched_cfg_guided(np_ptr(omc), np_ptr(omu), g, np_ptr(omo), n)
    orc.orc_sched_flow_match_step(np_ptr(z), np_ptr(omo), sigma, sigma_next, np_ptr(ozn), n)
    orc.orc_sched_cfg_flow_step(np_ptr(z), np_ptr(xc), np_ptr(xu), sigma, sigma_next, g, np_ptr(ofz), n)
    assert (ozn == ofz).all()
    assert (mc.cpu().numpy() == omc).all()                      # one IEEE subtract and divide
    assert np.abs(mo.cpu().numpy() - omo).max() <= 4e-6 * max(1.0, float(np.abs(omo).max()))
    assert np.abs(torch_to_u16(zn).astype(np.int32) - ozn.astype(np.int32)).max() <= 1
    assert_close(torch_to_u16(zn), ozn, "B", "flow-match step")
    r = parity.reflib()
    if r is not None:
        m1, m2, m3 = (torch.empty(n, device=dev) for _ in range(3))
        z2 = empty_bf16(n, dev)
        r.hd_sched_vcond(pkg.ptr(zd), pkg.ptr(cd), sigma, pkg.ptr(m1), n)
        r.hd_sched_vcond(pkg.ptr(zd), pkg.ptr(ud), sigma, pkg.ptr(m2), n)
        r.hd_sched_cfg_guided(pkg.ptr(m1), pkg.ptr(m2), g, pkg.ptr(m3), n)
        r.hd_sched_flow_match_step(pkg.ptr(zd), pkg.ptr(m3), sigma, sigma_next, pkg.ptr(z2), n)
        torch.cuda.synchronize()
        assert torch.equal(mo, m3) and torch.equal(zn.view(torch.int16), z2.view(torch.int16)), \
            "scheduler chain vs reference CUDA kernels"
        assert torch.equal(fused.view(torch.int16), z2.view(torch.int16)), "fused step vs reference CUDA chain"


def test_flash_euler_and_unipc_kernels(pkg, orc, dev):
    n = 5000
    rng = np.random.default_rng(0)
    zf, mo, noise, old, conv = (rng.standard_normal(n).astype(np.float32) for _ in range(5))
    lib = pkg.lib
    den, zn = torch.empty(n, device=dev), torch.empty(n, device=dev)
    lib.hd_sched_denoised(pkg.ptr(dv(zf, dev)), pkg.ptr(dv(mo, dev)), 0.9, pkg.ptr(den), n)
    lib.hd_sched_z_next(pkg.ptr(dv(noise, dev)), pkg.ptr(den), 0.8, 8.0, pkg.ptr(zn), n)
    up = torch.empty(n, device=dev)
    zb = parity.f32_to_bf16_np(zf)
    lib.hd_sched_bf16_upcast(pkg.ptr(dv(zb, dev)), pkg.ptr(up), n)
    done(pkg, "flash euler")
    oden, ozn = np.empty(n, dtype=np.float32), np.empty(n, dtype=np.float32)
    orc.orc_sched_denoised(np_ptr(zf), np_ptr(mo), 0.9, np_ptr(oden), n)
    orc.orc_sched_z_next(np_ptr(noise), np_ptr(oden), 0.8, 8.0, np_ptr(ozn), n)
    assert np.abs(den.cpu().numpy() - oden).max() <= 1e-6 and np.abs(zn.cpu().numpy() - ozn).max() <= 4e-6
    assert (up.cpu().numpy() == parity.bf16_to_f32_np(zb)).all()
    c = (0.8, 0.9, 0.2, -0.11, 0.12, 0.4, 0.5, 1.3)
    out, oout = torch.empty(n, device=dev), np.empty(n, dtype=np.float32)
    for order in (1, 2):
        lib.hd_unipc_correct(pkg.ptr(dv(zf, dev)), pkg.ptr(dv(mo, dev)), pkg.ptr(dv(old, dev)), pkg.ptr(dv(conv, dev)),
                             *c, order, pkg.ptr(out), n)
        done(pkg, "unipc_correct")
        orc.orc_unipc_correct(np_ptr(zf), np_ptr(mo), np_ptr(old), np_ptr(conv), *c, order, np_ptr(oout), n)
        assert np.abs(out.cpu().numpy() - oout).max() <= 1e-5      # tests/unit/test_base_unipc_cuda.c:155
        lib.hd_unipc_predict(pkg.ptr(dv(zf, dev)), pkg.ptr(dv(mo, dev)), pkg.ptr(dv(old, dev)), c[0], c[1], c[2],
                             c[3], c[4], c[6], c[7], order, pkg.ptr(out), n)
        done(pkg, "unipc_predict")
        orc.orc_unipc_predict(np_ptr(zf), np_ptr(mo), np_ptr(old), c[0], c[1], c[2], c[3], c[4], c[6], c[7],
                              order, np_ptr(oout), n)
        assert np.abs(out.cpu().numpy() - oout).max() <= 1e-5
    lib.hd_unipc_convert(pkg.ptr(dv(zf, dev)), pkg.ptr(dv(mo, dev)), 0.7, pkg.ptr(out), n)
    done(pkg, "unipc_convert")
    orc.orc_unipc_convert(np_ptr(zf), np_ptr(mo), 0.7, np_ptr(oout), n)
    assert np.abs(out.cpu().numpy() - oout).max() <= 1e-6


def test_seeded_fill_is_bit_identical_on_host_and_device(pkg, orc, dev):
    n = 100003
    d16 = empty_bf16(n, dev)
    d32 = torch.empty(n, device=dev)
    assert pkg.lib.o1_fill_normal_bf16(pkg.ptr(d16), n, 99, 1.0, 0.02) == 0
    assert pkg.lib.o1_fill_normal_f32(pkg.ptr(d32), n, 99, 0.0, 1.0) == 0
    done(pkg, "fill")
    h16, h32 = np.empty(n, dtype=np.uint16), np.empty(n, dtype=np.float32)
    orc.orc_fill_normal_bf16(np_ptr(h16), n, 99, 1.0, 0.02)
    orc.orc_fill_normal_f32(np_ptr(h32), n, 99, 0.0, 1.0)
    assert (torch_to_u16(d16) == h16).all()
    assert (d32.cpu().numpy().view(np.uint32) == h32.view(np.uint32)).all()


@pytest.mark.parametrize("M,N,K,ldy,bn", [(300, 512, 256, 512 + 384, 0), (1024, 1024, 512, 1024, 256), (130, 256, 128, 256, 128)])
def test_projection_with_norm_and_rope_in_the_epilogue(pkg, dev, M, N, K, ldy, bn):
    """GEMM whose epilogue applies the per-head RMSNorm + rotary (epilogue 6) == plain GEMM followed by the
    in-place norm + rope kernel, bit for bit; columns of the output row beyond the projection stay untouched."""
    heads = N // 128
    x = dv(seeded_bf16((M, K), 71), dev)
    w = dv(seeded_bf16((N, K), 72, 0.0, 0.05), dev)
    nw = dv(seeded_bf16(128, 73, 1.0, 0.1), dev)
    pos, _ = pkg.seq_t2i(20, 10, (M - 20 + 9) // 10)
    tab = torch.empty(pos.shape[1], 128, device=dev)
    pkg.lib.o1_mrope_table(pkg.ptr(pos.to(dev)), pos.shape[1], 5e6, pkg.ptr(tab))
    assert pos.shape[1] >= M
    fill = seeded_bf16((M, ldy), 74)
    y_fused, y_plain = dv(fill, dev), dv(fill, dev)
    rc = pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y_fused), ldy, M, N, K, 6, pkg.ptr(nw), pkg.ptr(tab),
                         0, 1e-6, bn)
    assert rc == 0, pkg.last_error()
    rc = pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y_plain), ldy, M, N, K, 0, None, None, 0, 0.0, bn)
    assert rc == 0, pkg.last_error()
    assert pkg.lib.o1_qk_norm_rope(pkg.ptr(y_plain), ldy, M, heads, pkg.ptr(nw), pkg.ptr(tab), 1e-6) == 0
    done(pkg, "gemm + norm + rope")
    assert torch.equal(y_fused.view(torch.int16), y_plain.view(torch.int16))
    assert (torch_to_u16(y_fused)[:, N:] == fill[:, N:]).all()
    # shapes the tensor-core tiles do not cover refuse the fused epilogue instead of falling back silently
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y_fused), ldy, 4, N, K, 6, pkg.ptr(nw), pkg.ptr(tab),
                           0, 1e-6, 0) != 0


@pytest.mark.parametrize("M,qc,kc,K", [(300, 512, 128, 256), (1280, 4096, 1024, 4096), (4115, 1024, 256, 512)])
def test_qkv_projections_as_one_launch(pkg, dev, M, qc, kc, K):
    """o1_gemm_qkv (one launch over the three weight tensors, norm + rope on the q and k tiles) == three separate
    projections with the same epilogues, bit for bit; the row pitch may exceed the used columns."""
    ld = qc + 2 * kc + 128
    x = dv(seeded_bf16((M, K), 81), dev)
    wq, wk, wv = (dv(seeded_bf16((n, K), 82 + i, 0.0, 0.05), dev) for i, n in enumerate((qc, kc, kc)))
    nq, nk = dv(seeded_bf16(128, 86, 1.0, 0.1), dev), dv(seeded_bf16(128, 87, 1.0, 0.1), dev)
    pos, _ = pkg.seq_t2i(20, 10, (M - 20 + 9) // 10)
    tab = torch.empty(pos.shape[1], 128, device=dev)
    pkg.lib.o1_mrope_table(pkg.ptr(pos.to(dev)), pos.shape[1], 5e6, pkg.ptr(tab))
    fill = seeded_bf16((M, ld), 88)
    one, three = dv(fill, dev), dv(fill, dev)
    rc = pkg.lib.o1_gemm_qkv(pkg.ptr(x), K, pkg.ptr(wq), pkg.ptr(wk), pkg.ptr(wv), pkg.ptr(one), ld, M, qc, kc, K,
                             pkg.ptr(nq), pkg.ptr(nk), pkg.ptr(tab), 1e-6)
    assert rc == 0, pkg.last_error()
    P = lambda t, off: C.c_void_p(t.data_ptr() + off * 2)
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wq), None, P(three, 0), ld, M, qc, K, 6, pkg.ptr(nq), pkg.ptr(tab), 0, 1e-6, 0) == 0
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wk), None, P(three, qc), ld, M, kc, K, 6, pkg.ptr(nk), pkg.ptr(tab), 0, 1e-6, 0) == 0
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wv), None, P(three, qc + kc), ld, M, kc, K, 0, None, None, 0, 0.0, 0) == 0
    done(pkg, "qkv")
    assert torch.equal(one.view(torch.int16), three.view(torch.int16))
    assert (torch_to_u16(one)[:, qc + 2 * kc:] == fill[:, qc + 2 * kc:]).all()


@pytest.mark.parametrize("M,N,K,epi", [(4352, 4096, 512, 0), (4115, 4096, 256, 2), (4200, 3072, 320, 1), (8320, 4096, 192, 2),
                                       (1280, 4096, 2048, 3), (1400, 4096, 2056, 3), (2304, 4096, 2048, 0), (2561, 4096, 2104, 2),
                                       (2048, 4096, 512, 1), (1921, 4096, 1032, 2), (2304, 4096, 1024, 0),
                                       (2242, 4096, 2048, 3)])
def test_gemm_on_cta_pairs_equals_single_cta_tiles(pkg, dev, M, N, K, epi):
    """The cta_group::2 form (two CTAs per 256 x 256 tile, each with half of the B tile) adds a row's K products in the
    same order as the one-CTA form: same bits, for an even and an odd number of row tiles, a partly filled last row
    tile and a ragged last K block, with the epilogues that take the pair form (plain, +bias, +residual, SwiGLU), by the
    rule for a short K and by the one from K = 2048 on."""
    if pkg.lib.o1_sm_count() == 148:
        assert gemm_form(pkg, M, N, K, epi, 0) == (2, 256, 2)
    x = dv(seeded_bf16((M, K), 91), dev)
    w = dv(seeded_bf16((N, K), 92, 0.0, 0.05), dev)
    up = dv(seeded_bf16((N, K), 95, 0.0, 0.05), dev) if epi == 3 else None
    bias = dv(seeded_bf16(N, 93, 0.0, 0.5), dev) if epi == 1 else None
    resid = dv(seeded_bf16((M, N), 94), dev) if epi == 2 else None
    outs = []
    try:
        for mode in (0, 1):
            pkg.lib.o1_gemm_pair_mode(mode)
            if mode == 0:
                assert gemm_form(pkg, M, N, K, epi, 0)[2] == 1
            y = torch.zeros(M, N, dtype=torch.bfloat16, device=dev)
            rc = pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), pkg.ptr(up), pkg.ptr(y), N, M, N, K, epi,
                                 pkg.ptr(bias) if bias is not None else None,
                                 pkg.ptr(resid) if resid is not None else None, N, 0.0, 0)
            assert rc == 0, pkg.last_error()
            done(pkg, "gemm pair mode %d" % mode)
            outs.append(y)
    finally:
        pkg.lib.o1_gemm_pair_mode(1)
    assert torch.equal(outs[0].view(torch.int16), outs[1].view(torch.int16))
    ref = x.float() @ w.float().t()
    if epi == 1: ref = (ref.bfloat16().float() + bias.float())
    if epi == 2: ref = (ref.bfloat16().float() + resid.float())
    if epi == 3: ref = torch.nn.functional.silu(ref.bfloat16().float()).bfloat16().float() * (x.float() @ up.float().t()).bfloat16().float()
    err = (outs[1].float() - ref).abs().max().item() / max(ref.abs().max().item(), 1e-6)
    assert err < 1e-2, err     # the pair form really computed the product (fp32 reference, bf16 rounding of the result)


@pytest.mark.parametrize("M,N,qc,kc", [(77, 1536, 512, 256), (129, 1536, 512, 256), (144, 1536, 512, 256), (257, 1536, 512, 256), (296, 1536, 512, 256),
                                       (513, 1536, 512, 256), (592, 1536, 512, 256), (785, 1536, 512, 256), (1030, 1536, 512, 256), (1300, 1536, 512, 256),
                                       (300, 12288, 4096, 1024), (785, 12288, 4096, 1024), (1300, 12288, 4096, 1024)])
@pytest.mark.parametrize("K", [2048, 2104])
def test_pairs_with_tokens_as_columns(pkg, dev, M, N, qc, kc, K):
    """gate | up + SwiGLU and q | k | v with the weights as the MMA's rows (tiles of 256 weight rows and a number of tokens that fits)
    give the bits of one-CTA tiles: partly filled token tiles, fewer than a round of tiles and up to eight of them for a pair, a ragged last K
    block, q, k and v tiles of one launch; nothing is written beside the result.  (77 rows of gate | up and q | k | v of 1030 and 1300 rows and
    1024 columns are left to other kernels.)"""
    if pkg.lib.o1_sm_count() == 148:
        assert pkg.lib.o1_gemm_pair_tile(M, N, K, 3, 0) == pkg.lib.o1_gemm_pair_tile(M, N, K, 3, -1)
        assert (pkg.lib.o1_gemm_pair_tile(M, N, K, 3, 0) >= 64) == (M != 77)
        assert (pkg.lib.o1_gemm_qkv_pair_rows(M, qc, kc, K) >= 64) == (qc != 512 or M < 1030)
        assert pkg.lib.o1_gemm_pair_tile(M, N, K, 3, 256) == 0
    x, wg, wu = (dv(seeded_bf16((r, K), 60 + i, 0.0, 1.0 if i == 0 else 0.05), dev) for i, r in enumerate((M, N, N)))
    ys = []
    for bn in (0, 256):
        y = torch.full((M + 1, N + 8), 777.0, dtype=torch.bfloat16, device=dev)
        assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wg), pkg.ptr(wu), pkg.ptr(y), N + 8, M, N, K, 3, None, None, 0, 0.0, bn) == 0, pkg.last_error()
        done(pkg, "swiglu")
        assert (y[M:] == 777.0).all() and (y[:, N:] == 777.0).all(), "written beside the matrix"
        ys.append(y)
    assert torch.equal(ys[0].view(torch.int16), ys[1].view(torch.int16))
    g, u = ((x.float() @ w.float().t()).bfloat16().float() for w in (wg, wu))
    ref = torch.nn.functional.silu(g).bfloat16().float() * u
    assert (ys[0][:M, :N].float() - ref).abs().max().item() < 1e-2 * ref.abs().max().item()
    wq, wk, wv = (dv(seeded_bf16((n, K), 70 + i, 0.0, 0.05), dev) for i, n in enumerate((qc, kc, kc)))
    nq, nk = dv(seeded_bf16(128, 75, 1.0, 0.1), dev), dv(seeded_bf16(128, 76, 1.0, 0.1), dev)
    tab = torch.empty(M, 128, device=dev).uniform_(-1, 1)
    ld = qc + 2 * kc + 8
    one, three = (torch.full((M + 1, ld), 777.0, dtype=torch.bfloat16, device=dev) for _ in range(2))
    assert pkg.lib.o1_gemm_qkv(pkg.ptr(x), K, pkg.ptr(wq), pkg.ptr(wk), pkg.ptr(wv), pkg.ptr(one), ld, M, qc, kc, K, pkg.ptr(nq),
                               pkg.ptr(nk), pkg.ptr(tab), 1e-6) == 0, pkg.last_error()
    at = lambda off: C.c_void_p(three.data_ptr() + off * 2)  # noqa: E731
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wq), None, at(0), ld, M, qc, K, 6, pkg.ptr(nq), pkg.ptr(tab), 0, 1e-6, 128) == 0
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wk), None, at(qc), ld, M, kc, K, 6, pkg.ptr(nk), pkg.ptr(tab), 0, 1e-6, 128) == 0
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wv), None, at(qc + kc), ld, M, kc, K, 0, None, None, 0, 0.0, 128) == 0
    done(pkg, "qkv")
    assert torch.equal(one.view(torch.int16), three.view(torch.int16))
    assert pkg.lib.o1_device_error() == 0


@pytest.mark.parametrize("M,K", [(130, 72), (256, 192), (200, 64)])
@pytest.mark.parametrize("blocks", [149, 185, 186, 259, 295])
def test_last_tiles_as_halves(pkg, dev, M, K, blocks):
    """gate | up + SwiGLU on CTA pairs (blocks of 128 columns, 74 pairs): the tiles of a last round that at most half of the pairs have,
    1 and 37 of them, are taken as two halves, more of them whole; the bits of one-CTA tiles, nothing written beside the result."""
    N = blocks * 128
    x, wg, wu = (dv(seeded_bf16((r, K), 80 + i, 0.0, 1.0 if i == 0 else 0.05), dev) for i, r in enumerate((M, N, N)))
    ys = []
    try:
        for on in (1, 0):
            pkg.lib.o1_gemm_pair_mode(on)
            if pkg.lib.o1_sm_count() == 148:
                assert gemm_form(pkg, M, N, K, 3, -1)[2] == 1 + on and pkg.lib.o1_gemm_pair_tile(M, N, K, 3, -1) == 0
            y = torch.full((M + 1, N + 8), 777.0, dtype=torch.bfloat16, device=dev)
            assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wg), pkg.ptr(wu), pkg.ptr(y), N + 8, M, N, K, 3, None, None, 0, 0.0, -1) == 0, pkg.last_error()
            done(pkg, "swiglu")
            assert (y[M:] == 777.0).all() and (y[:, N:] == 777.0).all(), "written beside the matrix"
            ys.append(y)
    finally:
        pkg.lib.o1_gemm_pair_mode(1)
    assert torch.equal(ys[0].view(torch.int16), ys[1].view(torch.int16))
    assert pkg.lib.o1_device_error() == 0


@pytest.mark.parametrize("M,N,K", [(1280, 12288, 2048), (1280, 12288, 2104), (2048, 12288, 4096), (2242, 12288, 2048), (1400, 1536, 2104)])
def test_gate_up_on_whole_pair_tiles_of_a_long_k(pkg, dev, M, N, K):
    """gate | up + SwiGLU on tiles of 256 x 256, more K blocks to a tile than there are stages: last rounds of halves (36 and 28 of 74 pairs), a whole
    one (50), a single round, ragged K and rows; the bits of one-CTA tiles, nothing written beside the result."""
    if pkg.lib.o1_sm_count() == 148:
        assert gemm_form(pkg, M, N, K, 3, 0) == (2, 256, 2) and pkg.lib.o1_gemm_pair_tile(M, N, K, 3, 0) == 0
    x, wg, wu = (dv(seeded_bf16((r, K), 50 + i, 0.0, 1.0 if i == 0 else 0.05), dev) for i, r in enumerate((M, N, N)))
    ys = []
    for bn in (0, 256):
        y = torch.full((M + 1, N + 8), 777.0, dtype=torch.bfloat16, device=dev)
        assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wg), pkg.ptr(wu), pkg.ptr(y), N + 8, M, N, K, 3, None, None, 0, 0.0, bn) == 0, pkg.last_error()
        done(pkg, "swiglu")
        assert (y[M:] == 777.0).all() and (y[:, N:] == 777.0).all(), "written beside the matrix"
        ys.append(y)
    assert torch.equal(ys[0].view(torch.int16), ys[1].view(torch.int16))


def check_linear_f64(y, x, w, bias, what):
    """y against 64 bits: an FP32 sum of K products in any order is within K * 2^-23 * sum|x||w| of the exact one, and the
    two bf16 roundings (of the sum, of the sum plus bias) are monotonic, so the result lies between the rounded ends."""
    acc = x.double() @ w.double().t()
    bound = (x.double().abs() @ w.double().abs().t()) * x.shape[1] * 2.0 ** -23
    lo, hi = (acc - bound).bfloat16().double(), (acc + bound).bfloat16().double()
    if bias is not None:
        lo, hi = (lo + bias.double()).bfloat16().double(), (hi + bias.double()).bfloat16().double()
    bad = ((y.double() < lo) | (y.double() > hi)).sum().item()
    assert bad == 0, f"{what}: {bad} of {y.numel()} outside the rounding interval"


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 7, 8, 33, 127, 128, 129, 300, 517])
@pytest.mark.parametrize("N,K", [(72, 40), (128, 64), (1032, 200), (4096, 256), (96, 4104), (1152, 1160), (2400, 2056)])
def test_linear_of_few_tiles(pkg, dev, M, N, K):
    """hd_linear where there are few output tiles: the row kernel below eight rows, then tiles of 32, 96 or 128
    columns, with a ragged last tile, a ragged last K block and fewer K blocks than stages; nothing is written behind."""
    g = torch.Generator(device=dev).manual_seed(M * 7 + N + K)
    x, w, b = (torch.empty(s, device=dev).normal_(0, d, generator=g).bfloat16() for s, d in (((M, K), 1.0), ((N, K), 0.05), ((N,), 0.5)))
    for bias in (b, None):
        y = torch.full((M + 1, N), 777.0, dtype=torch.bfloat16, device=dev)
        pkg.lib.hd_linear(pkg.ptr(x), pkg.ptr(w), pkg.ptr(bias), pkg.ptr(y), M, N, K, 1)
        done(pkg, "linear")
        check_linear_f64(y[:M], x, w, bias, f"linear {M}x{N}x{K}")
        assert (y[M:] == 777.0).all(), "rows beyond M were written"
    assert pkg.lib.o1_device_error() == 0


def gemm_form(pkg, M, N, K, epi, bn):
    """(form, tile width or rows, CTAs that share a tile) of o1_gemm_form."""
    width, ctas = C.c_int(0), C.c_int(0)
    return pkg.lib.o1_gemm_form(M, N, K, epi, bn, C.byref(width), C.byref(ctas)), width.value, ctas.value


@pytest.mark.parametrize("M,N,K,cols", [(8, 72, 256, 32), (77, 4096, 632, 32), (40, 4096, 320, 32), (16, 1032, 4096, 32), (17, 512, 832, 32), (33, 1024, 640, 32),
                                        (100, 768, 1024, 32), (113, 640, 384, 32), (64, 1024, 576, 32), (65, 3072, 520, 32), (128, 4608, 1152, 32),
                                        (129, 2048, 1032, 32), (300, 1024, 4096, 32), (520, 896, 2048, 32), (256, 4608, 1088, 64), (130, 3072, 1088, 48),
                                        (520, 1152, 1152, 48), (300, 1160, 2056, 32)])
@pytest.mark.parametrize("epi", [0, 1, 2, 7, 8, 9])
def test_narrow_tiles_on_pairs_give_the_bits_of_single_ctas(pkg, dev, M, N, K, cols, epi):
    """The 32-column form with two CTAs per tile of 128 x 64, 96 or 128 and four K blocks to a copy against the one-CTA form (pair mode 0), every
    epilogue: rows shared by the two CTAs in eights, row tiles whose second half has no rows or few, a ragged last column tile, K blocks
    that are no whole number of copies."""
    if epi in (2, 8, 9) and N % 128:
        pytest.skip("the residual epilogues take whole 128-column tiles")
    g = torch.Generator(device=dev).manual_seed(M + N + K + epi)
    x, w, b, r = (torch.empty(s, device=dev).normal_(0, d, generator=g).bfloat16()
                  for s, d in (((M, K), 1.0), ((N, K), 0.05), ((N,), 0.5), ((M, N), 1.0)))
    ys = []
    try:
        for mode in (1, 0):
            pkg.lib.o1_gemm_pair_mode(mode)
            if pkg.lib.o1_sm_count() == 148:
                assert gemm_form(pkg, M, N, K, epi, 0) == (4, 32, 1)
                assert pkg.lib.o1_gemm_pair_tile(M, N, K, epi, 0) == (cols if mode else 0)
            y = torch.full((M + 1, N + 8), 777.0, dtype=torch.bfloat16, device=dev)
            assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y), N + 8, M, N, K, epi, pkg.ptr(b), pkg.ptr(r), N, 0.0, 0) == 0, pkg.last_error()
            done(pkg, "narrow tiles")
            assert (y[M:] == 777.0).all() and (y[:, N:] == 777.0).all(), "written beyond the matrix"
            ys.append(y)
    finally:
        pkg.lib.o1_gemm_pair_mode(1)
    assert torch.equal(ys[0].view(torch.int16), ys[1].view(torch.int16))
    check_epilogue_f64(ys[0][:M, :N], x, w, b, r, epi, "narrow tiles")
    assert pkg.lib.o1_device_error() == 0


@pytest.mark.parametrize("M,N,K", [(520, 1152, 4304), (9, 72, 2120), (96, 1152, 4304), (128, 4608, 2048), (257, 1160, 2112), (640, 1024, 2000),
                                   (300, 128, 4104)])
def test_k_in_parts_is_added_in_the_order_of_the_parts(pkg, dev, M, N, K):
    """A K that is summed in parts: a part's first product is all there is in it, 2^24, 1, -2^24, 1, .., so that the FP32 sum of the parts from
    zero on is 1 or 2 more where their order is another (2^24 + 1 is 2^24 there)."""
    form = gemm_form(pkg, M, N, K, 0, -1)
    if pkg.lib.o1_sm_count() == 148:
        assert form[:2] == (4, 128) and form[2] > 1
    x, w = (torch.zeros(r, K, dtype=torch.bfloat16, device=dev) for r in (M, N))
    kb, want = (K + 63) // 64, np.float32(0)
    for p in range(form[2]):
        big = {0: 4096.0, 2: -4096.0}.get(p)
        x[:, p * kb // form[2] * 64] = big or 1.0
        w[:, p * kb // form[2] * 64] = 4096.0 if big else 1.0
        want = np.float32(want + np.float32(4096.0 * big if big else 1.0))
    y = torch.full((M + 1, N + 8), 777.0, dtype=torch.bfloat16, device=dev)
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y), N + 8, M, N, K, 0, None, None, N, 0.0, -1) == 0, pkg.last_error()
    done(pkg, "K in parts")
    assert (y[:M, :N] == float(want)).all(), (y[0, 0].item(), want)
    assert (y[M:] == 777.0).all() and (y[:, N:] == 777.0).all(), "written beyond the matrix"
    assert pkg.lib.o1_device_error() == 0


def gelu_tanh_f64(v):
    """0.5 v (1 + tanh u) = v / (1 + e^-2u): in 64 bits too, 1 + tanh u has no digits left where u is far below zero."""
    return v / (1 + torch.exp(-2 * 0.7978845608028654 * (v + 0.044715 * v ** 3)))


def check_epilogue_f64(y, x, w, b, r, epi, what):
    """As check_linear_f64, carried through the epilogue's further roundings, each of which is monotonic; GELU is not, so there
    its slope (at most 1.13) times the interval is allowed, the rounding to bf16 (2^-8 of the value just above a power of two)
    and the fp32 evaluation: an exponent of up to 88 with three roundings of 2^-24, so 2^-15 of the value, and two ulp each for
    exponential and division; 2^-14 in all."""
    acc = x.double() @ w.double().t()
    bound = (x.double().abs() @ w.double().abs().t()) * x.shape[1] * 2.0 ** -23
    rnd = lambda t: t.bfloat16().double()  # noqa: E731
    lo, hi = rnd(acc - bound), rnd(acc + bound)
    if epi in (1, 7, 8):
        lo, hi = rnd(lo + b.double()), rnd(hi + b.double())
    if epi == 9:
        ends = rnd(lo * b.double()), rnd(hi * b.double())
        lo, hi = torch.minimum(*ends), torch.maximum(*ends)
    if epi in (2, 8, 9):
        lo, hi = rnd(r.double() + lo), rnd(r.double() + hi)
    if epi == 7:
        mid = gelu_tanh_f64((lo + hi) / 2)
        room = 1.13 * (hi - lo) / 2 + (2.0 ** -8 + 2.0 ** -14) * mid.abs() + 1e-30
        lo, hi = mid - room, mid + room
    bad = (y.double() < lo) | (y.double() > hi)
    first = [t[bad][:4].tolist() for t in (y.double(), lo, hi)]
    assert not bad.any(), f"{what}: {bad.sum().item()} of {y.numel()} outside the rounding interval: {first}"


@pytest.mark.parametrize("M,N,K,ctas", [(520, 1152, 4304, 5), (96, 1152, 4304, 6), (128, 4608, 4608, 6), (300, 128, 2048, 6),
                                        (300, 1160, 2112, 6), (700, 1024, 2112, 4), (96, 1152, 1152, 1), (130, 4608, 4608, 1),
                                        (64, 4304, 1152, 1), (9, 72, 520, 1)])
@pytest.mark.parametrize("epi", [0, 1, 2, 7, 8, 9])
def test_gemm_with_k_split_over_a_cluster(pkg, dev, M, N, K, ctas, epi):
    """A tile's K shared by four to six CTAs of a cluster where force_bn = -1 chooses that (and, last, shapes where it does not),
    every epilogue, against 64 bits and against the whole-K tile: the FP32 sums differ by their order only, so the results are
    equal or neighbours."""
    if epi in (2, 8, 9) and N % 128:
        pytest.skip("the residual epilogues take whole 128-column tiles")
    if pkg.lib.o1_sm_count() == 148:
        assert gemm_form(pkg, M, N, K, epi, -1) == (4, 128 if ctas > 1 else 32, ctas)
    assert gemm_form(pkg, M, N, K, epi, 0)[2] == 1
    g = torch.Generator(device=dev).manual_seed(M + N + K + epi)
    x, w, b, r = (torch.empty(s, device=dev).normal_(0, d, generator=g).bfloat16()
                  for s, d in (((M, K), 1.0), ((N, K), 0.05), ((N,), 0.5), ((M, N), 1.0)))
    ys = []
    for bn in (-1, 0):
        y = torch.full((M + 1, N), 777.0, dtype=torch.bfloat16, device=dev)
        rc = pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y), N, M, N, K, epi, pkg.ptr(b), pkg.ptr(r), N, 0.0, bn)
        assert rc == 0, pkg.last_error()
        done(pkg, "gemm")
        assert (y[M:] == 777.0).all(), "rows beyond M were written"
        check_epilogue_f64(y[:M], x, w, b, r, epi, f"epilogue {epi}, force_bn {bn}")
        ys.append(y[:M])
    # one bf16 step of the sum, carried through the epilogue: 2^-7 of the largest term
    scale = (x.float() @ w.float().t()).abs() * (b.abs().float() if epi == 9 else 1.0) + b.abs().float() + r.abs().float() + 1e-3
    assert ((ys[0].float() - ys[1].float()).abs() <= scale * 2.0 ** -6).all()
    assert (ys[0] != ys[1]).float().mean() < 0.02
    assert pkg.lib.o1_device_error() == 0


@pytest.mark.parametrize("sigma", [0.857, 1.0, 0.008, 1.0 / 3.0, 0.99999994, 3e-10, 1e-12, 2e9, 1e30])
@pytest.mark.parametrize("n", [8, 4096 * 8, 1003])
def test_fused_step_equals_the_chain_for_every_kind_of_value(pkg, dev, sigma, n):
    """The fused guidance + Euler step shares one reciprocal of sigma among all its divisions; its bits are those of the
    separate kernels with their IEEE divisions, also where the short division does not apply: equal operands, signed
    zeros, tiny and huge values, infinities, NaN, and sigmas outside its range."""
    g = torch.Generator(device=dev).manual_seed(n)
    special = torch.tensor([0.0, -0.0, 1e-38, -1e-38, 2e-30, -3e-17, 1e20, -1e20, 3e38, float("inf"), -float("inf"), float("nan"),
                            1.0, -1.0, 0.5, 8.0], device=dev).bfloat16()
    z, xc, xu = (torch.empty(n, device=dev).normal_(0, s, generator=g).bfloat16() for s in (4.0, 1.0, 1.0))
    for t in (z, xc, xu):           # a run of ordinary vectors, then specials in every combination that falls out
        at = torch.randperm(n, device=dev, generator=g)[:max(1, n // 3)]
        t[at] = special[torch.randint(0, 16, (at.numel(),), device=dev, generator=g)]
    xc[:: 5] = z[:: 5]
    fused, chain = torch.empty_like(z), torch.empty_like(z)
    s1 = sigma * 0.9
    assert pkg.lib.o1_sched_cfg_flow_step(pkg.ptr(z), pkg.ptr(xc), pkg.ptr(xu), sigma, s1, 5.0, pkg.ptr(fused), n) == 0
    mc, mu, mo = (torch.empty(n, device=dev) for _ in range(3))
    pkg.lib.hd_sched_vcond(pkg.ptr(z), pkg.ptr(xc), sigma, pkg.ptr(mc), n)
    pkg.lib.hd_sched_vcond(pkg.ptr(z), pkg.ptr(xu), sigma, pkg.ptr(mu), n)
    pkg.lib.hd_sched_cfg_guided(pkg.ptr(mc), pkg.ptr(mu), 5.0, pkg.ptr(mo), n)
    pkg.lib.hd_sched_flow_match_step(pkg.ptr(z), pkg.ptr(mo), sigma, s1, pkg.ptr(chain), n)
    done(pkg, "sched")
    nan = chain.isnan()
    assert torch.equal(nan, fused.isnan())
    assert torch.equal(fused.view(torch.int16)[~nan], chain.view(torch.int16)[~nan])


@pytest.mark.parametrize("M,N,K,width", [(592, 4096, 2112, 144), (513, 4096, 2056, 144), (700, 4096, 3000, 176), (1280, 4096, 2112, 144),
                                         (1500, 4096, 2048, 176), (1000, 3072, 2240, 176), (1664, 3072, 2104, 144), (2400, 4096, 2048, 192),
                                         (2050, 3072, 2048, 192), (592, 4096, 256, 0)])
@pytest.mark.parametrize("epi", [1, 2])
def test_tiles_fitted_to_the_sms(pkg, dev, M, N, K, width, epi):
    """Tile widths between 128 and 256 columns (chosen where they make whole rounds of tiles) give the bits of 128-column
    tiles: partly filled last row and column tiles, ragged K, and a K too short for the form."""
    if pkg.lib.o1_sm_count() == 148:
        assert gemm_form(pkg, M, N, K, epi, 0) == ((3, width, 1) if width else (4, 96, 1))
    g = torch.Generator(device=dev).manual_seed(M + K)
    x, w, b, r = (torch.empty(s, device=dev).normal_(0, d, generator=g).bfloat16()
                  for s, d in (((M, K), 1.0), ((N, K), 0.05), ((N,), 0.5), ((M, N), 1.0)))
    ys = []
    for bn in (0, 128):
        y = torch.full((M + 1, N + 8), 777.0, dtype=torch.bfloat16, device=dev)
        rc = pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y), N + 8, M, N, K, epi, pkg.ptr(b), pkg.ptr(r), N, 0.0, bn)
        assert rc == 0, pkg.last_error()
        done(pkg, "gemm")
        assert (y[M:] == 777.0).all() and (y[:, N:] == 777.0).all(), "written beyond the matrix"
        ys.append(y)
    assert torch.equal(ys[0].view(torch.int16), ys[1].view(torch.int16))
    if epi == 1:
        check_linear_f64(ys[0][:M, :N], x, w, b, "fitted")
    assert pkg.lib.o1_device_error() == 0


def test_a_refused_launch_is_reported_once(pkg, dev):
    """A launch that CUDA refuses on the host (a grid of 70000 rows, the limit being 65535: no kernel runs) is an error of the
    call that asked for it and of no later one."""
    M, N, K = 70000, 9, 8
    x, w, y = (torch.zeros(s, dtype=torch.bfloat16, device=dev) for s in ((M, K), (N, K), (M, N)))
    assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y), N, M, N, K, 0, None, None, 0, 0.0, 0) != 0
    assert "launch" in pkg.last_error()
    pkg.lib.hd_cuda_clear_error()
    for rows in (4, 200):           # the row kernel and a norm, which look at CUDA's last error after their launch
        pkg.lib.hd_linear(pkg.ptr(x), pkg.ptr(w), None, pkg.ptr(y), rows, N, K, 1)
        pkg.check_cuda_errbuf("hd_linear after a refused launch")
    pkg.lib.hd_rmsnorm(pkg.ptr(x), pkg.ptr(w), pkg.ptr(y), 4, K, 1e-6)
    pkg.check_cuda_errbuf("hd_rmsnorm after a refused launch")
    assert float(torch.ones(8, device=dev).sum()) == 8.0


LATE = [("128 columns", 300, 512, 256, 1, 128, (1, 128)), ("256 columns", 300, 512, 256, 2, 256, (1, 256)),
        ("SwiGLU", 300, 512, 256, 3, 0, (1, 256)), ("pairs", 2304, 4096, 2048, 0, 0, (2, 256)),
        ("fitted, bias", 592, 4096, 2112, 1, 0, (3, 144)), ("fitted, residual", 592, 4096, 2112, 2, 0, (3, 144)),
        ("few, two K blocks a stage", 77, 1024, 512, 2, 0, (4, 32)), ("few, one K block a stage", 300, 3136, 256, 0, 0, (4, 32)),
        ("few, 96 columns", 520, 4304, 1152, 7, 0, (4, 96)), ("few, shared K", 520, 1152, 4304, 8, -1, (4, 128))]


@pytest.mark.parametrize("what,M,N,K,epi,bn,form", LATE, ids=[c[0] for c in LATE])
def test_gemm_after_a_late_failure_stores_nothing(pkg, dev, what, M, N, K, epi, bn, form):
    """A chained launch may start while the kernel before it still runs.  If that one then fails, the GEMM must not leave
    results behind: every form looks at the error word again before it stores."""
    from latefail import late_failure
    g = torch.Generator(device=dev).manual_seed(7)
    x, w, w2, b, r = (torch.empty(s, device=dev).normal_(0, d, generator=g).bfloat16()
                      for s, d in (((M, K), 1.0), ((N, K), 0.05), ((N, K), 0.05), ((N,), 0.5), ((M, N), 1.0)))
    y = torch.full((M, N), 777.0, dtype=torch.bfloat16, device=dev)

    def call():
        return pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), pkg.ptr(w2), pkg.ptr(y), N, M, N, K, epi, pkg.ptr(b), pkg.ptr(r), N, 0.0, bn)

    if pkg.lib.o1_sm_count() == 148:
        assert gemm_form(pkg, M, N, K, epi, bn)[:2] == form
    assert call() == 0, pkg.last_error()        # (a kernel's first launch loads it, which takes longer than the failure does)
    y.fill_(777.0)
    torch.cuda.synchronize()
    late_failure(pkg, 98)
    try:
        assert call() == 0, pkg.last_error()
        torch.cuda.synchronize()
        assert (y == 777.0).all(), f"{(y != 777.0).sum().item()} results stored after a failure"
    finally:
        torch.cuda.synchronize()
        assert pkg.lib.o1_device_error() == 98
    assert call() == 0
    done(pkg, "gemm")
    assert (y != 777.0).float().mean() > 0.99


def test_qkv_projection_after_a_late_failure_stores_nothing(pkg, dev):
    from latefail import late_failure
    M, qc, kc, K = 300, 512, 128, 256
    ld = qc + 2 * kc
    g = torch.Generator(device=dev).manual_seed(8)
    x, wq, wk, wv, nw = (torch.empty(s, device=dev).normal_(0, 0.1, generator=g).bfloat16() for s in ((M, K), (qc, K), (kc, K), (kc, K), (128,)))
    tab = torch.zeros(M, 128, device=dev)
    y = torch.full((M, ld), 777.0, dtype=torch.bfloat16, device=dev)
    def call():
        return pkg.lib.o1_gemm_qkv(pkg.ptr(x), K, pkg.ptr(wq), pkg.ptr(wk), pkg.ptr(wv), pkg.ptr(y), ld, M, qc, kc, K, pkg.ptr(nw),
                                   pkg.ptr(nw), pkg.ptr(tab), 1e-6)

    assert call() == 0, pkg.last_error()
    y.fill_(777.0)
    torch.cuda.synchronize()
    late_failure(pkg, 98)
    try:
        assert call() == 0
        torch.cuda.synchronize()
        assert (y == 777.0).all()
    finally:
        torch.cuda.synchronize()
        assert pkg.lib.o1_device_error() == 98


@pytest.mark.parametrize("M", [1, 2, 3, 4, 5, 6, 7, 9, 11])
@pytest.mark.parametrize("N,K,pad", [(9473, 1032, 0), (9473, 1032, 3), (515, 1024, 8), (515, 1024, 1), (13, 77, 0), (4097, 264, 5)])
def test_row_kernel_groups_and_pitches(pkg, dev, M, N, K, pad):
    """The row kernel with one to four rows to a warp, a last group that is not full, row pitches that leave the rows aligned
    and that do not, and a K without whole 16-byte pieces; nothing is written beside the result."""
    g = torch.Generator(device=dev).manual_seed(M + N + K + pad)
    x, w, b = (torch.empty(s, device=dev).normal_(0, d, generator=g).bfloat16() for s, d in (((M, K + pad), 1.0), ((N, K), 0.05), ((N,), 0.5)))
    ldy = N + 3
    y = torch.full((M + 1, ldy), 777.0, dtype=torch.bfloat16, device=dev)
    rc = pkg.lib.o1_gemm(pkg.ptr(x), K + pad, pkg.ptr(w), None, pkg.ptr(y), ldy, M, N, K, 1, pkg.ptr(b), None, 0, 0.0, 0)
    assert rc == 0, pkg.last_error()
    done(pkg, "rows")
    check_linear_f64(y[:M, :N], x[:, :K], w, b, "rows")
    assert (y[M:] == 777.0).all() and (y[:, N:] == 777.0).all(), "written beside the result"
    if pad % 8 == 0:       # a row is the same whatever it shares a warp with (where the rows' alignment is the same)
        one = torch.empty(M, N, dtype=torch.bfloat16, device=dev)
        for i in range(M):
            rc = pkg.lib.o1_gemm(C.c_void_p(x.data_ptr() + 2 * i * (K + pad)), K + pad, pkg.ptr(w), None,
                                 C.c_void_p(one.data_ptr() + 2 * i * N), N, 1, N, K, 1, pkg.ptr(b), None, 0, 0.0, 0)
            assert rc == 0, pkg.last_error()
        done(pkg, "rows")
        assert torch.equal(one.view(torch.int16), y[:M, :N].contiguous().view(torch.int16))


def test_gelu_is_rounded_once_for_every_bf16_value(pkg, dev):
    """The tanh form of GELU over all finite bf16 values: the result is the 64-bit value rounded to bf16, down to the smallest
    normal numbers (an fp32 evaluation may fall on the other side of a rounding boundary, but none of these values does; a form
    that computes 1 + tanh u misses about 150 of them, between -3 and -10)."""
    x = torch.arange(65536, dtype=torch.int32, device=dev).to(torch.int16).view(torch.bfloat16)
    y = torch.empty_like(x)
    pkg.lib.hd_vision_gelu(pkg.ptr(x), pkg.ptr(y), x.numel())
    done(pkg, "gelu")
    want = gelu_tanh_f64(x.double())
    normal = torch.isfinite(x) & (want.abs() > 2.0 ** -120)
    assert normal.sum() > 30000
    assert torch.equal(y[normal], want[normal].bfloat16())
    tiny = torch.isfinite(x) & ~normal & (x.abs() > 9)
    assert (y[tiny].double().abs() <= 2.0 ** -119).all()
    assert (y[x == float("inf")] == float("inf")).all() and y[torch.isnan(x)].isnan().all()


def test_every_kind_of_launch_reports_its_refusal(pkg, dev):
    """On a stream whose capture has become invalid CUDA refuses every launch, on the host; each entry point says so, and none
    leaves the error to the next call of an ordinary stream."""
    from cuda.bindings import driver
    M, N, K = 16, 128, 128
    x, w, y = (torch.zeros(s, dtype=torch.bfloat16, device=dev) for s in ((M, K), (N, K), (M, N)))
    f, cs = torch.zeros(3, M, device=dev), torch.zeros(M, 128, device=dev)
    p, lib = pkg.ptr, pkg.lib
    calls = {
        "rmsnorm, 32 threads a row": lambda: lib.hd_rmsnorm(p(x), p(w), p(y), M, K, 1e-6),
        "rmsnorm, 128 threads a row": lambda: lib.hd_rmsnorm(p(x), p(w), p(y), 1, 8 * K + 8 * M, 1e-6),
        "layernorm": lambda: lib.hd_vision_layernorm(p(x), p(w), None, p(y), M, K, 1e-6),
        "mrope": lambda: lib.o1_mrope_table(p(f), M, 5e6, p(cs)),
        "sched": lambda: lib.o1_sched_cfg_flow_step(p(x), p(x), p(x), 0.8, 0.7, 5.0, p(y), 256),
        "linear, tiles": lambda: lib.hd_linear(p(x), p(w), None, p(y), M, N, K, 1),
        "linear, rows": lambda: lib.hd_linear(p(x), p(w), None, p(y), 1, N, K, 1),
        "attention": lambda: lib.o1_flash_attention(p(x), K, p(x), K, p(x), K, p(y), K, M, 1, 1, 0, 0.1),
    }
    for call in calls.values():
        call()                       # (the kernels are loaded before the capture)
    done(pkg, "warm-up")
    stream = torch.cuda.Stream()
    h = stream.cuda_stream
    assert int(driver.cuStreamBeginCapture(h, driver.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL)[0]) == 0
    lib.o1_set_stream(C.c_void_p(h))
    said = {}
    try:
        assert int(driver.cuStreamSynchronize(h)[0]) != 0        # not allowed while capturing: the capture is invalid now
        for name, call in calls.items():
            lib.hd_cuda_clear_error()
            call()
            said[name] = lib.hd_cuda_last_error()
    finally:
        assert int(driver.cuStreamEndCapture(h)[0]) != 0
        pkg.use_torch_stream()
        lib.hd_cuda_clear_error()
    assert all(said.values()), said
    for call in calls.values():
        call()
        done(pkg, "afterwards")
    assert float(torch.ones(8, device=dev).sum()) == 8.0


@pytest.mark.parametrize("rows", [1, 3, 4, 5, 130, 4096, 4097, 5000])
@pytest.mark.parametrize("cols", [8, 128, 1024, 1032, 4096, 4104, 8192])
def test_norms_by_rows_and_columns(pkg, dev, rows, cols):
    """RMSNorm and LayerNorm over their forms' edges (a warp or a block to a row, few and many rows, weights requested early or
    late) against 64 bits; rows behind the last one stay as they are.  bf16 rounding is 2^-9 of a value, an fp32 sum of `cols`
    squares cols * 2^-24 at the most; with mean and variance as differences 2^-7 of the largest term covers both."""
    g = torch.Generator(device=dev).manual_seed(rows + cols)
    x, w, b = (torch.empty(s, device=dev).normal_(m, 0.5, generator=g).bfloat16() for s, m in (((rows, cols), 0.2), ((cols,), 1.0), ((cols,), 0.0)))
    y = torch.full((rows + 1, cols), 777.0, dtype=torch.bfloat16, device=dev)
    pkg.lib.hd_rmsnorm(pkg.ptr(x), pkg.ptr(w), pkg.ptr(y), rows, cols, 1e-6)
    done(pkg, "rmsnorm")
    xd = x.double()
    want = xd * w.double() * torch.rsqrt((xd * xd).mean(-1, keepdim=True) + 1e-6)
    assert ((y[:rows].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-9).all()
    assert (y[rows:] == 777.0).all()
    pkg.lib.hd_vision_layernorm(pkg.ptr(x), pkg.ptr(w), pkg.ptr(b), pkg.ptr(y), rows, cols, 1e-6)
    done(pkg, "layernorm")
    term = (xd - xd.mean(-1, keepdim=True)) * torch.rsqrt(xd.var(-1, unbiased=False, keepdim=True) + 1e-6) * w.double()
    want = term + b.double()
    assert ((y[:rows].double() - want).abs() <= 2.0 ** -7 * (term.abs() + b.double().abs())).all()
    assert (y[rows:] == 777.0).all()


@pytest.mark.parametrize("M", [8, 200])
def test_fused_swiglu_equals_the_pass_for_every_gate(pkg, dev, M):
    """gate | up + SwiGLU as one GEMM against the projections and hd_swiglu, for all bf16 gates: the epilogue's quotient is the
    IEEE one, far below zero, at infinities and at NaN too (where a warp holds one of those it divides for all its values)."""
    N, K = 65536, 64
    gates = torch.arange(N, dtype=torch.int32, device=dev).to(torch.int16).view(torch.bfloat16)
    order = torch.randperm(N, generator=torch.Generator().manual_seed(3)).to(dev)
    x = torch.zeros(M, K, dtype=torch.bfloat16, device=dev)
    x[:, 0] = 1
    for mixed in (False, True):        # neighbours alike, and every group with some extreme value in it
        wg, wu = torch.zeros(2, N, K, dtype=torch.bfloat16, device=dev)
        wg[:, 0] = gates[order] if mixed else gates
        wu[:, 0] = torch.linspace(-3, 3, N, device=dev).bfloat16()
        g, u, one, two = (torch.empty(M, N, dtype=torch.bfloat16, device=dev) for _ in range(4))
        for w, y in ((wg, g), (wu, u)):
            assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y), N, M, N, K, 0, None, None, 0, 0.0, 0) == 0
        assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(wg), pkg.ptr(wu), pkg.ptr(one), N, M, N, K, 3, None, None, 0, 0.0, 0) == 0
        pkg.lib.hd_swiglu(pkg.ptr(g), pkg.ptr(u), pkg.ptr(two), M * N)
        done(pkg, "swiglu")
        nan = two.isnan()
        assert torch.equal(nan, one.isnan())
        assert torch.equal(one.view(torch.int16)[~nan], two.view(torch.int16)[~nan])


@pytest.mark.parametrize("M,N,K,epi,bn,width", [(1280, 4096, 4096, 2, 0, 144), (1000, 3072, 4096, 1, 0, 176), (300, 4096, 3136, 2, 0, 128),
                                                (257, 4096, 3072, 0, 0, 128), (2600, 4096, 4160, 2, 0, 160), (300, 4096, 3072, 9, 0, 128),
                                                (2304, 1152, 4304, 8, -2, 144), (800, 1152, 4304, 8, -2, 96), (3000, 1152, 4304, 8, -2, 192),
                                                (520, 4608, 4608, 7, -2, 192), (1024, 4608, 4608, 7, -2, 256), (1000, 4104, 2056, 1, -2, 112),
                                                (700, 4312, 2048, 7, -2, 192), (1200, 4304, 1152, 7, -2, 160), (1100, 1152, 1152, 8, -2, 96),
                                                (300, 4096, 3080, 2, 0, 128), (592, 4096, 3072, 0, 0, 176), (3000, 4096, 3080, 7, 0, 176),
                                                (1700, 4096, 3072, 9, 0, 208), (2242, 4096, 3072, 8, 0, 256), (1700, 2176, 3136, 8, 0, 224),
                                                (257, 4608, 4608, 7, -2, 128), (1025, 1152, 1152, 8, -2, 96)])
def test_pair_tiles_of_any_width(pkg, dev, M, N, K, epi, bn, width):
    """CTA pairs with a width chosen by the rounds of tiles give the bits of 128-column tiles: partly filled last row and column
    tiles, an odd number of row tiles, a ragged N and K, every epilogue."""
    if pkg.lib.o1_sm_count() == 148:
        assert gemm_form(pkg, M, N, K, epi, bn) == (1 if width == 128 and bn == 0 else 3, width, 2)
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    x, w, b, r = (torch.empty(s, device=dev).normal_(0, d, generator=g).bfloat16()
                  for s, d in (((M, K), 1.0), ((N, K), 0.05), ((N,), 0.5), ((M, N), 1.0)))
    ys = []
    for force in (bn, 128):
        y = torch.full((M + 1, N + 8), 777.0, dtype=torch.bfloat16, device=dev)
        rc = pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y), N + 8, M, N, K, epi, pkg.ptr(b), pkg.ptr(r), N, 0.0, force)
        assert rc == 0, pkg.last_error()
        done(pkg, "gemm")
        assert (y[M:] == 777.0).all() and (y[:, N:] == 777.0).all(), "written beyond the matrix"
        ys.append(y)
    assert torch.equal(ys[0].view(torch.int16), ys[1].view(torch.int16))
    check_epilogue_f64(ys[0][:M, :N], x, w, b, r, epi, "pair tiles")
    assert pkg.lib.o1_device_error() == 0


@pytest.mark.parametrize("M,N,K,epi", [(520, 4608, 4608, 7), (2304, 1152, 4304, 8), (1100, 4304, 1152, 7), (77, 1152, 1152, 8)])
def test_the_towers_linears_keep_their_bits_without_clusters(pkg, dev, M, N, K, epi):
    """force_bn -2 (the vision tower's linears) in pair mode 0: one CTA per tile, and where no K is shared the same bits."""
    g = torch.Generator(device=dev).manual_seed(M)
    x, w, b, r = (torch.empty(s, device=dev).normal_(0, d, generator=g).bfloat16()
                  for s, d in (((M, K), 1.0), ((N, K), 0.05), ((N,), 0.5), ((M, N), 1.0)))
    ys = []
    try:
        for mode in (1, 0):
            pkg.lib.o1_gemm_pair_mode(mode)
            form = gemm_form(pkg, M, N, K, epi, -2)
            assert form[2] == 1 if mode == 0 else form[2] <= 2      # (a shared K takes four CTAs and more)
            y = torch.empty(M, N, dtype=torch.bfloat16, device=dev)
            assert pkg.lib.o1_gemm(pkg.ptr(x), K, pkg.ptr(w), None, pkg.ptr(y), N, M, N, K, epi, pkg.ptr(b), pkg.ptr(r), N, 0.0, -2) == 0
            done(pkg, "gemm")
            ys.append(y)
    finally:
        pkg.lib.o1_gemm_pair_mode(1)
    assert torch.equal(ys[0].view(torch.int16), ys[1].view(torch.int16))
