"""Load-time LoRA merge (hd_lora_merge_gpu, o1.c include/hd_lora.h:71-79) against the FP32 restatement
of the documented contract W' = bf16(f32(W) + multiplier*alpha/rank * up@down) (hd_lora.h:10-14,
lora_merge.cu:26-33): the merged bf16 weights must be bit-identical except where the FP32 sum lands on
a rounding tie (counted, must be a vanishing fraction).

The reference's own GPU merge is NOT run here: its cublasSgemm call passes the row-major up-chunk
with leading dimension C instead of rank (lora_merge.cu:86-93), which reads beyond the adapter
buffer whenever out_dim != rank."""
import ctypes as C

import numpy as np
import pytest
import torch

import parity
from parity import np_ptr, seeded_bf16, torch_to_u16, u16_to_torch

pytestmark = pytest.mark.gpu


def check_merged(got, ref, w0, max_frac=2e-4):
    """Bit-identical except on rounding ties: where the two FP32 sums round to different bf16 values
    they must be neighbours at the scale of the operands (one bf16 ulp of max(|W|, |W'|)), and such
    elements must be a vanishing fraction."""
    g, r_, w = (parity.bf16_to_f32_np(a).astype(np.float64) for a in (got, ref, w0))
    neq = got != ref
    assert neq.mean() <= max_frac, f"{neq.mean():.2e} of the merged weights differ"
    ulp = np.maximum(np.abs(w), np.abs(r_)) * 2.0 ** -7 + 1e-30
    assert (np.abs(g - r_) <= ulp).all()


def entry(pkg, w, up, down, R, K, N, alpha, mult):
    e = pkg.LoraEntry()
    e.rank, e.in_dim, e.out_dim, e.alpha, e.multiplier = R, K, N, alpha, mult
    e.down_dev, e.up_dev, e.base_dev = down.data_ptr(), up.data_ptr(), w.data_ptr()
    return e


@pytest.mark.parametrize("N,K,R", [(1024, 4096, 64), (4096, 1024, 16), (384, 256, 8), (100, 72, 4), (512, 1280, 200)])
def test_lora_merge(pkg, orc, dev, N, K, R):
    w0 = seeded_bf16((N, K), 51, 0.0, 0.02)
    up = np.empty((N, R), dtype=np.float32)
    down = np.empty((R, K), dtype=np.float32)
    orc.orc_fill_normal_f32(np_ptr(up), up.size, 52, 0.0, 0.01)
    orc.orc_fill_normal_f32(np_ptr(down), down.size, 53, 0.0, 0.01)
    alpha, mult = float(R), 1.0
    wd = u16_to_torch(w0, dev)
    ents = (pkg.LoraEntry * 1)(entry(pkg, wd, torch.from_numpy(up).to(dev), torch.from_numpy(down).to(dev), R, K, N,
                                     alpha, mult))
    upd, dnd = torch.from_numpy(up).to(dev), torch.from_numpy(down).to(dev)
    ents[0].up_dev, ents[0].down_dev = upd.data_ptr(), dnd.data_ptr()
    rc = pkg.lib.hd_lora_merge_gpu(ents, 1, None)
    torch.cuda.synchronize()
    assert rc == 0, pkg.last_error()
    ref = w0.copy()
    orc.orc_lora_merge(np_ptr(ref), np_ptr(up), np_ptr(down), N, K, R, mult * alpha / R)
    got = torch_to_u16(wd)
    assert (got != w0).mean() > 0.01, "merge changed nothing"
    # 9 x 256 exact products per element are summed by the tensor core in its own order: more tie flips than at rank 64
    check_merged(got, ref, w0, max_frac=2e-4 if R <= 64 else 2e-3)


def test_lora_sequential_adapters_and_errors(pkg, orc, dev):
    """Two adapters on one weight: one bf16 rounding per adapter, in order (contract sequential-bf16-v1)."""
    N, K, R = 256, 512, 8
    w0 = seeded_bf16((N, K), 61, 0.0, 0.02)
    ups = [np.empty((N, R), dtype=np.float32) for _ in range(2)]
    dns = [np.empty((R, K), dtype=np.float32) for _ in range(2)]
    for i in range(2):
        orc.orc_fill_normal_f32(np_ptr(ups[i]), ups[i].size, 70 + i, 0.0, 0.05)
        orc.orc_fill_normal_f32(np_ptr(dns[i]), dns[i].size, 80 + i, 0.0, 0.05)
    wd = u16_to_torch(w0, dev)
    keep = [torch.from_numpy(a).to(dev) for a in ups + dns]
    ents = (pkg.LoraEntry * 2)(entry(pkg, wd, keep[0], keep[2], R, K, N, 4.0, 1.0),
                               entry(pkg, wd, keep[1], keep[3], R, K, N, 8.0, 0.5))
    assert pkg.lib.hd_lora_merge_gpu(ents, 2, None) == 0
    torch.cuda.synchronize()
    ref = w0.copy()
    orc.orc_lora_merge(np_ptr(ref), np_ptr(ups[0]), np_ptr(dns[0]), N, K, R, 1.0 * 4.0 / R)
    orc.orc_lora_merge(np_ptr(ref), np_ptr(ups[1]), np_ptr(dns[1]), N, K, R, 0.5 * 8.0 / R)
    check_merged(torch_to_u16(wd), ref, w0, 5e-4)
    bad = (pkg.LoraEntry * 1)(entry(pkg, wd, keep[0], keep[2], 0, K, N, 4.0, 1.0))
    assert pkg.lib.hd_lora_merge_gpu(bad, 1, None) == 5          # HD_ERR_MISMATCH


def test_lora_merge_against_the_reference_python_contract(pkg, dev, golden):
    """hd_lora_merge_gpu against weights merged by the reference's own Python (merge_linear of o1.c
    tools/lora/tests/test_lora_formula.py:20 + the bf16 rounding of tools/lora/merge_gguf.py:44-49,164-171);
    fixture tests/golden/lora_ref.npz, including a multiplier != 1 and a negative one."""
    import os
    g = np.load(os.path.join(golden, "lora_ref.npz"))
    for i in range(int(g["n_cases"])):
        N, K, R, alpha, mult = g[f"c{i}_meta"]
        N, K, R = int(N), int(K), int(R)
        w0 = np.ascontiguousarray(g[f"c{i}_w"])
        wd = u16_to_torch(w0, dev)
        upd = torch.from_numpy(np.ascontiguousarray(g[f"c{i}_up"])).to(dev)
        dnd = torch.from_numpy(np.ascontiguousarray(g[f"c{i}_down"])).to(dev)
        ents = (pkg.LoraEntry * 1)(entry(pkg, wd, upd, dnd, R, K, N, float(alpha), float(mult)))
        assert pkg.lib.hd_lora_merge_gpu(ents, 1, None) == 0, pkg.last_error()
        torch.cuda.synchronize()
        check_merged(torch_to_u16(wd), g[f"c{i}_merged"], w0, max_frac=1e-3)


def merged_f64(w0, up, down, s):
    return w0.double() + s * (up.double() @ down.double())


@pytest.mark.parametrize("shapes", [
    [(8, 128, 1)],                                            # one tile, eight of its rows
    [(127, 256, 15), (129, 128, 16), (128, 384, 17)],         # a row short of a tile, a row over; one and two MMA steps
    [(256, 128, 63), (200, 256, 64), (130, 128, 65)],         # around one chunk of ranks
    [(300, 640, 129), (64, 128, 192), (1, 128, 8)],           # several chunks; the last one runs without tensor cores
    [(128 * (i % 3 + 1), 128 * (i % 4 + 1), 4 + i) for i in range(37)],   # more targets than one launch takes
    [(20000, 128, 8)],                                        # every SM walks a column of row blocks
], ids=["one", "rows", "rank", "chunks", "many", "tall"])
@pytest.mark.parametrize("shift", [0, 1])
def test_lora_merge_tile_edges(pkg, dev, shapes, shift):
    """Edges of the merge kernel's tiles, rank chunks and launch groups against 64 bits, all targets in one call.  shift:
    adapters that begin 4 bytes off a 16-byte boundary.  The FP32 sum of 6 R products is within R * 2^-22 of the exact
    delta's magnitude sum, so a weight may differ from the rounded 64-bit value only where that bound crosses a rounding
    boundary, and then by one bf16 step."""
    g = torch.Generator(device=dev).manual_seed(len(shapes) * 2 + shift)
    ents, keep = (pkg.LoraEntry * len(shapes))(), []
    for e, (n, k, r) in zip(ents, shapes):
        w = torch.empty(n + 1, k, device=dev).normal_(0, 0.02, generator=g).bfloat16()      # a canary row behind
        up = torch.empty(n * r + shift, device=dev).normal_(0, 0.05, generator=g)[shift:]
        down = torch.empty(r * k + shift, device=dev).normal_(0, 0.05, generator=g)[shift:]
        ee = entry(pkg, w, up, down, r, k, n, 0.7 * r, -1.3)
        C.memmove(C.byref(e), C.byref(ee), C.sizeof(e))
        keep.append((w, w.clone(), up, down))
    assert pkg.lib.hd_lora_merge_gpu(ents, len(shapes), None) == 0, pkg.last_error()
    assert pkg.lib.o1_device_error() == 0
    for (n, k, r), (w, w0, up, down) in zip(shapes, keep):
        u, d = up.view(n, r), down.view(r, k)
        want = merged_f64(w0[:n], u, d, 0.7 * -1.3)
        bound = (u.abs().double() @ d.abs().double() + w0[:n].abs().double()) * (r + 4) * 2.0 ** -22
        # rounding is monotonic: the result lies between the rounded ends of the interval around the exact value
        lo, hi = (want - bound).bfloat16().double(), (want + bound).bfloat16().double()
        got = w[:n].double()
        assert ((got >= lo) & (got <= hi)).all(), (n, k, r, ((got < lo) | (got > hi)).sum().item())
        assert torch.equal(w[n:].view(torch.int16), w0[n:].view(torch.int16)), "rows beyond N were written"


def test_lora_merge_reports_a_device_that_has_failed(pkg, dev):
    """After a kernel ran into its wait limit the merge kernel does nothing, and the call says so; once the error word has been
    read, the same call merges."""
    from latefail import late_failure
    n, k, r = 256, 128, 8
    g = torch.Generator(device=dev).manual_seed(3)
    w = torch.empty(n, k, device=dev).normal_(0, 0.02, generator=g).bfloat16()
    up = torch.empty(n, r, device=dev).normal_(0, 0.05, generator=g)
    down = torch.empty(r, k, device=dev).normal_(0, 0.05, generator=g)
    w0 = w.clone()
    ents = (pkg.LoraEntry * 1)(entry(pkg, w, up, down, r, k, n, 1.0, 1.0))
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    late_failure(pkg, 99)
    try:
        assert pkg.lib.hd_lora_merge_gpu(ents, 1, stream) == 8            # HD_ERR_RUNTIME
        assert "error word" in pkg.last_error()
        assert torch.equal(w.view(torch.int16), w0.view(torch.int16))
    finally:
        assert pkg.lib.o1_device_error() == 99       # reads and clears the word
    pkg.lib.hd_cuda_clear_error()
    assert pkg.lib.hd_lora_merge_gpu(ents, 1, stream) == 0
    assert not torch.equal(w.view(torch.int16), w0.view(torch.int16))


def test_lora_merge_without_tiles_can_be_captured(pkg, dev):
    """Targets that take the simple kernel (in_dim no multiple of 128) need neither a wait nor host work between their
    launches: the call can be captured, and each replay merges the adapter once more."""
    n, k, r = 40, 100, 4
    g = torch.Generator(device=dev).manual_seed(5)
    w = torch.empty(n, k, device=dev).normal_(0, 0.02, generator=g).bfloat16()
    up = torch.empty(n, r, device=dev).normal_(0, 0.05, generator=g)
    down = torch.empty(r, k, device=dev).normal_(0, 0.05, generator=g)
    w0 = w.clone()
    ents = (pkg.LoraEntry * 1)(entry(pkg, w, up, down, r, k, n, 1.0, 1.0))
    eager = []
    for _ in range(2):
        assert pkg.lib.hd_lora_merge_gpu(ents, 1, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
        eager.append(w.clone())
    w.copy_(w0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert pkg.lib.hd_lora_merge_gpu(ents, 1, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0, pkg.last_error()
    assert torch.equal(w.view(torch.int16), w0.view(torch.int16))
    for want in eager:
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(w.view(torch.int16), want.view(torch.int16))
