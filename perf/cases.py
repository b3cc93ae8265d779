"""What the performance of this framework is measured on: single calls, layers and whole steps through the public
entry points, with the sizes of the model (32 / 8 heads of 128, width 4096, MLP 12288, 36 blocks; vision tower of 27
blocks of width 1152), of the benchmark's workloads and of ordinary requests between them.

Kinds of case
  linear   hd_linear: y = x W^T + b, from the single row of the timestep MLP to a few thousand token rows
  sched    o1_sched_cfg_flow_step: guidance and the flow-match Euler update of a latent
  sdpa     hd_sdpa_execute_split: prefix-causal attention on head-major q / k / v
  block    Engine.block: one decoder block
  step     Engine.denoise_step_cfg[_branches]: a whole guided step (two forwards of 36 blocks and the update)
  edit     Engine.forward with visual conditioning: the 36-block forward of an image-editing request
  vision   hd_vision_forward: the tower that encodes an edit request's reference images
  lora     hd_lora_merge_gpu: a low-rank adapter merged into the linears of one decoder block, in place
"""
import ctypes as C
import math

import torch

from __graft_entry__ import load_package

HIDDEN, HEADS, KV_HEADS, D, FF, PATCH, XE = 4096, 32, 8, 128, 12288, 3072, 1024
LAYERS, VOCAB, TMS_ID, IMAGE_PAD, VISION_START, BOI = 36, 151936, 151673, 151655, 151652, 151669
QKV = (HEADS + 2 * KV_HEADS) * D
# (out, in) of the linear layers a program calls through hd_linear: the decoder's, the embedders' and the head's
LINEARS = [(4096, 4096), (1024, 4096), (12288, 4096), (4096, 12288), (4096, 256), (1024, 3072), (4096, 1024),
           (3072, 4096), (24576, 4096)]
LORA_TARGETS = {"attention": ("q_proj", "k_proj", "v_proj", "o_proj"),
                "all": ("q_proj", "k_proj", "v_proj", "o_proj", "gate_proj", "up_proj", "down_proj")}
VH, VHEADS, VD, VFF, VM, VOUT, VPATCH, VDEPTH = 1152, 16, 72, 4304, 4608, 4096, 1536, 27


def listed():
    return [
        # second layer of the timestep MLP: one row, once per forward -- the smallest call there is
        {"name": "linear_timestep", "kind": "linear", "m": 1, "n": 4096, "k": 4096},
        # a prompt's text rows through one projection: few rows, an odd count
        {"name": "linear_text", "kind": "linear", "m": 77, "n": 4096, "k": 4096},
        # the latent update of a 4096 x 4096 image (16384 tokens of 32 x 32 pixels)
        {"name": "sched_16384", "kind": "sched", "tokens": 16384},
        # attention of a portrait image (48 x 64 tokens) behind a prompt of 85 tokens: nothing is a multiple of a tile
        {"name": "sdpa_3157", "kind": "sdpa", "s": 3157, "ar": 84},
        # one block at 1024^2, 2048^2 and 4096^2 pixels behind the usual 256 tokens of text
        {"name": "block_1280", "kind": "block", "text": 256, "gh": 32, "gw": 32},
        {"name": "block_4352", "kind": "block", "text": 256, "gh": 64, "gw": 64},
        {"name": "block_16640", "kind": "block", "text": 256, "gh": 128, "gw": 128},
        # a whole guided step of a 512^2 image: the preview size, where latency counts most
        {"name": "step_512px", "kind": "step", "text": 40, "text_u": 40, "gh": 16, "gw": 16},
        # the forward of an edit at 1024^2 with one reference image (its tower rows and its pixel tokens)
        {"name": "edit_1024px", "kind": "edit", "text": 60, "gh": 32, "gw": 32, "refs": 1, "rh": 32, "rw": 32,
         "ch": 13, "cw": 10},
        # the tower on a 416 x 320 reference image, and on a 1024 x 1024 one
        {"name": "vision_520", "kind": "vision", "gh": 26, "gw": 20},
        {"name": "vision_4096", "kind": "vision", "gh": 64, "gw": 64},
        # a rank-64 adapter for every linear of a block
        {"name": "lora_block", "kind": "lora", "rank": 64, "targets": "all"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "sched", "sdpa", "block", "block", "step", "edit", "vision", "vision", "lora"])
    if kind == "linear":
        n, k = rng.choice(LINEARS)
        return {"kind": kind, "m": _log(rng, 1, 4096), "n": n, "k": k}
    if kind == "sched":
        return {"kind": kind, "tokens": _log(rng, 64, 16384)}
    if kind == "sdpa":
        s = _log(rng, 130, 8200)
        return {"kind": kind, "s": s, "ar": rng.randint(0, min(s, 600))}
    if kind == "block":
        g = _log(rng, 6, 100)
        return {"kind": kind, "text": _log(rng, 8, 500), "gh": g, "gw": rng.randint(max(4, g // 2), min(128, 2 * g))}
    if kind == "step":
        t = _log(rng, 12, 256)
        return {"kind": kind, "text": t, "text_u": rng.choice([t, rng.randint(6, t)]), "gh": rng.randint(8, 28), "gw": rng.randint(8, 28)}
    if kind == "edit":
        return {"kind": kind, "text": rng.randint(20, 200), "gh": rng.randint(16, 30), "gw": rng.randint(16, 30),
                "refs": rng.randint(1, 2), "rh": rng.randint(8, 22), "rw": rng.randint(8, 22), "ch": rng.randint(4, 16),
                "cw": rng.randint(4, 16)}
    if kind == "vision":
        return {"kind": kind, "gh": 2 * rng.randint(3, 32), "gw": 2 * rng.randint(3, 32)}
    return {"kind": "lora", "rank": rng.choice([4, 8, 16, 32, 48, 64, 96, 128]), "targets": rng.choice(["attention", "all"])}


# ------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 131 + salt)
    return g


def _normal(shape, g, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return torch.empty(shape, dtype=torch.float32, device="cuda").normal_(mean, std, generator=g).to(dtype)


def _text_ids(n, seed):
    g = torch.Generator().manual_seed(int(seed))
    ids = torch.randint(0, 151000, (n,), generator=g, dtype=torch.int64)
    ids[-1] = TMS_ID
    return ids


def _weights(pkg, layers, seed, **dims):
    # norm weights around 1, matrices N(0, 0.02^2): attention logits and MLP activations of ordinary size
    return pkg.Weights(n_layers=layers, seed=seed, weight_set="B", device="cuda:0", **dims)


def _edit_sequence(pkg, case, seed):
    """Token ids, positions, causal prefix and the mask of the rows that take the tower's output."""
    k, cond = case["refs"], case["ch"] * case["cw"]
    text = _text_ids(case["text"] + k * (1 + cond) + 2, seed).tolist()
    at = 4
    for _ in range(k):
        text[at] = VISION_START
        text[at + 1:at + 1 + cond] = [IMAGE_PAD] * cond
        at += 1 + cond
    text[-2] = BOI
    refs = [(case["rh"] * case["rw"], case["rh"], case["rw"], case["ch"], case["cw"])] * k
    ids, pos, ar = pkg.seq_ref(text, refs, case["gh"], case["gw"])
    mask = torch.zeros(ids.numel(), dtype=torch.uint8)
    mask[:len(text)] = (ids[:len(text)] == IMAGE_PAD).to(torch.uint8)
    return ids, pos, ar, mask, len(text)


def _vision_shapes():
    out = [("w", (VH, VPATCH)), ("b", (VH,)), ("w", (2304, VH))]
    for _ in range(VDEPTH):
        out += [("ln", (VH,)), ("b", (VH,)), ("ln", (VH,)), ("b", (VH,)), ("w", (3 * VH, VH)), ("b", (3 * VH,)),
                ("w", (VH, VH)), ("b", (VH,)), ("w", (VFF, VH)), ("b", (VFF,)), ("w", (VH, VFF)), ("b", (VH,))]
    for nd in (VH, VM, VM, VM):
        out += [("ln", (nd,)), ("b", (nd,)), ("w", (VM, VM)), ("b", (VM,)), ("w", (VOUT, VM)), ("b", (VOUT,))]
    return out


def prepare(case, seed):
    torch.cuda.set_device(0)
    pkg = load_package()
    pkg.use_torch_stream()
    g = _gen(seed)
    kind = case["kind"]
    s = {"case": case, "pkg": pkg, "lib": pkg.lib}
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        s["x"], s["w"], s["b"] = _normal((m, k), g), _normal((n, k), g, 0.02), _normal((n,), g, 0.02)
        s["y"] = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    elif kind == "sched":
        shape = (case["tokens"], PATCH)
        s["z"], s["xc"], s["xu"] = _normal(shape, g, 4.0), _normal(shape, g), _normal(shape, g)
        s["z_next"] = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
    elif kind == "sdpa":
        n = case["s"]
        # q and k as they leave the per-head norm: elements of unit size, so logits of a few units
        s["q"], s["k"], s["v"] = _normal((HEADS, n, D), g), _normal((KV_HEADS, n, D), g), _normal((KV_HEADS, n, D), g)
        s["out"] = torch.empty(HEADS, n, D, dtype=torch.bfloat16, device="cuda")
        plan = C.c_void_p()
        rc = pkg.lib.hd_sdpa_create_split(C.byref(plan), 1, HEADS, KV_HEADS, n, case["ar"], D, D ** -0.5)
        assert rc == 0, pkg.last_error()
        s["plan"] = plan
    elif kind == "block":
        n = case["text"] + case["gh"] * case["gw"]
        pos, ar = pkg.seq_t2i(case["text"], case["gh"], case["gw"])
        s["weights"] = _weights(pkg, 1, seed, vocab=64)
        s["engine"] = pkg.Engine(s["weights"], case["text"], n - case["text"], ar_len=ar)
        s["x"], s["pos"], s["ar"] = _normal((n, HIDDEN), g), pos.cuda(), ar
    elif kind == "step":
        t, img = case["text"], case["gh"] * case["gw"]
        s["weights"] = _weights(pkg, LAYERS, seed)
        s["cond"], s["uncond"] = [
            (_text_ids(n, seed + i).cuda(), p.cuda(), ar)
            for i, n in enumerate((t, case["text_u"])) for p, ar in [pkg.seq_t2i(n, case["gh"], case["gw"])]]
        s["engine"] = pkg.Engine(s["weights"], t, img, ar_len=s["cond"][2])
        s["z"] = _normal((img, PATCH), g, 4.0)
        s["z_next"] = torch.empty_like(s["z"])
    elif kind == "edit":
        ids, pos, ar, mask, t = _edit_sequence(pkg, case, seed)
        img, v = ids.numel() - t, int(mask.sum())
        s["weights"] = _weights(pkg, LAYERS, seed)
        s["engine"] = pkg.Engine(s["weights"], t, img, ar_len=ar)
        s["ids"], s["pos"], s["ar"], s["t"] = ids.cuda(), pos.cuda(), ar, t
        s["vin"] = _normal((img, PATCH), g)
        s["visual"] = (mask.cuda(), _normal((v, HIDDEN), g), tuple(_normal((v, HIDDEN), g, 0.5) for _ in range(3)))
        s["out"] = torch.empty(ids.numel(), PATCH, dtype=torch.bfloat16, device="cuda")
    elif kind == "vision":
        gh, gw = case["gh"], case["gw"]
        n, lib = gh * gw, pkg.lib
        s["tensors"] = [_normal(sh, g, 0.02, 1.0 if what == "ln" else 0.0) for what, sh in _vision_shapes()]
        s["binding"] = pkg.VisionBinding(*[t.data_ptr() for t in s["tensors"]])
        s["px"] = _normal((n, VPATCH), g)
        s["emb"] = torch.empty(n // 4, VOUT, dtype=torch.bfloat16, device="cuda")
        s["ds"] = torch.empty(3, n // 4, VOUT, dtype=torch.bfloat16, device="cuda")
        s["dsp"] = (C.c_void_p * 3)(*[s["ds"][j].data_ptr() for j in range(3)])
        s["space"] = torch.empty(lib.hd_vision_workspace_bytes(n), dtype=torch.uint8, device="cuda")
        s["tables"] = torch.empty(lib.hd_vision_tables_bytes(n), dtype=torch.uint8, device="cuda")
        s["ws"] = pkg.VisionWorkspace()
        s["ws"].patch_out, s["ws"].tables, s["ws"].tables_n = s["space"].data_ptr(), s["tables"].data_ptr(), -1
        assert lib.hd_vision_prepare_tables(C.byref(s["ws"]), n, gh, gw) == 0, pkg.last_error()
    else:
        names, r = LORA_TARGETS[case["targets"]], case["rank"]
        s["w"], s["up"], s["down"] = [], [], []
        s["entries"] = (pkg.LoraEntry * len(names))()
        for e, name in zip(s["entries"], names):
            n, k = pkg.tensor_shape(name)
            w, up, down = _normal((n, k), g, 0.02), _normal((n, r), g, 0.05, dtype=torch.float32), _normal((r, k), g, 0.02, dtype=torch.float32)
            e.rank, e.in_dim, e.out_dim, e.alpha, e.multiplier = r, k, n, float(r), 0.8
            e.up_dev, e.down_dev, e.base_dev = up.data_ptr(), down.data_ptr(), w.data_ptr()
            s["w"].append(w), s["up"].append(up), s["down"].append(down)
    return s


SIGMA, SIGMA_NEXT, GUIDANCE, EDIT_T = 0.857, 0.836, 5.0, 0.3


def run(s):
    pkg, lib, case = s["pkg"], s["lib"], s["case"]
    kind, p = case["kind"], s["pkg"].ptr
    if kind == "linear":
        lib.hd_linear(p(s["x"]), p(s["w"]), p(s["b"]), p(s["y"]), case["m"], case["n"], case["k"], 1)
        pkg.check_cuda_errbuf("hd_linear")
        return s["y"]
    if kind == "sched":
        rc = lib.o1_sched_cfg_flow_step(p(s["z"]), p(s["xc"]), p(s["xu"]), SIGMA, SIGMA_NEXT, GUIDANCE, p(s["z_next"]), s["z"].numel())
        assert rc == 0, pkg.last_error()
        return s["z_next"]
    if kind == "sdpa":
        rc = lib.hd_sdpa_execute_split(s["plan"], p(s["q"]), p(s["k"]), p(s["v"]), p(s["out"]), None)
        assert rc == 0, pkg.last_error()
        return s["out"]
    if kind == "block":
        return s["engine"].block(s["x"], s["pos"], 0)
    if kind == "step":
        e = s["engine"]
        if case["text_u"] == case["text"]:
            e.denoise_step_cfg(s["cond"][0], s["uncond"][0], s["cond"][1], s["z"], SIGMA, SIGMA_NEXT, GUIDANCE, s["z_next"])
        else:
            e.denoise_step_cfg_branches(s["cond"], s["uncond"], s["z"], SIGMA, SIGMA_NEXT, GUIDANCE, s["z_next"])
        # both predictions, each [rows of its branch, 3072], lie behind one another in the engine's buffer
        rows = case["text"] + case["text_u"] + 2 * case["gh"] * case["gw"]
        return {"z_next": s["z_next"], "x_pred": e.xp[:rows * PATCH].view(rows, PATCH)}
    if kind == "edit":
        return s["engine"].forward(s["ids"], s["pos"], s["vin"], EDIT_T, out=s["out"], visual=s["visual"])
    if kind == "vision":
        n = case["gh"] * case["gw"]
        rc = lib.hd_vision_forward(C.byref(s["binding"]), C.byref(s["ws"]), p(s["px"]), n, case["gh"], case["gw"], p(s["emb"]), C.byref(s["dsp"]))
        assert rc == 0, pkg.last_error()
        return {"image_embeds": s["emb"], "deepstack": s["ds"]}
    rc = lib.hd_lora_merge_gpu(s["entries"], len(s["entries"]), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, pkg.last_error()
    return s["w"]


# ------------------------------------------------------------------ what a pass cannot do without
def _attn_flops(s, ar, heads, d):
    return 4.0 * heads * d * (0.5 * ar * (ar + 1.0) + (s - ar) * float(s))


BLOCK_PARAMS = HIDDEN * QKV + HIDDEN * HIDDEN + 3 * HIDDEN * FF


def _forward_work(text, img, ar):
    s = text + img
    flops = LAYERS * (2.0 * s * BLOCK_PARAMS + _attn_flops(s, ar, HEADS, D)) + 2.0 * img * (PATCH * XE + XE * HIDDEN) + 2.0 * s * HIDDEN * PATCH
    params = LAYERS * BLOCK_PARAMS + PATCH * XE + XE * HIDDEN + HIDDEN * PATCH + HIDDEN * HIDDEN
    return flops, 2.0 * params, 2.0 * PATCH * (img + s)


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2.0 * (m * k + n * k + m * n), "flops": 2.0 * m * n * k}
    if kind == "sched":
        return {"bytes": 8.0 * case["tokens"] * PATCH, "flops": 0.0}
    if kind == "sdpa":
        s = case["s"]
        return {"bytes": 2.0 * s * D * (2 * HEADS + 2 * KV_HEADS), "flops": _attn_flops(s, case["ar"], HEADS, D)}
    if kind == "block":
        s = case["text"] + case["gh"] * case["gw"]
        return {"bytes": 2.0 * (BLOCK_PARAMS + 2 * s * HIDDEN), "flops": 2.0 * s * BLOCK_PARAMS + _attn_flops(s, case["text"] - 1, HEADS, D)}
    if kind == "step":
        img = case["gh"] * case["gw"]
        fc, wb, ac = _forward_work(case["text"], img, case["text"] - 1)
        fu, _, au = _forward_work(case["text_u"], img, case["text_u"] - 1)
        return {"bytes": wb + ac + au + 4.0 * img * PATCH, "flops": fc + fu}
    if kind == "edit":
        t = case["text"] + case["refs"] * (1 + case["ch"] * case["cw"]) + 2
        img = case["gh"] * case["gw"] + case["refs"] * case["rh"] * case["rw"]
        f, wb, a = _forward_work(t, img, t - 1)
        return {"bytes": wb + a + 8.0 * HIDDEN * case["refs"] * case["ch"] * case["cw"], "flops": f}
    if kind == "vision":
        n = case["gh"] * case["gw"]
        m = n // 4
        block, merger = VH * 4 * VH + 2 * VH * VFF, VM * VM + VM * VOUT
        return {"bytes": 2.0 * (VDEPTH * block + 4 * merger + VH * VPATCH + n * VPATCH + 4 * m * VOUT),
                "flops": 2.0 * n * (VDEPTH * block + VH * VPATCH) + VDEPTH * _attn_flops(n, 0, VHEADS, VD) + 8.0 * m * merger}
    r, by, fl = case["rank"], 0.0, 0.0
    for name in LORA_TARGETS[case["targets"]]:
        n, k = load_package().tensor_shape(name)
        by, fl = by + 4.0 * n * k + 4.0 * r * (n + k), fl + 2.0 * r * n * k
    return {"bytes": by, "flops": fl}


def tolerance(case):
    # One bf16 rounding is 1.7e-3 in the 2-norm.  linear and lora round a 32-bit sum once at the end: another order of
    # the sum moves few results to the next value.  A layer adds the roundings of its intermediate tensors (error
    # against 64 bits 2e-3 to 5e-3), the tower's 27 blocks reach 1.5e-2, the 36 blocks of a forward 3.6e-2 to 4.6e-2.
    return {"linear": {"rel": 5e-4}, "sched": {"rel": 1e-4}, "sdpa": {"rel": 1e-2}, "block": {"rel": 1e-2},
            "step": {"rel": 0.1}, "edit": {"rel": 0.1}, "vision": {"rel": 4e-2}, "lora": {"rel": 2e-4}}[case["kind"]]


# ------------------------------------------------------------------ the same in 64 bits
def _mrope(pos):
    """cos, sin [S, 64]: frequency kk takes its position from axis kk % 3 while kk < 60, from axis 0 beyond."""
    kk = torch.arange(64, device="cuda")
    axis = torch.where(kk < 60, kk % 3, torch.zeros_like(kk))
    ang = pos.double().cuda()[axis].t() * torch.exp(-math.log(5e6) * 2.0 * kk.double() / 128.0)
    return torch.cos(ang), torch.sin(ang)


def _rms(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w.double()


def _rot(x, cos, sin):
    a, b = x[..., :64], x[..., 64:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(q, k, v, ar, scale):
    """q [H, S, d], k / v [Hk, S, d]: rows below ar see the keys up to themselves, the others every key."""
    out, s = torch.empty_like(q), q.shape[1]
    for h in range(q.shape[0]):
        kh = h // (q.shape[0] // k.shape[0])
        for r0 in range(0, s, 4096):
            sc = q[h, r0:r0 + 4096] @ k[kh].t() * scale
            if r0 < ar:
                rows = torch.arange(r0, r0 + sc.shape[0], device="cuda")[:, None]
                sc.masked_fill_((rows < ar) & (torch.arange(s, device="cuda")[None] > rows), -math.inf)
            out[h, r0:r0 + 4096] = torch.softmax(sc, -1) @ v[kh]
    return out


def _block(x, w, layer, cos, sin, ar):
    t = lambda name: w.tensor(layer, name).double()  # noqa: E731
    heads = lambda y, n: y.view(y.shape[0], n, D).transpose(0, 1)  # noqa: E731
    a = _rms(x, t("input_ln"))
    q = _rot(_rms(heads(a @ t("q_proj").t(), HEADS), t("q_norm")), cos, sin)
    k = _rot(_rms(heads(a @ t("k_proj").t(), KV_HEADS), t("k_norm")), cos, sin)
    v = heads(a @ t("v_proj").t(), KV_HEADS)
    x = x + _attend(q, k, v, ar, D ** -0.5).transpose(0, 1).reshape(x.shape[0], -1) @ t("o_proj").t()
    a = _rms(x, t("post_ln"))
    return x + (torch.nn.functional.silu(a @ t("gate_proj").t()) * (a @ t("up_proj").t())) @ t("down_proj").t()


def _forward(w, ids, pos, ar, vin, t, visual=None):
    g = lambda name: w.tensor(-1, name).double()  # noqa: E731
    half = torch.arange(128, dtype=torch.float64, device="cuda")
    arg = t * 1000.0 * torch.exp(-math.log(1e4) * half / 128.0)
    e = torch.cat([torch.cos(arg), torch.sin(arg)])
    e = torch.nn.functional.silu(g("te0_w") @ e + g("te0_b"))
    e = g("te2_w") @ e + g("te2_b")
    n = ids.numel() if visual is None else ids.numel() - vin.shape[0]
    x = w.tensor(-1, "embed_tokens")[ids[:n].clamp(max=VOCAB - 1)].double()
    if visual is not None:
        rows = visual[0].bool().nonzero().flatten()
        x[rows] = visual[1].double()
    x[ids[:n] == TMS_ID] = e
    x = torch.cat([x, vin.double() @ g("xe1_w").t() @ g("xe2_w").t() + g("xe2_b")])
    cos, sin = _mrope(pos)
    for i in range(LAYERS):
        x = _block(x, w, i, cos, sin, ar)
        if visual is not None and i < 3:
            x[rows] += visual[2][i].double()
    return _rms(x, g("fnorm_w")) @ g("fl_w").t() + g("fl_b")


def _gelu(x, tanh):
    return torch.nn.functional.gelu(x, approximate="tanh" if tanh else "none")


def _layernorm(x, w, b):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], w, b, 1e-6)


def _vision(case, tensors, px):
    t = iter([x.double() for x in tensors])
    gh, gw = case["gh"], case["gw"]
    n = gh * gw
    # patches come in 2 x 2 blocks; each takes the bilinear mix of a learned 48 x 48 grid of positions
    r = torch.arange(n, device="cuda")
    h, w = (r // 4) // (gw // 2) * 2 + (r % 4) // 2, (r // 4) % (gw // 2) * 2 + r % 2
    x = px.double() @ next(t).t() + next(t)
    pe = next(t)
    hf, wf = h.double() * 47 / (gh - 1), w.double() * 47 / (gw - 1)
    h0, w0 = hf.long().clamp(max=47), wf.long().clamp(max=47)
    h1, w1 = (h0 + 1).clamp(max=47), (w0 + 1).clamp(max=47)
    dh, dw = (hf - h0)[:, None], (wf - w0)[:, None]
    x = x + (1 - dh) * (1 - dw) * pe[h0 * 48 + w0] + (1 - dh) * dw * pe[h0 * 48 + w1] + dh * (1 - dw) * pe[h1 * 48 + w0] + dh * dw * pe[h1 * 48 + w1]
    inv = 1.0 / 10000.0 ** (torch.arange(18, dtype=torch.float64, device="cuda") / 18.0)
    # the angles themselves are defined as bf16 numbers
    ang = torch.cat([h[:, None] * inv.float(), w[:, None] * inv.float()], -1).bfloat16().double()
    cos, sin = torch.cos(ang), torch.sin(ang)

    def rot(y):
        a, b = y[..., :36], y[..., 36:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    ds_in = []
    for i in range(VDEPTH):
        n1w, n1b, n2w, n2b, qw, qb, pw, pb, f1w, f1b, f2w, f2b = [next(t) for _ in range(12)]
        q, k, v = (_layernorm(x, n1w, n1b) @ qw.t() + qb).view(n, 3, VHEADS, VD).permute(1, 2, 0, 3)
        a = _attend(rot(q), rot(k), v.contiguous(), 0, VD ** -0.5).transpose(0, 1).reshape(n, VH)
        x = x + a @ pw.t() + pb
        x = x + _gelu(_layernorm(x, n2w, n2b) @ f1w.t() + f1b, True) @ f2w.t() + f2b
        if i in (8, 16, 24):
            ds_in.append(x)
    outs = []
    for j, y in enumerate([x] + ds_in):
        nw, nb, f1w, f1b, f2w, f2b = [next(t) for _ in range(6)]
        y = _layernorm(y, nw, nb).view(-1, VM) if j == 0 else _layernorm(y.view(-1, VM), nw, nb)
        outs.append(_gelu(y @ f1w.t() + f1b, False) @ f2w.t() + f2b)
    return {"image_embeds": outs[0], "deepstack": torch.stack(outs[1:])}


def exact(case, seed):
    s = prepare(case, seed)
    kind = case["kind"]
    if kind == "linear":
        return s["x"].double() @ s["w"].double().t() + s["b"].double()
    if kind == "sched":
        z, xc, xu = s["z"].double(), s["xc"].double(), s["xu"].double()
        return _euler(z, xc, xu)
    if kind == "sdpa":
        return _attend(s["q"].double(), s["k"].double(), s["v"].double(), case["ar"], D ** -0.5)
    if kind == "block":
        return _block(s["x"].double(), s["weights"], 0, *_mrope(s["pos"]), s["ar"])
    if kind == "step":
        xs = [_forward(s["weights"], ids, pos, ar, s["z"], 1.0 - SIGMA) for ids, pos, ar in (s["cond"], s["uncond"])]
        img = s["z"].shape[0]
        return {"z_next": _euler(s["z"].double(), xs[0][-img:], xs[1][-img:]), "x_pred": torch.cat(xs)}
    if kind == "edit":
        return _forward(s["weights"], s["ids"], s["pos"], s["ar"], s["vin"], EDIT_T, s["visual"])
    if kind == "vision":
        return _vision(case, s["tensors"], s["px"])
    return [w.double() + (e.multiplier * e.alpha / e.rank) * (u.double() @ d.double()) for w, u, d, e in zip(s["w"], s["up"], s["down"], s["entries"])]


def _euler(z, xc, xu):
    vc, vu = (xc - z) / SIGMA, (xu - z) / SIGMA
    return z + (SIGMA_NEXT - SIGMA) * -(vu + GUIDANCE * (vc - vu))
