"""Performance cases of the quantized-weight matmul path: what a program that runs a GGUF model over this library asks
of it, from one small matrix to a whole token's pass, decode and prefill, dense and routed, over the block formats.

Kinds of case
  gemv      one matrix times 1..8 activation rows (capi.gemv)
  decode    the matmuls of decoder layers for 1..8 tokens, device pointers: q/k/v in one group, the attention output
            projection, gate/up with the silu fold, the down projection added onto the residual
  backend   the same through the host-facing Backend object: pinned host activations in, results out to pinned host memory
  head      the end of a token: output head, top-k of the logits, embedding row of the picked token
  prefill   one matrix times a prompt's rows (capi.gemm), f16 or f32 activations
  moe       router and routed-expert FFN (capi.moe_ffn_routed), decode batches and prefill

Inputs are synthetic: uniform quants, block scales in the range real files have, activations and router logits ~ N(0, 1).
"""
import ctypes as C
import math

import torch

from kraken_b200 import capi

FORMATS = {"q4_0": capi.Q4_0, "q5_0": capi.Q5_0, "q5_1": capi.Q5_1, "q8_0": capi.Q8_0, "q2_k": capi.Q2_K, "q3_k": capi.Q3_K,
           "q4_k": capi.Q4_K, "q5_k": capi.Q5_K, "q6_k": capi.Q6_K, "iq4_nl": capi.IQ4_NL}
BLOCK = {"q4_0": (32, 18), "q5_0": (32, 22), "q5_1": (32, 24), "q8_0": (32, 34), "iq4_nl": (32, 18), "q2_k": (256, 84),
         "q3_k": (256, 110), "q4_k": (256, 144), "q5_k": (256, 176), "q6_k": (256, 210)}
# f16 fields of a block: (byte offset, lowest, highest value)
SCALES = {"q4_0": [(0, 1e-3, 2e-2)], "q5_0": [(0, 1e-3, 2e-2)], "q5_1": [(0, 1e-3, 2e-2), (2, -0.2, 0.2)], "q8_0": [(0, 1e-3, 2e-2)],
          "iq4_nl": [(0, 1e-4, 2e-3)], "q2_k": [(80, 1e-3, 1e-2), (82, 0.0, 5e-3)], "q3_k": [(108, 1e-3, 1e-2)],
          "q4_k": [(0, 1e-3, 1e-2), (2, 0.0, 5e-3)], "q5_k": [(0, 1e-3, 1e-2), (2, 0.0, 5e-3)], "q6_k": [(208, 1e-4, 2e-3)]}


def listed():
    return [
        # the smallest call: one attention projection of a Q8_0 file, one token
        {"name": "gemv_q8_0", "kind": "gemv", "wt": "q8_0", "n_out": 4096, "n_in": 4096, "rows": 1},
        # one token's matmuls through a Q4_K file of Llama-2-7B shapes: 32 layers, every weight read once
        {"name": "decode_q4_k", "kind": "decode", "wt": "q4_k", "wt_down": "q4_k", "hidden": 4096, "kv": 4096, "ff": 11008, "layers": 32, "rows": 1},
        # four sequences (or four drafted tokens) at once, mixed Q4_K / Q6_K file, host activations in and out
        {"name": "backend_mixed_b4", "kind": "backend", "wt": "q4_k", "wt_down": "q6_k", "hidden": 4096, "kv": 1024, "ff": 11008, "layers": 8, "rows": 4},
        # a small model whose widths are whole 32-value blocks but not whole 256-value super-blocks
        {"name": "decode_q8_0_odd", "kind": "decode", "wt": "q8_0", "wt_down": "q8_0", "hidden": 2080, "kv": 416, "ff": 5600, "layers": 8, "rows": 1},
        # the end of every token: Q6_K head over a 128256-entry vocabulary, top 40, next embedding row
        {"name": "head_q6_k", "kind": "head", "wt": "q6_k", "n_vocab": 128256, "hidden": 4096, "k": 40},
        # prompt of 512 tokens against one FFN matrix, f16 activations
        {"name": "prefill_q4_k_m512", "kind": "prefill", "wt": "q4_k", "n_out": 14336, "n_in": 4096, "rows": 512, "x": "f16"},
        # a long prompt
        {"name": "prefill_q4_k_m2048", "kind": "prefill", "wt": "q4_k", "n_out": 14336, "n_in": 4096, "rows": 2048, "x": "f16"},
        # a short prompt of odd length, f32 activations, down projection
        {"name": "prefill_q6_k_m37", "kind": "prefill", "wt": "q6_k", "n_out": 4096, "n_in": 11008, "rows": 37, "x": "f32"},
        # a middling prompt against a low-bit file
        {"name": "prefill_q3_k_m300", "kind": "prefill", "wt": "q3_k", "n_out": 11008, "n_in": 4096, "rows": 300, "x": "f32"},
        # routed experts (128 experts, top 8, Q4_K gate/up, Q6_K down): one token, a decode batch, a prompt
        {"name": "moe_b1", "kind": "moe", "wt": "q4_k", "wt_down": "q6_k", "experts": 128, "k": 8, "hidden": 4096, "ff": 1536, "rows": 1},
        {"name": "moe_b8", "kind": "moe", "wt": "q4_k", "wt_down": "q6_k", "experts": 128, "k": 8, "hidden": 4096, "ff": 1536, "rows": 8},
        {"name": "moe_prefill_512", "kind": "moe", "wt": "q4_k", "wt_down": "q6_k", "experts": 128, "k": 8, "hidden": 4096, "ff": 1536, "rows": 512},
    ]


def _log(rng, lo, hi, unit=1):
    """A multiple of unit in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))
    return max(lo, min(hi, int(v))) // unit * unit or unit


def draw(rng):
    kind = rng.choices(["gemv", "decode", "backend", "head", "prefill", "moe"], [10, 25, 10, 10, 30, 15])[0]
    wt = rng.choices(["q4_k", "q6_k", "q8_0", "q4_0", "q5_k", "q5_0", "q5_1", "q3_k", "q2_k", "iq4_nl"], [30, 15, 15, 10, 10, 4, 4, 4, 4, 4])[0]
    small = BLOCK[wt][0] == 32 and rng.random() < 0.3   # widths that are whole blocks, not whole super-blocks
    unit = 32 if small else 256
    if kind == "gemv":
        return {"kind": kind, "wt": wt, "n_out": _log(rng, 256, 65536), "n_in": _log(rng, 512, 14336, unit), "rows": rng.randint(1, 8)}
    if kind in ("decode", "backend"):
        hidden = _log(rng, 1024, 4096, unit)
        ff = min(11264, max(1024, int(hidden * rng.uniform(1.5, 4.0)))) // unit * unit
        down = wt if small or rng.random() < 0.5 else "q6_k"
        return {"kind": kind, "wt": wt, "wt_down": down, "hidden": hidden, "kv": hidden // rng.choice([1, 2, 4, 8]), "ff": ff,
                "layers": _log(rng, 2, 12), "rows": rng.choice([1, 1, 1, 1, 2, 3, 4, 6, 8])}
    if kind == "head":
        return {"kind": kind, "wt": rng.choice(["q6_k", "q6_k", "q8_0", "q4_k"]), "n_vocab": _log(rng, 16000, 150000), "hidden": _log(rng, 1024, 4096, 256),
                "k": rng.choice([1, 20, 40, rng.randint(1, 64)])}
    if kind == "prefill":
        n_out, n_in = _log(rng, 512, 14336, rng.choice([1, 32, 256])), _log(rng, 1024, 8192 if small else 11264, unit)
        rows = min(_log(rng, 9, 256 if small else 2048), 2048 * 14336 * 4096 // (n_out * n_in))
        return {"kind": kind, "wt": wt, "n_out": n_out, "n_in": n_in, "rows": rows, "x": "f32" if small or rng.random() < 0.5 else "f16"}
    experts = rng.choice([8, 16, 32, 64, 128])
    return {"kind": kind, "wt": wt, "wt_down": rng.choice([wt, "q6_k"]), "experts": experts, "k": min(experts // 2, rng.randint(2, 8)),
            "hidden": _log(rng, 1024, 4096, 256), "ff": _log(rng, 512, 1536, 256), "rows": _log(rng, 1, 512)}


# ---- inputs ----------------------------------------------------------------------------------------------------

def _bytes(wt, n_out, n_in):
    return n_out * (n_in // BLOCK[wt][0]) * BLOCK[wt][1]


def _weights(wt, n_out, n_in, gen):
    """A matrix of random blocks, [n_out][row bytes] as a GGUF file holds it."""
    n_blk = n_out * (n_in // BLOCK[wt][0])
    bb = BLOCK[wt][1]
    w = torch.randint(0, 256, (n_blk, bb), dtype=torch.uint8, device="cuda", generator=gen)
    for off, lo, hi in SCALES[wt]:
        s = torch.rand(n_blk, device="cuda", generator=gen).mul_(hi - lo).add_(lo).half()
        w[:, off:off + 2] = s.view(torch.uint8).view(n_blk, 2)
    if wt == "q6_k":   # sub-scales in [-64, 63]
        sc = w[:, 192:208]
        sc.copy_((sc & 127) - 64)
    return w.view(-1)


def _normal(gen, *shape, dtype=torch.float32):
    return torch.randn(shape, device="cuda", generator=gen).to(dtype)


def _layers(case, gen):
    hid, kv, ff, wt = case["hidden"], case["kv"], case["ff"], case["wt"]
    return [{"wq": _weights(wt, hid, hid, gen), "wk": _weights(wt, kv, hid, gen), "wv": _weights(wt, kv, hid, gen), "wo": _weights(wt, hid, hid, gen),
             "gate": _weights(wt, ff, hid, gen), "up": _weights(wt, ff, hid, gen), "down": _weights(case["wt_down"], hid, ff, gen)}
            for _ in range(case["layers"])]


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    kind, rows = case["kind"], case.get("rows", 1)
    s = {"case": case, "wt": FORMATS[case["wt"]]}
    if kind in ("gemv", "prefill"):
        s["w"] = _weights(case["wt"], case["n_out"], case["n_in"], gen)
        s["x"] = _normal(gen, rows, case["n_in"], dtype=torch.float16 if case.get("x") == "f16" else torch.float32)
        s["y"] = torch.empty((rows, case["n_out"]), device="cuda")
        if kind == "prefill":
            need = capi.gemm_workspace_bytes(capi.X_F16 if case["x"] == "f16" else capi.X_F32, case["n_out"], case["n_in"], rows)
            s["ws"] = torch.empty(max(need, 256), dtype=torch.uint8, device="cuda")
    elif kind in ("decode", "backend"):
        hid, kv, ff, n = case["hidden"], case["kv"], case["ff"], case["layers"]
        s["layers"] = _layers(case, gen)
        s["wt_down"] = FORMATS[case["wt_down"]]
        # per layer: the normed input of attention, its output, the normed input of the FFN (what the parts of a model
        # between the matmuls hand over)
        s["xa"], s["ao"], s["xf"] = (_normal(gen, n, rows, hid) for _ in range(3))
        s["q"] = torch.empty((n, rows, hid), device="cuda")
        s["k"], s["v"] = (torch.empty((n, rows, kv), device="cuda") for _ in range(2))
        s["r"] = torch.empty((n, rows, hid), device="cuda")
        s["g"], s["u"] = (torch.empty((rows, ff), device="cuda") for _ in range(2))
        if kind == "decode":
            one = lambda t: [x.view(-1) if rows == 1 else x for x in t]  # noqa: E731
            s["steps"] = [{"x": xa, "ao": ao, "xf": xf, "q": q, "k": k, "v": v, "r": r, **lay} for xa, ao, xf, q, k, v, r, lay in
                          zip(one(s["xa"]), one(s["ao"]), one(s["xf"]), one(s["q"]), one(s["k"]), one(s["v"]), one(s["r"]), s["layers"])]
            s["g1"], s["u1"] = one([s["g"], s["u"]])
        else:
            s["be"] = capi.Backend(torch.cuda.current_device())
            s["x_host"] = s["xa"].cpu().pin_memory()
            s["out_host"] = [torch.empty(s[name].shape).pin_memory() for name in "qkvr"]
            s["ptrs"] = [{name: t.data_ptr() for name, t in lay.items()} for lay in s["layers"]]
    elif kind == "head":
        s["w"] = _weights(case["wt"], case["n_vocab"], case["hidden"], gen)
        s["table"] = _weights(case["wt"], case["n_vocab"], case["hidden"], gen)
        s["x"] = _normal(gen, 1, case["hidden"])
        s["logits"] = torch.empty((1, case["n_vocab"]), device="cuda")
        s["emb"] = torch.empty((1, case["hidden"]), device="cuda")
        need = capi.lib.krk_cuda_logits_topk_workspace_bytes(case["n_vocab"], case["k"])
        s["ws"] = torch.empty(need, dtype=torch.uint8, device="cuda")
    else:
        e, hid, ff = case["experts"], case["hidden"], case["ff"]
        s["bank"] = capi.make_bank(_weights(case["wt"], e * ff, hid, gen), _weights(case["wt"], e * ff, hid, gen),
                                   _weights(case["wt_down"], e * hid, ff, gen), s["wt"], FORMATS[case["wt_down"]], e, 0, hid, ff)
        s["x"] = _normal(gen, rows, hid)
        s["logits"] = _normal(gen, rows, e)
        s["y"] = torch.empty((rows, hid), device="cuda")
        need = capi.lib.krk_cuda_moe_workspace_bytes(C.byref(s["bank"]), case["k"], rows)
        s["ws"] = torch.empty(need, dtype=torch.uint8, device="cuda")
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------

def _run_decode(s):
    case, wt = s["case"], s["wt"]
    hid, kv, ff, rows = case["hidden"], case["kv"], case["ff"], case["rows"]
    g, u = s["g1"], s["u1"]
    for t in s["steps"]:
        if rows == 1:
            capi.gemv_group([t["x"]] * 3, [t["wq"], t["wk"], t["wv"]], [wt] * 3, [hid, kv, kv], hid,
                            outs=[t["q"], t["k"], t["v"]])
        else:
            capi.gemv(t["x"], t["wq"], wt, hid, hid, out=t["q"])
            capi.gemv(t["x"], t["wk"], wt, kv, hid, out=t["k"])
            capi.gemv(t["x"], t["wv"], wt, kv, hid, out=t["v"])
        capi.gemv(t["ao"], t["wo"], wt, hid, hid, out=t["r"])
        if rows == 1:
            capi.gemv_group([t["xf"]] * 2, [t["gate"], t["up"]], [wt] * 2, [ff, ff], hid, outs=[g, u], fuse_silu_pair=True)
        else:
            capi.gemv(t["xf"], t["gate"], wt, ff, hid, out=g)
            capi.gemv(t["xf"], t["up"], wt, ff, hid, out=u)
            capi.silu_mul(g, u, out=g)
        capi.gemv(g, t["down"], s["wt_down"], hid, ff, out=t["r"], accumulate=True)
    return s["q"], s["k"], s["v"], s["r"]


def _run_backend(s):
    case, be, wt = s["case"], s["be"], s["wt"]
    hid, kv, ff, rows = case["hidden"], case["kv"], case["ff"], case["rows"]
    be.upload(s["xa"].data_ptr(), s["x_host"].data_ptr(), s["x_host"].nbytes)
    xa, ao, xf, q, k, v, r = (s[n].data_ptr() for n in ("xa", "ao", "xf", "q", "k", "v", "r"))
    g, u = s["g"].data_ptr(), s["u"].data_ptr()
    at, at_kv = 0, 0
    for p in s["ptrs"]:
        be.gemm_group([q + at, k + at_kv, v + at_kv], xa + at, [p["wq"], p["wk"], p["wv"]], wt, [hid, kv, kv], hid, rows)
        be.gemm(r + at, ao + at, p["wo"], wt, hid, hid, rows)
        _, fused = be.gemm_group([g, u], xf + at, [p["gate"], p["up"]], wt, [ff, ff], hid, rows, silu=True)
        if not fused:
            capi.lib.krk_cuda_backend_silu_mul(be.h, g, g, u, rows * ff, ff, None)
        be.gemm_accumulate(r + at, g, p["down"], s["wt_down"], hid, ff, rows)
        at += 4 * rows * hid
        at_kv += 4 * rows * kv
    for t, name in zip(s["out_host"], "qkvr"):
        be.download(t.data_ptr(), s[name].data_ptr(), t.nbytes)
    return s["out_host"]


def run(state):
    s, case = state, state["case"]
    kind = case["kind"]
    if kind == "gemv":
        return capi.gemv(s["x"], s["w"], s["wt"], case["n_out"], case["n_in"], out=s["y"])
    if kind == "prefill":
        return capi.gemm(s["x"], s["w"], s["wt"], case["n_out"], case["n_in"], out=s["y"], workspace=s["ws"])
    if kind == "decode":
        return _run_decode(s)
    if kind == "backend":
        return _run_backend(s)
    if kind == "head":
        logits = capi.gemv(s["x"], s["w"], s["wt"], case["n_vocab"], case["hidden"], out=s["logits"])
        ids, vals, mass = capi.logits_topk(logits, case["k"], temp=0.8, workspace=s["ws"])
        emb = capi.embed(s["table"], s["wt"], case["n_vocab"], case["hidden"], ids[:1], out=s["emb"])
        return logits, ids, vals, mass, emb
    return capi.moe_ffn_routed(s["x"], s["logits"], case["k"], s["bank"], out=s["y"], workspace=s["ws"])


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _matmul(wt, n_out, n_in, rows, x_size=4):
    return _bytes(wt, n_out, n_in) + rows * (n_in * x_size + 4 * n_out), 2 * rows * n_out * n_in


def work(case):
    kind, rows = case["kind"], case.get("rows", 1)
    if kind in ("gemv", "prefill"):
        b, f = _matmul(case["wt"], case["n_out"], case["n_in"], rows, 2 if case.get("x") == "f16" else 4)
    elif kind in ("decode", "backend"):
        hid, kv, ff, n = case["hidden"], case["kv"], case["ff"], case["layers"]
        b = n * (_bytes(case["wt"], 2 * hid + 2 * kv + 2 * ff, hid) + _bytes(case["wt_down"], hid, ff) + 4 * rows * (5 * hid + 2 * kv))
        f = n * 2 * rows * (hid * (2 * hid + 2 * kv + 2 * ff) + hid * ff)
    elif kind == "head":
        b, f = _matmul(case["wt"], case["n_vocab"], case["hidden"], 1)
        b += _bytes(case["wt"], 1, case["hidden"]) + 4 * case["hidden"] + 8 * case["k"]
    else:
        e, k, hid, ff = case["experts"], case["k"], case["hidden"], case["ff"]
        met = e * (1.0 - (1.0 - k / e) ** rows)   # experts that at least one token picks
        b = met * (_bytes(case["wt"], 2 * ff, hid) + _bytes(case["wt_down"], hid, ff)) + 4 * rows * (2 * hid + e + 2 * k)
        f = 2 * rows * k * 3 * hid * ff
    return {"bytes": b, "flops": f}


def tolerance(case):
    kind = case["kind"]
    if kind == "prefill":
        # f16 operands: weights and activations are each rounded to 11 bits (K not whole super-blocks: f32 throughout)
        return {"rel": 1e-3} if case["n_in"] % 256 == 0 else {"rel": 2e-5}
    if kind == "moe":
        # prefill of an expert's rows runs on f16 operands, twice in a row
        return {"rel": 2e-3} if case["rows"] > 8 else {"rel": 2e-5}
    return {"rel": 2e-5}   # f32 sums; router picks and top-k ids are whole values and stay the same
