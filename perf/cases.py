"""The work that the performance of this repository is measured on: operators called through the C ABI with tensors that are already on the
GPU, and decode calls of whole models.

`listed()` names the cases, `draw()` gives further ones of the same ranges, `prepare()` makes what a program holds before the call (weights on the
device, inputs, a context), `run()` is one pass, `work()` the bytes and operations it cannot do without, `exact()` the same result in 64-bit
arithmetic by plain torch.  The library runs with its default numerics (fast).

Models have the layer shapes of the benchmark's configurations with fewer layers, and a vocabulary that keeps the output head's share of a step
about what it is in the full model.  Weights are synthetic."""
import ctypes
import importlib
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GROUP = {"Q4_K": 144, "Q6_K": 210, "Q8_0": 272, "Q4_0": 144, "MXFP4": 136}   # bytes per 256 weights
VOCAB = 32000


def _library(module=None):
    """the package (its folder's name has a dot, so it is loaded by path), or one of its modules"""
    if "llama_rust_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("llama_rust_b200", os.path.join(ROOT, "llama.rust_b200", "__init__.py"))
        mod = importlib.util.module_from_spec(spec)
        sys.modules["llama_rust_b200"] = mod
        spec.loader.exec_module(mod)
    return importlib.import_module("llama_rust_b200." + module) if module else sys.modules["llama_rust_b200"]


def listed():
    return [
        # one token against one projection of a 4096-wide model: the smallest call there is, all latency
        {"name": "mul_mat_row_q4_k", "op": "mul_mat", "type": "Q4_K", "n": 4096, "k": 4096, "m": 1},
        # a prompt batch against an FFN matrix of a Q8_0 model
        {"name": "mul_mat_prompt_q8_0", "op": "mul_mat", "type": "Q8_0", "n": 14336, "k": 4096, "m": 512},
        # the expert projection of a mixture-of-experts layer for a prompt batch (128 experts, 8 per token, MXFP4)
        {"name": "experts_mxfp4", "op": "experts", "type": "MXFP4", "n": 768, "k": 2048, "experts": 128, "top": 8, "tokens": 512},
        # one new token over a long F16 cache, grouped-query heads
        {"name": "attention_row_32768", "op": "attention", "heads": 32, "kv_heads": 8, "dim": 128, "rows": 1, "n_kv": 32768},
        # the last 512 tokens of a 4096-token prompt
        {"name": "attention_prompt_4096", "op": "attention", "heads": 32, "kv_heads": 8, "dim": 128, "rows": 512, "n_kv": 4096},
        # a Q4_K_M model of the 8B layer shape: reading a prompt, up to the first token's logits
        {"name": "llama_prompt_512", "op": "llama", "width": 4096, "ff": 14336, "kv_heads": 8, "layers": 8, "seqs": 1, "prompt": 512, "steps": 0},
        # the same model answering: a short prompt, then single tokens (the case decode speed is quoted on)
        {"name": "llama_steps", "op": "llama", "width": 4096, "ff": 14336, "kv_heads": 8, "layers": 8, "seqs": 1, "prompt": 64, "steps": 32},
        # the same model serving 16 conversations at once
        {"name": "llama_16_sequences", "op": "llama", "width": 4096, "ff": 14336, "kv_heads": 8, "layers": 8, "seqs": 16, "prompt": 32, "steps": 16},
        # a Rukusun model (gated linear attention, every fourth layer latent attention) reading a prompt
        {"name": "rukusun_prompt_2048", "op": "rukusun", "width": 2048, "layers": 8, "dtype": "bfloat16", "prompt": 2048, "steps": 0},
        # the widest Rukusun layers the benchmark has, answering
        {"name": "rukusun_steps", "op": "rukusun", "width": 4096, "layers": 4, "dtype": "bfloat16", "prompt": 65, "steps": 32},
        # a Lenolix model (grouped-query attention, window and kept first tokens) of the widest layers, reading a prompt
        {"name": "lenolix_prompt_2048", "op": "lenolix", "width": 4096, "layers": 4, "dtype": "bfloat16", "prompt": 2048, "steps": 0},
        # a small Lenolix model answering: launches and latency count most
        {"name": "lenolix_steps", "op": "lenolix", "width": 1024, "layers": 8, "dtype": "bfloat16", "prompt": 65, "steps": 32},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["mul_mat", "mul_mat", "experts", "attention", "attention", "llama", "llama", "rukusun", "lenolix"])
    if op == "mul_mat":
        c = {"op": op, "type": rng.choice(sorted(GROUP)), "n": log(250, 14336), "k": 256 * log(1, 56), "m": log(1, 2048)}
        while c["n"] * c["k"] * c["m"] > 14336 * 4096 * 512:
            c["m"] = max(1, c["m"] // 2 - rng.randrange(2))
        whole = 32 if rng.random() < 0.6 else 8 if c["type"] in ("Q4_0", "MXFP4") else 1   # most matrices have whole row tiles, as heads and FFNs do
        c["n"] = (c["n"] + whole - 1) // whole * whole
        return c
    if op == "experts":
        return {"op": op, "type": rng.choice(["MXFP4", "MXFP4", "Q4_0", "Q4_K"]), "n": 64 * rng.randint(4, 12), "k": 256 * rng.randint(2, 8), "experts": rng.choice([8, 32, 60, 128]),
                "top": rng.choice([2, 4, 8]), "tokens": log(1, 512)}
    if op == "attention":
        kv = rng.choice([4, 8])
        return {"op": op, "heads": kv * rng.choice([1, 2, 4]), "kv_heads": kv, "dim": rng.choice([64, 128, 128]), "rows": rng.choice([1, 1, log(2, 63), log(64, 512)]), "n_kv": log(512, 4096) if rng.random() < 0.5 else log(512, 32768)}
    seqs = rng.choice([1, 1, 4, 16])
    steps = rng.choice([0, rng.randint(4, 16)])
    if op == "llama":
        width = rng.choice([1024, 2048, 4096])
        return {"op": op, "width": width, "ff": 256 * rng.randint(width // 128, width * 7 // 512), "kv_heads": 8, "layers": rng.randint(2, 4), "seqs": seqs,
                "prompt": log(8, 512 // seqs), "steps": steps}
    small = rng.random() < 0.25
    return {"op": op, "width": 1024 if small else rng.choice([1024, 2048]), "layers": 4, "dtype": "float32" if small else "bfloat16", "prompt": log(16, 512 if small else 2048), "steps": steps}


# ---- configurations of the models ---------------------------------------------------------------------------------------------------

def _rukusun(width, layers):
    gla = {"type": "gla", "mixer": {"heads": width // 256, "dim": 128, "vdim": 256, "tau": 16.0}, "mlp": {"kind": "dense", "ff": 4 * width}}
    lat = {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 4 * width},
           "mixer": {"heads": width // 128, "dim": 128, "rot_dim": 64, "kv_rank": 512, "vdim": 128, "mask": {"size": 1024}, "scale": 192 ** -0.5, "rot": {"base": 10000.0, "dims": 64}}}
    return {"architecture": "Rukusun", "embedding": {"scale": float(width) ** 0.5}, "layers": [lat if i % 4 == 3 else gla for i in range(layers)], "norm": {"eps": 1e-5},
            "vocab": VOCAB, "width": width}


def _lenolix(width, layers):
    heads, groups = width // 128, max(1, width // 512)
    ff = round((12 * width - (2 * heads + 2 * groups) * 128) / 3 / 128) * 128
    lay = {"type": "attention", "mlp": {"kind": "dense", "ff": ff, "limit": 7.0},
           "mixer": {"heads": heads, "kv_heads": groups, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024, "keep_first": 64},
                     "rot": {"base": 500000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}}
    return {"architecture": "Lenolix", "embedding": {"scale": float(width) ** 0.5, "bigram": {"buckets": 4093, "mul_prev": 31, "mul_cur": 17}}, "layers": [lay] * layers, "loop": None,
            "norm": {"eps": 1e-5}, "vocab": VOCAB, "width": width}


def _model_tensors(case, gen):
    """(name, tensor on the GPU, values that are BF16 numbers) of a Rukusun or Lenolix model"""
    cfg = (_rukusun if case["op"] == "rukusun" else _lenolix)(case["width"], case["layers"])
    E, V = cfg["width"], cfg["vocab"]

    def rnd(*shape, mean=0.0, dev=1.0):
        return torch.randn(shape, device="cuda", generator=gen, dtype=torch.float32).mul_(dev).add_(mean).bfloat16()

    def mat(n, k):
        return rnd(n, k, dev=k ** -0.5)

    yield "embed", mat(V, E)
    if case["op"] == "rukusun":
        yield "head", mat(V, E)
        yield "final.norm", rnd(E, dev=0.1)
        for i, lay in enumerate(cfg["layers"]):
            p, m = "l%d." % i, lay["mixer"]
            H, d, e = m["heads"], m["dim"], m["vdim"]
            yield p + "norm1", rnd(E, dev=0.1)
            yield p + "norm2", rnd(E, dev=0.1)
            yield p + "mlp.up", mat(lay["mlp"]["ff"], E)
            yield p + "mlp.down", mat(E, lay["mlp"]["ff"])
            yield p + "mix.o", mat(E, H * e)
            if lay["type"] == "gla":
                yield p + "mix.a1", mat(16, E)
                yield p + "mix.a2", mat(H * d, 16)
                yield p + "mix.a2.b", rnd(H * d, mean=2.0)
                yield p + "mix.norm", rnd(e, mean=1.0, dev=0.1)
                for n, rows in (("q", H * d), ("k", H * d), ("v", H * e), ("g", H * e)):
                    yield p + "mix." + n, mat(rows, E)
            else:
                R, rot = m["kv_rank"], m["rot_dim"]
                yield p + "mix.q", mat(H * (d + rot), E)
                yield p + "mix.dkv", mat(R + rot, E)
                yield p + "mix.dkv.norm", rnd(R, mean=1.0, dev=0.1)
                yield p + "mix.uk", mat(H * d, R)
                yield p + "mix.uv", mat(H * e, R)
                yield p + "mix.sink", rnd(H)
                yield p + "mix.g", mat(H, E)
        return
    yield "bigram", mat(cfg["embedding"]["bigram"]["buckets"] + 1, E)
    for i, lay in enumerate(cfg["layers"]):
        p, m, ff = "l%d." % i, lay["mixer"], lay["mlp"]["ff"]
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            yield p + n, rnd(E, mean=1.0, dev=0.1)
            yield p + n + ".b", rnd(E, dev=0.1)
        for n in ("ls1", "ls2"):
            yield p + n, rnd(E, mean=0.5, dev=0.1)
        for n, rows in (("q", m["heads"] * m["dim"]), ("k", m["kv_heads"] * m["dim"]), ("v", m["kv_heads"] * m["vdim"])):
            yield p + "mix." + n, mat(rows, E)
        yield p + "mix.sink", rnd(m["heads"])
        yield p + "mix.o", mat(E, m["heads"] * m["vdim"])
        yield p + "mlp.gate", mat(ff, E)
        yield p + "mlp.up", mat(ff, E)
        yield p + "mlp.down", mat(E, ff)
    yield "final.norm", rnd(E, mean=1.0, dev=0.1)
    yield "final.norm.b", rnd(E, dev=0.1)


def _llama_hparams(case):
    return dict(n_vocab=VOCAB, n_embd=case["width"], n_head=case["width"] // 128, n_head_kv=case["kv_heads"], n_embd_head=128, n_ff=case["ff"], n_layer=case["layers"], n_ctx_train=8192,
                rope_mode=0, norm_rms_eps=1e-5, rope_freq_base=500000.0, rope_freq_scale=1.0)


def _blocks(ty, rows, k, gen, times=1.0):
    """random ggml blocks on the GPU, uint8 [rows, row bytes], whose weights have mean 0 and a spread of about 0.02 x times"""
    per = {"Q4_K": 144, "Q6_K": 210, "Q8_0": 34, "Q4_0": 18, "MXFP4": 17}[ty]
    n = rows * (k // 256) * (GROUP[ty] // per)

    def scale(mean):
        return times * mean * (torch.rand(n, device="cuda", generator=gen) + 0.5)

    def f16(x):
        return x.half().view(torch.uint8).reshape(n, 2)

    b = torch.randint(0, 256, (n, per), device="cuda", generator=gen, dtype=torch.uint8)
    if ty == "Q4_K":
        d = scale(1.2e-4)   # every 32 weights' minimum is 7.5 steps of theirs below zero: the middle of the 16 values is zero
        b[:, 0:2], b[:, 2:4], b[:, 8:12], b[:, 12:16] = f16(d), f16(7.5 * d), b[:, 4:8], (b[:, 12:16] & 15) * 17
    elif ty == "Q6_K":
        b[:, 192:208] = torch.randint(-32, 33, (n, 16), device="cuda", generator=gen, dtype=torch.int8).view(torch.uint8)
        b[:, 208:210] = f16(scale(5.8e-5))
    elif ty == "Q8_0":
        b[:, 0:2] = f16(scale(2.7e-4))
    elif ty == "Q4_0":
        b[:, 0:2] = f16(scale(4.3e-3))
    else:
        b[:, 0] = torch.randint(119, 122, (n,), device="cuda", generator=gen, dtype=torch.uint8)
    return b.reshape(rows, -1)


def _llama_tensors(case, gen):
    """(name, type, tensor on the GPU, ne0, ne1) of a Q4_K_M model: matrices of spread 0.02, less for those whose result joins the residual stream
    (1 / sqrt(2 layers), as such models are initialised), embeddings of spread 4: the stream is larger than what one layer adds to it"""
    shapes = _library("shapes")
    for name, (ne0, ne1) in shapes.tensor_shapes(_llama_hparams(case)).items():
        ty = {shapes.F32: "F32", shapes.Q4_K: "Q4_K", shapes.Q6_K: "Q6_K"}[shapes.q4_k_m_type(name, case["layers"])]
        if ty == "F32":
            yield name, ty, 1.0 + 0.1 * torch.randn(ne0, device="cuda", generator=gen), ne0, ne1
        else:
            times = 200.0 if name == "token_embd.weight" else (2 * case["layers"]) ** -0.5 if "attn_output" in name or "ffn_down" in name else 1.0
            yield name, ty, _blocks(ty, ne1, ne0, gen, times), ne0, ne1


# ---- what a program has in hand --------------------------------------------------------------------------------------------------------

def _generators(seed):
    """for the weights and for the other inputs"""
    return torch.Generator("cuda").manual_seed(2 * seed + 1), torch.Generator("cuda").manual_seed(2 * seed + 2)


def _tokens(case, seed):
    """int32 [seqs, prompt + steps]"""
    return np.random.default_rng(seed + 7).integers(0, VOCAB, (case.get("seqs", 1), case["prompt"] + case["steps"])).astype(np.int32)


def _op_inputs(case, seed):
    """seeded inputs on the GPU"""
    gw, gx = _generators(seed)

    def normal(*shape):
        return torch.randn(shape, device="cuda", generator=gx)

    if case["op"] == "mul_mat":
        return {"w": _blocks(case["type"], case["n"], case["k"], gw), "x": normal(case["m"], case["k"])}
    if case["op"] == "experts":
        ids = torch.rand((case["tokens"], case["experts"]), device="cuda", generator=gx).argsort(dim=1)[:, :case["top"]]
        return {"w": _blocks(case["type"], case["experts"] * case["n"], case["k"], gw), "x": normal(case["tokens"], case["k"]), "ids": ids.int().contiguous()}
    H, G, d, T, N = case["heads"], case["kv_heads"], case["dim"], case["rows"], case["n_kv"]
    mask = None
    if T > 1:   # causal: the rows are the last T of the N positions
        T0 = N - T if N >= T else 0
        seen = torch.arange(N, device="cuda")[None, :] <= torch.arange(T, device="cuda")[:, None] + T0
        mask = torch.where(seen, 0.0, -math.inf).half().contiguous()
    return {"q": normal(T, H, d), "k": normal(N, G, d).half(), "v": normal(N, G, d).half(), "mask": mask}


def prepare(case, seed):
    lib = _library()
    if case["op"] in ("mul_mat", "experts"):
        x = _op_inputs(case, seed)
        ty = getattr(lib, case["type"])
        blocks = x.pop("w").cpu().numpy()
        if case["op"] == "mul_mat":
            return dict(x, case=case, w=lib.Weight(ty, blocks, case["k"]), out=torch.empty((case["m"], case["n"]), device="cuda"))
        return dict(x, case=case, w=lib.ExpertWeights(ty, blocks, case["n"], case["k"]), out=torch.empty((case["tokens"], case["top"], case["n"]), device="cuda"))
    if case["op"] == "attention":
        x = _op_inputs(case, seed)
        H, G, d, T, N = case["heads"], case["kv_heads"], case["dim"], case["rows"], case["n_kv"]
        out = torch.empty((T, H, d), device="cuda")
        a = lib.FlashAttnArgs()
        a.dk, a.dv, a.n_tok, a.n_head, a.n_head_kv, a.n_kv = d, d, T, H, G, N
        a.q, a.q_nb1, a.q_nb2 = x["q"].data_ptr(), H * d * 4, d * 4
        a.k, a.k_nb1, a.k_nb2 = x["k"].data_ptr(), G * d * 2, d * 2
        a.v, a.v_nb1, a.v_nb2 = x["v"].data_ptr(), G * d * 2, d * 2
        if x["mask"] is not None:
            a.mask, a.mask_nb1 = x["mask"].data_ptr(), N * 2
        a.scale, a.dst = d ** -0.5, out.data_ptr()
        return dict(x, case=case, args=a, out=out)
    llama = _library("llama")
    gw, _ = _generators(seed)
    seqs, length = case.get("seqs", 1), case["prompt"] + case["steps"]
    n_ctx, n_batch = (seqs * length + 255) // 256 * 256, seqs * case["prompt"]
    if case["op"] == "llama":
        ctx = llama.Llama(_llama_hparams(case), n_ctx, n_batch)
        for name, ty, t, ne0, ne1 in _llama_tensors(case, gw):
            ctx.set_tensor(name, getattr(lib, ty), t.cpu().numpy(), ne0, ne1)
    else:
        cfg = (_rukusun if case["op"] == "rukusun" else _lenolix)(case["width"], case["layers"])
        ctx = llama.Model(cfg, n_ctx, n_batch, n_seq=max(1, seqs), dtype=case["dtype"])
        for name, t in _model_tensors(case, gw):
            ctx.set_tensors({name: t.view(torch.int16).cpu().numpy().view(np.uint16)})
    return {"case": case, "ctx": ctx, "tokens": _tokens(case, seed)}


def run(state):
    case, lib = state["case"], _library()
    if case["op"] == "mul_mat":
        lib.mul_mat_device(state["w"], state["x"].data_ptr(), case["m"], state["out"].data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if case["op"] == "experts":
        w = state["w"]
        lib.check(lib.lib.b200_mul_mat_id(w.ty, w.n, w.k, w.n_expert, 1, case["tokens"], case["top"], w.ptr, state["x"].data_ptr(), state["ids"].data_ptr(), state["out"].data_ptr(), 0,
                                          torch.cuda.current_stream().cuda_stream), "mul_mat_id")
        return state["out"]
    if case["op"] == "attention":
        lib.check(lib.lib.b200_flash_attn_ext(ctypes.byref(state["args"]), torch.cuda.current_stream().cuda_stream), "flash_attn_ext")
        return state["out"]
    # a whole request: an empty cache, the prompts in one call, then a token of every sequence per call (given tokens, so that what is
    # computed does not hang on near ties).  Logits of each prompt's last token and of every step, [1 + steps, seqs, vocabulary]
    ctx, toks = state["ctx"], state["tokens"]
    S, P = toks.shape[0], case["prompt"]
    ctx.kv_clear()
    if S == 1:
        out = [ctx.decode(toks[0, :P], np.arange(P))]
        for i in range(P, P + case["steps"]):
            out.append(ctx.decode(toks[0, i:i + 1], [i]))
        return np.stack(out)[:, None, :]
    seq = np.arange(S)
    out = [ctx.decode_seqs(toks[:, :P].reshape(-1), np.tile(np.arange(P), S), np.repeat(seq, P), seq * P + P - 1)[0]]
    for i in range(P, P + case["steps"]):
        out.append(ctx.decode_seqs(toks[:, i], np.full(S, i), seq, seq)[0])
    return np.stack(out)


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------------------

def work(case):
    if case["op"] == "mul_mat":
        n, k, m = case["n"], case["k"], case["m"]
        return {"bytes": n * (k // 256) * GROUP[case["type"]] + 4 * m * k + 4 * m * n, "flops": 2 * n * k * m}
    if case["op"] == "experts":
        n, k, pairs = case["n"], case["k"], case["tokens"] * case["top"]
        touched = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** case["tokens"])   # expected
        return {"bytes": touched * n * (k // 256) * GROUP[case["type"]] + 4 * case["tokens"] * k + 4 * pairs * n + 4 * pairs, "flops": 2 * n * k * pairs}
    if case["op"] == "attention":
        H, G, d, T, N = case["heads"], case["kv_heads"], case["dim"], case["rows"], case["n_kv"]
        seen = N if T == 1 else sum(min(N, t + 1 + max(0, N - T)) for t in range(T)) / T
        return {"bytes": 4 * N * G * d + 8 * T * H * d + (2 * T * N if T > 1 else 0), "flops": 4 * T * seen * H * d}
    S, P, E, calls = case.get("seqs", 1), case["prompt"], case["width"], 1 + case["steps"]
    rows, total = S * calls, S * (P + case["steps"])
    if case["op"] == "llama":
        shapes = _library("shapes")
        body = head = body_bytes = head_bytes = 0
        for name, (ne0, ne1) in shapes.tensor_shapes(_llama_hparams(case)).items():
            ty = shapes.q4_k_m_type(name, case["layers"])
            if ty == shapes.F32 or name == "token_embd.weight":
                continue
            nbytes = ne0 * ne1 * (144 if ty == shapes.Q4_K else 210) // 256
            if name == "output.weight":
                head, head_bytes = ne0 * ne1, nbytes
            else:
                body, body_bytes = body + ne0 * ne1, body_bytes + nbytes
        attn = case["layers"] * 2 * E * sum(2 * (i + 1) for i in range(P + case["steps"])) * S
        cells = case["layers"] * 4 * case["kv_heads"] * 128 * S * sum(P + i for i in range(calls))
        return {"bytes": calls * (body_bytes + head_bytes) + cells + 4 * rows * VOCAB, "flops": 2 * body * total + 2 * head * rows + attn}
    size = 2 if case["dtype"] == "bfloat16" else 4
    cfg = (_rukusun if case["op"] == "rukusun" else _lenolix)(E, case["layers"])
    body, mix, cells = 0, 0.0, 0.0
    for lay in cfg["layers"]:
        m, ff = lay["mixer"], lay["mlp"]["ff"]
        H, d, e = m["heads"], m["dim"], m["vdim"]
        seen = sum(min(i + 1, 1024 + (64 if case["op"] == "lenolix" else 0)) for i in range(P + case["steps"]))
        last = sum(min(P + i, 1024) for i in range(calls))
        if lay["type"] == "gla":
            body += E * (2 * H * d + 3 * H * e + 16) + 16 * H * d + 2 * E * ff
            mix += 5.0 * H * d * e * total          # decay, rank-1 update and product with the state, a token at a time
            cells += 8.0 * H * d * e * calls        # the state, read and written once per call
        elif lay["type"] == "latent_attention":
            body += E * (H * (d + 64) + 512 + 64 + H * e + H) + 512 * H * (d + e) + 2 * E * ff
            mix += 2.0 * H * (d + 64 + e) * seen
            cells += size * (512 + 64) * last
        else:
            body += E * (2 * H * d + 2 * m["kv_heads"] * d) + 3 * E * ff
            mix += 2.0 * H * (d + e) * seen
            cells += size * m["kv_heads"] * (d + e) * last
    return {"bytes": size * calls * (body + VOCAB * E) + cells + 4 * rows * VOCAB, "flops": 2 * body * total + 2 * VOCAB * E * rows + mix}


def tolerance(case):
    """About four times what the default and the bit-exact kernels differ by.  Mat-muls: the activations' quantization is part of the operation, the
    sums are in 32 bits.  Attention: queries and probabilities enter the tensor cores as 16-bit floats.  Models: in a Q4_K_M model a sum's last bit
    can move an activation to the next of its 255 steps, in a BF16 model every row that enters a matrix product is rounded, through all layers."""
    if case["op"] in ("mul_mat", "experts"):
        return {"rel": 2e-6, "max": 4e-5}
    if case["op"] == "attention":
        return {"rel": 1.2e-3, "max": 2e-2}
    if case["op"] == "llama":
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 2e-5, "max": 2e-4} if case["dtype"] == "float32" else {"rel": 0.02, "max": 0.2}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------------------------

F = torch.float64


def _decode_blocks(ty, b, k):
    """ggml blocks uint8 [rows, row bytes] -> float64 [rows, k]"""
    rows = b.shape[0]
    b = b.reshape(-1, {"Q4_K": 144, "Q6_K": 210, "Q8_0": 34, "Q4_0": 18, "MXFP4": 17}[ty])

    def half(lo):
        return b[:, lo:lo + 2].contiguous().view(torch.float16).to(F)

    if ty == "Q4_K":
        s, q = b[:, 4:16].int(), b[:, 16:144].reshape(-1, 4, 1, 32)
        sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | (s[:, 0:4] >> 6 << 4)], 1).to(F)
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | (s[:, 4:8] >> 6 << 4)], 1).to(F)
        w = torch.cat([q & 15, q >> 4], 2).reshape(-1, 8, 32).to(F)
        w = half(0)[:, :, None] * sc[:, :, None] * w - half(2)[:, :, None] * mn[:, :, None]
    elif ty == "Q6_K":
        lo, hi = b[:, 0:128].int().reshape(-1, 2, 2, 32), b[:, 128:192].int().reshape(-1, 2, 1, 32)
        lo = torch.cat([lo & 15, lo >> 4], 2)                      # [.., 2, 4, 32]
        hi = torch.cat([hi >> s & 3 for s in (0, 2, 4, 6)], 2)
        sc = b[:, 192:208].contiguous().view(torch.int8).to(F).reshape(-1, 16, 1)
        w = ((lo | hi << 4) - 32).to(F).reshape(-1, 16, 16) * sc * half(208)[:, :, None]
    elif ty == "Q8_0":
        w = half(0) * b[:, 2:34].contiguous().view(torch.int8).to(F)
    elif ty == "Q4_0":
        w = half(0) * (torch.cat([b[:, 2:18] & 15, b[:, 2:18] >> 4], 1).to(F) - 8.0)
    else:
        values = torch.tensor([0, 1, 2, 3, 4, 6, 8, 12, 0, -1, -2, -3, -4, -6, -8, -12], dtype=F, device=b.device)
        w = values[torch.cat([b[:, 1:17] & 15, b[:, 1:17] >> 4], 1).long()] * torch.exp2(b[:, 0:1].to(F) - 128.0)
    return w.reshape(rows, k)


def _quantized(x, k_quant):
    """the activations as the operation's 8-bit blocks hold them: 256 elements with an F32 scale, or 32 with an F16 one"""
    x = x.float()
    blocks = x.reshape(-1, 256 if k_quant else 32)
    top = blocks.abs().amax(1, keepdim=True)
    steps = torch.full_like(top, 127.0)   # tensors on both sides: torch divides by a number through its reciprocal
    inv = torch.where(top > 0, steps / top, torch.zeros_like(top))
    q = torch.round(blocks * inv).to(F)
    scale = torch.where(top > 0, torch.ones_like(top) / inv, torch.zeros_like(top)).to(F) if k_quant else (top / steps).half().to(F)
    return (q * scale).reshape(x.shape)


def _product(x, ty, blocks, k):
    return _quantized(x, ty in ("Q4_K", "Q6_K")) @ _decode_blocks(ty, blocks, k).T


def _rotate(x, cos, sin, halves):
    """x [T, H, d]; cos, sin [T, dims / 2]: the first dims channels turn in pairs (2i, 2i + 1), or (i, i + dims / 2)"""
    n = cos.shape[1]
    u, v = (x[..., :n], x[..., n:2 * n]) if halves else (x[..., 0:2 * n:2], x[..., 1:2 * n:2])
    c, s = cos[:, None, :], sin[:, None, :]
    a, b = u * c - v * s, u * s + v * c
    turned = torch.cat([a, b], -1) if halves else torch.stack([a, b], -1).flatten(-2)
    return torch.cat([turned, x[..., 2 * n:]], -1)


def _attend(q, k, v, scale, seen, sink=None):
    """q [T, H, d], k [N, G, d], v [N, G, e], seen [T, N] (None: all) -> [T, H, e]; a sink joins the denominator"""
    per = q.shape[1] // k.shape[1]
    out = []
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // per].T * scale
        if seen is not None:
            s = s.masked_fill(~seen, -math.inf)
        top = s.amax(1, keepdim=True) if sink is None else torch.maximum(s.amax(1, keepdim=True), sink[h])
        p = torch.exp(s - top)
        total = p.sum(1, keepdim=True) + (0.0 if sink is None else torch.exp(sink[h] - top))
        out.append(p / total @ v[:, h // per])
    return torch.stack(out, 1)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _exact_llama(case, seed):
    gw, _ = _generators(seed)
    hp, w = _llama_hparams(case), {}
    for name, ty, t, ne0, _ in _llama_tensors(case, gw):
        w[name] = (ty, t, ne0)
    toks = torch.from_numpy(_tokens(case, seed)).cuda().long()
    S, P, L = toks.shape[0], case["prompt"], toks.shape[1]
    pos = torch.arange(L, device="cuda", dtype=F).repeat(S)
    half = torch.arange(64, device="cuda", dtype=F)
    angle = pos[:, None] * hp["rope_freq_base"] ** (-half / 64.0)[None, :]
    cos, sin = torch.cos(angle), torch.sin(angle)
    causal = torch.ones((L, L), dtype=torch.bool, device="cuda").tril()

    def mm(name, x):
        ty, t, k = w[name]
        return _product(x, ty, t, k)

    def norm(name, x):
        return _rms(x, hp["norm_rms_eps"]) * w[name][1].to(F)

    ty, t, k = w["token_embd.weight"]
    x = _decode_blocks(ty, t[toks.reshape(-1)], k)
    H, G = hp["n_head"], hp["n_head_kv"]
    for il in range(hp["n_layer"]):
        p = "blk.%d." % il
        h = norm(p + "attn_norm.weight", x)
        q = _rotate(mm(p + "attn_q.weight", h).reshape(-1, H, 128), cos, sin, False)
        k = _rotate(mm(p + "attn_k.weight", h).reshape(-1, G, 128), cos, sin, False).half().to(F)   # the cache holds 16-bit floats
        v = mm(p + "attn_v.weight", h).reshape(-1, G, 128).half().to(F)
        o = torch.cat([_attend(q[s * L:s * L + L], k[s * L:s * L + L], v[s * L:s * L + L], 128 ** -0.5, causal) for s in range(S)])
        x = x + mm(p + "attn_output.weight", o.reshape(-1, H * 128))
        h = norm(p + "ffn_norm.weight", x)
        gate, up = mm(p + "ffn_gate.weight", h), mm(p + "ffn_up.weight", h)
        x = x + mm(p + "ffn_down.weight", gate * torch.sigmoid(gate) * up)
    x = x.reshape(S, L, -1)[:, P - 1:].transpose(0, 1).reshape(S * (1 + case["steps"]), -1)
    return mm("output.weight", norm("output_norm.weight", x)).reshape(1 + case["steps"], S, VOCAB)


def _exact_rukusun(case, seed):
    gw, _ = _generators(seed)
    w = dict(_model_tensors(case, gw))
    cfg = _rukusun(case["width"], case["layers"])
    toks = torch.from_numpy(_tokens(case, seed)).cuda().long()[0]
    T, eps = toks.numel(), cfg["norm"]["eps"]
    pos = torch.arange(T, device="cuda", dtype=F)
    ago = pos[:, None] - pos[None, :]

    def mm(name, x):
        return x @ w[name].to(F).T

    x = w["embed"][toks].to(F) * cfg["embedding"]["scale"]
    for i, lay in enumerate(cfg["layers"]):
        p, m = "l%d." % i, lay["mixer"]
        H, d, e = m["heads"], m["dim"], m["vdim"]
        h = _rms(x, eps) * (1.0 + w[p + "norm1"].to(F))
        if lay["type"] == "gla":
            q, k, v = mm(p + "mix.q", h).reshape(T, H, d) * d ** -0.5, mm(p + "mix.k", h).reshape(T, H, d), mm(p + "mix.v", h).reshape(T, H, e)
            z = mm(p + "mix.a2", mm(p + "mix.a1", h)) + w[p + "mix.a2.b"].to(F)
            decay = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).reshape(T, H, d)
            S, o = torch.zeros((H, d, e), device="cuda", dtype=F), torch.empty((T, H, e), device="cuda", dtype=F)
            for t in range(T):
                S = decay[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.bmm(q[t][:, None, :], S)[:, 0]
            o = (_rms(o, eps) * w[p + "mix.norm"].to(F)).reshape(T, H * e)
            g = mm(p + "mix.g", h)
            o = o * g * torch.sigmoid(g)
        else:
            R, rot = m["kv_rank"], m["rot_dim"]
            angle = pos[:, None] * m["rot"]["base"] ** (-torch.arange(rot // 2, device="cuda", dtype=F) / (rot // 2))[None, :]
            cos, sin = torch.cos(angle), torch.sin(angle)
            q = mm(p + "mix.q", h).reshape(T, H, d + rot)
            q = torch.cat([q[..., :d], _rotate(q[..., d:], cos, sin, False)], -1)
            both = mm(p + "mix.dkv", h)
            c = _rms(both[:, :R], eps) * w[p + "mix.dkv.norm"].to(F)
            kr = _rotate(both[:, None, R:], cos, sin, False)
            k = torch.cat([mm(p + "mix.uk", c).reshape(T, H, d), kr.expand(T, H, rot)], -1)
            v = mm(p + "mix.uv", c).reshape(T, H, e)
            o = _attend(q, k, v, m["scale"], (ago >= 0) & (ago < m["mask"]["size"]), w[p + "mix.sink"].to(F))
            o = (o * torch.sigmoid(mm(p + "mix.g", h))[:, :, None]).reshape(T, H * e)
        x = x + mm(p + "mix.o", o)
        up = mm(p + "mlp.up", _rms(x, eps) * (1.0 + w[p + "norm2"].to(F)))
        x = x + mm(p + "mlp.down", 0.5 * up * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (up + 0.044715 * up ** 3))))
    x = x[case["prompt"] - 1:]
    return mm("head", _rms(x, eps) * (1.0 + w["final.norm"].to(F)))[:, None, :]


def _exact_lenolix(case, seed):
    gw, _ = _generators(seed)
    w = dict(_model_tensors(case, gw))
    cfg = _lenolix(case["width"], case["layers"])
    toks = torch.from_numpy(_tokens(case, seed)).cuda().long()[0]
    T, eps, pair = toks.numel(), cfg["norm"]["eps"], cfg["embedding"]["bigram"]
    pos = torch.arange(T, device="cuda", dtype=F)
    ago = pos[:, None] - pos[None, :]

    def mm(name, x):
        return x @ w[name].to(F).T

    def norm(name, x):
        dev = x - x.mean(-1, keepdim=True)
        return dev / torch.sqrt((dev * dev).mean(-1, keepdim=True) + eps) * w[name].to(F) + w[name + ".b"].to(F)

    row = torch.cat([toks.new_tensor([pair["buckets"]]), (toks[:-1] * pair["mul_prev"] + toks[1:] * pair["mul_cur"]) % pair["buckets"]])
    x = w["embed"][toks].to(F) * cfg["embedding"]["scale"] + w["bigram"][row].to(F)
    for i, lay in enumerate(cfg["layers"]):
        p, m = "l%d." % i, lay["mixer"]
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        rot, sc = m["rot"], m["rot"]["scaling"]
        f = rot["base"] ** (-2.0 * torch.arange(rot["dims"] // 2, device="cuda", dtype=F) / rot["dims"])
        keep = ((sc["original"] * f / (2.0 * math.pi) - sc["low"]) / (sc["high"] - sc["low"])).clamp(0.0, 1.0)   # long waves are stretched, short ones kept
        angle = pos[:, None] * (keep * f + (1.0 - keep) * f / sc["factor"])[None, :]
        cos, sin = torch.cos(angle), torch.sin(angle)
        h = norm(p + "norm1", x)
        q, k = _rotate(mm(p + "mix.q", h).reshape(T, H, d), cos, sin, True), _rotate(mm(p + "mix.k", h).reshape(T, G, d), cos, sin, True)
        v = mm(p + "mix.v", h).reshape(T, G, d)
        seen = (ago >= 0) & ((ago < m["mask"]["size"]) | (pos[None, :] < m["mask"]["keep_first"]))
        y = mm(p + "mix.o", _attend(q, k, v, m["scale"], seen, w[p + "mix.sink"].to(F)).reshape(T, H * d))
        x = x + norm(p + "norm1b", y) * w[p + "ls1"].to(F)
        h, limit = norm(p + "norm2", x), lay["mlp"]["limit"]
        g, u = mm(p + "mlp.gate", h).clamp(max=limit), mm(p + "mlp.up", h).clamp(-limit, limit)
        y = mm(p + "mlp.down", g * torch.sigmoid(1.702 * g) * (u + 1.0))
        x = x + norm(p + "norm2b", y) * w[p + "ls2"].to(F)
    return mm("embed", norm("final.norm", x[case["prompt"] - 1:]))[:, None, :]


def exact(case, seed):
    if case["op"] == "mul_mat":
        x = _op_inputs(case, seed)
        return _product(x["x"], case["type"], x["w"], case["k"])
    if case["op"] == "experts":
        x = _op_inputs(case, seed)
        q, out = _quantized(x["x"], case["type"] in ("Q4_K", "Q6_K")), torch.empty((case["tokens"], case["top"], case["n"]), device="cuda", dtype=F)
        for e in range(case["experts"]):
            t, s = (x["ids"] == e).nonzero(as_tuple=True)
            out[t, s] = q[t] @ _decode_blocks(case["type"], x["w"][e * case["n"]:(e + 1) * case["n"]], case["k"]).T
        return out
    if case["op"] == "attention":
        x = _op_inputs(case, seed)
        return _attend(x["q"].to(F), x["k"].to(F), x["v"].to(F), case["dim"] ** -0.5, None if x["mask"] is None else x["mask"] == 0)
    return {"llama": _exact_llama, "rukusun": _exact_rukusun, "lenolix": _exact_lenolix}[case["op"]](case, seed).cpu()
