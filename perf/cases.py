"""The calls whose speed this framework is kept by, with their inputs, their results in 64 bits and their floors.

Three kinds.  "decoder": one micro-batch or decode step of a stage that holds a contiguous range of the layers of a
Q4_K_M decoder, through Stage.forward, as a serving stage runs it: hidden rows (or token ids) in, hidden rows (or logits
and the greedy token) out, at layer widths and context lengths of the benchmark configurations.  "matmul": one quantised
matrix product through ops.mul_mat, for callers that bind single ops.  "layers": a stage whose layers are described one by
one (gated linear recurrence and windowed latent attention, bf16 weights): a whole prompt, or a prompt replayed token by
token.  A stage of a few layers stands for its model: every layer of a model costs the same.

listed() names twelve such calls; draw() takes more from the same ranges.
"""
import math
import zlib

import numpy as np
import torch

F64 = torch.float64
Q4_K, Q6_K, BF16, F32 = 12, 14, 30, 0
BLOCK_BYTES = {Q4_K: 144, Q6_K: 210}
KV_F16, KV_Q4_0, KV_Q8_0 = 1, 2, 8

# layer widths of the benchmark configurations (bench.py names the models they come from)
SHAPES = {
    "3b": dict(n_layer=36, n_embd=2048, n_head=16, n_head_kv=2, n_ff=11008, n_vocab=151936, qkv_bias=1, rope_neox=1, rope_theta=1e6, rms_eps=1e-6),
    "32b": dict(n_layer=64, n_embd=5120, n_head=40, n_head_kv=8, n_ff=27648, n_vocab=152064, qkv_bias=1, rope_neox=1, rope_theta=1e6, rms_eps=1e-6),
    "70b": dict(n_layer=80, n_embd=8192, n_head=64, n_head_kv=8, n_ff=28672, n_vocab=128256, qkv_bias=0, rope_neox=0, rope_theta=5e5, rms_eps=1e-5),
    "moe": dict(n_layer=48, n_embd=2048, n_head=32, n_head_kv=4, n_ff=0, n_vocab=151936, qkv_bias=0, qk_norm=1, rope_neox=1, rope_theta=1e6,
                rms_eps=1e-6, n_expert=128, n_expert_used=8, n_ff_exp=768),
}
HEAD_DIM = 128
# sizes of the recurrent models of bench.py
WIDTHS = {"2b": dict(width=2560, blocks=10, ff=7680, heads=20), "4b": dict(width=3072, blocks=12, ff=9216, heads=24),
          "9b": dict(width=4096, blocks=16, ff=12288, heads=32)}
L_VOCAB, L_WINDOW, L_RANK, L_DIM, L_ROT, L_VDIM, L_LIMIT, L_ALPHA = 128256, 2048, 512, 128, 64, 128, 7.0, 1.702


def decoder(name, shape, layers, n_seq, T, pos0, part="middle", kv="f16"):
    """layers: how many; part: "first" takes token ids, "last" returns logits and greedy tokens; pos0: tokens already in the cache"""
    return dict(name=name, kind="decoder", shape=shape, layers=layers, n_seq=n_seq, T=T, pos0=pos0, part=part, kv=kv)


def listed():
    return [
        # the smallest call: one token through the last quarter of a small model, with the output head (chat, one user)
        decoder("step_3b_head", "3b", 9, 1, 1, 511, part="last"),
        # the headline: one token of a large model, with the cache rows a server starts a model of this size with
        decoder("step_32b", "32b", 4, 1, 1, 2047, kv="q8_0/q4_0"),
        # eight users decoding together
        decoder("step_32b_x8", "32b", 4, 8, 1, 1023),
        # one token of a mixture of experts
        decoder("step_moe", "moe", 4, 1, 1, 1023),
        # sixteen users of it
        decoder("step_moe_x16", "moe", 4, 16, 1, 1023),
        # a short question to a small model, odd length, token ids in
        decoder("prompt_3b_77", "3b", 9, 1, 77, 0, part="first"),
        # a micro-batch of the usual size, in the middle of a long prompt
        decoder("prompt_32b_512", "32b", 3, 1, 512, 1536),
        # the largest micro-batch that servers are started with, a large model
        decoder("prompt_70b_2048", "70b", 2, 1, 2048, 0),
        # a whole prompt through the experts
        decoder("prompt_moe_1024", "moe", 2, 1, 1024, 0),
        # one product for a batch between decode and prompt sizes, the wider weight type
        dict(name="matmul_q6_64", kind="matmul", type=Q6_K, N=28672, K=8192, M=64),
        # a prompt of odd length through described layers
        dict(name="layers_prompt", kind="layers", size="4b", layers=6, T=1000, steps=0),
        # token by token through the same layers: latency
        dict(name="layers_replay", kind="layers", size="4b", layers=6, T=8, steps=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "prompt", "prompt", "matmul", "layers"])
    if kind == "matmul":
        K = 256 * _log(rng, 8, 112)
        N = _log(rng, 256, 30000)
        return dict(kind="matmul", type=rng.choice([Q4_K, Q6_K]), N=N, K=K, M=_log(rng, 1, 2048))
    if kind == "layers":
        T, steps = (_log(rng, 9, 2048), 0) if rng.random() < 0.5 else (rng.randint(1, 8), rng.randint(4, 14))
        return dict(kind="layers", size=rng.choice(sorted(WIDTHS)), layers=rng.choice([3, 6]), T=T, steps=steps)
    shape = rng.choice(sorted(SHAPES))
    layers = rng.randint(4, 9) if shape == "3b" else rng.randint(2, 4)
    kv = rng.choice(["f16", "f16", "q8_0/q4_0", "q4_0/q4_0"])
    if kind == "step":
        n_seq = rng.choice([1, 1, 2, 3, 4, 8, rng.randint(1, 16)])
        c = decoder("", shape, layers, n_seq, 1, _log(rng, 16, 2047), kv=kv, part=rng.choice(["middle", "middle", "last"]))
    else:
        c = decoder("", shape, 2, 1, _log(rng, 9, 2048), rng.choice([0, 0, _log(rng, 16, 1500)]), kv=kv, part=rng.choice(["middle", "middle", "first"]))
    del c["name"]
    return c


# ---- weights ------------------------------------------------------------------------------------------
def _gen(seed, name):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + zlib.crc32(name.encode())) % (1 << 62))


def _rand(g, *shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo


def _ints(g, shape, lo, hi):
    return torch.randint(lo, hi + 1, shape, generator=g, device="cuda", dtype=torch.int16).to(torch.uint8)


def _f16_bytes(v):
    return v.to(torch.float16).view(torch.uint8).view(-1, 2)


def make_blocks(ty, rows, K, seed, name):
    """GGUF blocks [rows * K / 256, bytes] of about N(0, 0.02)-sized weights, as a quantiser leaves them: scales in the upper half
    of their range, minima of 7.5 steps (Q4_K), codes over their whole range"""
    g, n = _gen(seed, name), rows * K // 256
    size = 100 if name == "token_embd.weight" else 1  # the residual stream begins larger than what a layer adds to it
    out = torch.empty((n, BLOCK_BYTES[ty]), dtype=torch.uint8, device="cuda")
    if ty == Q4_K:
        d = (size * _rand(g, n, lo=0.8e-4, hi=1.1e-4)).to(torch.float16)
        out[:, 0:2] = _f16_bytes(d)
        out[:, 2:4] = _f16_bytes(d.float() * _rand(g, n, lo=7.0, hi=8.0))
        sc = _ints(g, (n, 8), 28, 60)
        m = sc + _ints(g, (n, 8), 0, 6) - 3
        out[:, 4:8] = (sc[:, :4] & 63) | ((sc[:, 4:] >> 4) << 6)
        out[:, 8:12] = (m[:, :4] & 63) | ((m[:, 4:] >> 4) << 6)
        out[:, 12:16] = (sc[:, 4:] & 15) | ((m[:, 4:] & 15) << 4)
        out[:, 16:] = _ints(g, (n, 128), 0, 255)
    else:
        out[:, :192] = _ints(g, (n, 192), 0, 255)
        sc = _ints(g, (n, 16), 64, 127).view(torch.int8)
        out[:, 192:208] = torch.where(_ints(g, (n, 16), 0, 1).bool(), sc, -sc).view(torch.uint8)
        out[:, 208:210] = _f16_bytes(_rand(g, n, lo=0.9e-5, hi=1.3e-5))
    return out


def decode_blocks(ty, blocks):
    """[n, bytes] -> [n, 256] in 64 bits"""
    b = blocks.to(torch.int32)
    f16 = lambda lo, hi: blocks[:, lo:hi].contiguous().view(torch.float16).to(F64)
    n = b.shape[0]
    if ty == Q4_K:
        s = b[:, 4:16]
        sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | ((s[:, 0:4] >> 6) << 4)], 1)
        m = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1)
        q = b[:, 16:].view(n, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).reshape(n, 8, 32)
        return (f16(0, 2).view(n, 1, 1) * (sc.view(n, 8, 1) * q) - f16(2, 4).view(n, 1, 1) * m.view(n, 8, 1)).reshape(n, 256)
    ql, qh = b[:, :128].view(n, 2, 1, 2, 32), b[:, 128:192].view(n, 2, 1, 32)
    low = torch.cat([ql & 15, ql >> 4], 2).reshape(n, 2, 4, 32)
    high = torch.cat([(qh >> s) & 3 for s in (0, 2, 4, 6)], 2)
    q = (low | (high << 4)) - 32
    sc = blocks[:, 192:208].contiguous().view(torch.int8).to(torch.int32)
    return (f16(208, 210) * (sc.view(n, 16, 1) * q.reshape(n, 16, 16)).reshape(n, 256))


def wide(ty, rows, K, seed, name):
    """the same matrix [rows, K] in 64 bits"""
    blocks, out = make_blocks(ty, rows, K, seed, name), torch.empty((rows * K // 256, 256), dtype=F64, device="cuda")
    for i in range(0, len(blocks), 1 << 18):
        out[i:i + (1 << 18)] = decode_blocks(ty, blocks[i:i + (1 << 18)])
    return out.view(rows, K)


def make_vector(n, seed, name):
    """norm weights around one half, biases around zero: a layer adds to the residual stream less than it holds, as in a trained model"""
    v = torch.randn(n, generator=_gen(seed, name), device="cuda")
    return 0.5 + 0.05 * v if "norm" in name else 0.1 * v


def config(case):
    s = dict(n_expert=0, n_expert_used=0, n_ff_exp=0, qk_norm=0)
    s.update(SHAPES[case["shape"]])
    first = {"first": 0, "middle": s["n_layer"] // 2, "last": s["n_layer"] - case["layers"]}[case["part"]]
    return s, first


def tensors(case):
    """name -> (type, rows, row length) of the stage's tensors in the Q4_K_M mix; F32: vectors, or the router's matrix"""
    s, first = config(case)
    h, nq, nkv, out = s["n_embd"], s["n_head"] * HEAD_DIM, s["n_head_kv"] * HEAD_DIM, {}
    if case["part"] == "first":
        out["token_embd.weight"] = (Q4_K, s["n_vocab"], h)
    for l in range(first, first + case["layers"]):
        alt, p = Q6_K if l & 1 else Q4_K, f"blk.{l}."
        out[p + "attn_norm.weight"] = out[p + "ffn_norm.weight"] = (F32, 1, h)
        out.update({p + "attn_q.weight": (Q4_K, nq, h), p + "attn_k.weight": (Q4_K, nkv, h), p + "attn_v.weight": (alt, nkv, h),
                    p + "attn_output.weight": (Q4_K, h, nq)})
        if s["qkv_bias"]:
            out.update({p + "attn_q.bias": (F32, 1, nq), p + "attn_k.bias": (F32, 1, nkv), p + "attn_v.bias": (F32, 1, nkv)})
        if s["qk_norm"]:
            out.update({p + "attn_q_norm.weight": (F32, 1, HEAD_DIM), p + "attn_k_norm.weight": (F32, 1, HEAD_DIM)})
        if s["n_expert"]:
            E, fe = s["n_expert"], s["n_ff_exp"]
            out.update({p + "ffn_gate_inp.weight": (F32, E, h), p + "ffn_gate_exps.weight": (Q4_K, E * fe, h),
                        p + "ffn_up_exps.weight": (Q4_K, E * fe, h), p + "ffn_down_exps.weight": (alt, E * h, fe)})
        else:
            out.update({p + "ffn_gate.weight": (Q4_K, s["n_ff"], h), p + "ffn_up.weight": (Q4_K, s["n_ff"], h), p + "ffn_down.weight": (alt, h, s["n_ff"])})
    if case["part"] == "last":
        out["output_norm.weight"] = (F32, 1, h)
        out["output.weight"] = (Q6_K, s["n_vocab"], h)
    return out


def make_f32(rows, n, seed, name):
    if rows == 1:
        return make_vector(n, seed, name)
    return 0.02 * torch.randn((rows, n), generator=_gen(seed, name), device="cuda")  # the router


def inputs(case, seed):
    """[n_seq, pos0 + T] token ids, or hidden rows [n_seq, pos0 + T, width]"""
    s, _ = config(case)
    g, shape = _gen(seed, "inputs"), (case["n_seq"], case["pos0"] + case["T"])
    if case["part"] == "first":
        return torch.randint(0, s["n_vocab"], shape, generator=g, device="cuda", dtype=torch.int32)
    return 4 * torch.randn(shape + (s["n_embd"],), generator=g, device="cuda")


# ---- described layers -----------------------------------------------------------------------------------
def layer_kinds(case):
    return ["attention" if i % 3 == 2 else "recurrence" for i in range(case["layers"])]


def layer_tensors(case):
    """name -> shape; two recurrent layers to one of attention"""
    z = WIDTHS[case["size"]]
    h, W, H, ff, out = z["width"], z["width"], z["heads"], z["ff"], {"embed": (L_VOCAB, z["width"])}
    m = W // z["blocks"]
    for i, kind in enumerate(layer_kinds(case)):
        p = f"l{i}."
        out.update({p + "norm1": (h,), p + "norm1b": (h,), p + "norm2": (h,), p + "norm2b": (h,)})
        if kind == "recurrence":
            out.update({p + "mix.y": (W, h), p + "mix.y.b": (W,), p + "mix.x": (W, h), p + "mix.x.b": (W,), p + "mix.conv": (W, 4), p + "mix.conv.b": (W,),
                        p + "mix.ra": (z["blocks"], m, m), p + "mix.ra.b": (z["blocks"], m), p + "mix.ri": (z["blocks"], m, m),
                        p + "mix.ri.b": (z["blocks"], m), p + "mix.lam": (W,), p + "mix.o": (h, W)})
        else:
            out.update({p + "mix.q": (H * (L_DIM + L_ROT), h), p + "mix.dkv": (L_RANK + L_ROT, h), p + "mix.dkv.norm": (L_RANK,),
                        p + "mix.uk": (H * L_DIM, L_RANK), p + "mix.uv": (H * L_VDIM, L_RANK), p + "mix.g": (H, h), p + "mix.o": (h, H * L_VDIM)})
        out.update({p + "mlp.gate": (ff, h), p + "mlp.up": (ff, h), p + "mlp.down": (h, ff)})
    out["final.norm"] = (h,)
    return out


def make_layer_tensor(name, shape, seed):
    """bf16; sized so that gates, decays and attention scores all vary"""
    g, leaf = _gen(seed, name), name.split(".", 1)[-1]
    w = torch.randn(shape, generator=g, device="cuda")
    if leaf == "mix.dkv.norm":
        w = 1 + 0.2 * w
    elif "norm" in leaf:
        w = 0.3 * w
    elif leaf == "mix.lam":
        w = _rand(g, *shape, lo=-5.0, hi=-0.5)
    elif leaf.endswith(".b"):
        w = 0.3 * w
    elif name == "embed":
        w = 0.02 * w
    else:
        w = w * (2.0 if leaf == "mix.q" else 1.0) / math.sqrt(shape[-1])
    return w.to(torch.bfloat16)


def layer_tokens(case, seed):
    return torch.randint(0, L_VOCAB, (case["T"] + case["steps"],), generator=_gen(seed, "inputs"), device="cuda", dtype=torch.int32)


# ---- the user's side --------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"decoder": prepare_decoder, "matmul": prepare_matmul, "layers": prepare_layers}[case["kind"]](case, seed)


def kv_types(case):
    return {"f16": (KV_F16, KV_F16), "q8_0/q4_0": (KV_Q8_0, KV_Q4_0), "q4_0/q4_0": (KV_Q4_0, KV_Q4_0)}[case["kv"]]


def prepare_decoder(case, seed):
    from mesh_llm_b200.stage import Stage

    s, first = config(case)
    n_seq, T, pos0 = case["n_seq"], case["T"], case["pos0"]
    ubatch = max(512, T)
    kt, vt = kv_types(case)
    st = Stage(head_dim=HEAD_DIM, layer_begin=first, layer_end=first + case["layers"], n_ctx=(pos0 + T + 256) // 256 * 256, n_seq=n_seq, n_ubatch=ubatch,
               has_embd=int(case["part"] == "first"), has_output=int(case["part"] == "last"), kv_type_k=kt, kv_type_v=vt, **s)
    for name, (ty, rows, n) in tensors(case).items():
        w = make_f32(rows, n, seed, name) if ty == F32 else make_blocks(ty, rows, n, seed, name)
        st.set_tensor(name, ty, w.cpu().numpy())
    x = inputs(case, seed)
    for i in range(n_seq):  # the tokens that are in the cache already
        for lo in range(0, pos0, ubatch):
            part = x[i, lo:min(pos0, lo + ubatch)].contiguous()
            st.forward(**{"tokens" if case["part"] == "first" else "hidden_in": part}, n_seq=1, T=len(part), pos0=lo, seq0=i)
    new = x[:, pos0:].reshape(n_seq * T, *x.shape[2:]).contiguous()
    out = dict(hidden_out=torch.empty((n_seq * T, s["n_embd"]), device="cuda"))
    if case["part"] == "last":
        out = dict(logits=torch.empty((n_seq, s["n_vocab"]), device="cuda"), next_tokens=torch.empty(n_seq, dtype=torch.int32, device="cuda"))
    st.synchronize()
    call = {"tokens" if case["part"] == "first" else "hidden_in": new, "n_seq": n_seq, "T": T, "pos0": pos0, **out}
    return dict(case=case, stage=st, call=call)


def prepare_matmul(case, seed):
    from mesh_llm_b200 import ops

    ty, N, K = case["type"], case["N"], case["K"]
    W = ops.upload_weights(ty, make_blocks(ty, N, K, seed, "W"), N, K)
    return dict(case=case, W=W, x=torch.randn((case["M"], K), generator=_gen(seed, "x"), device="cuda"))


def prepare_layers(case, seed):
    from mesh_llm_b200 import capi
    from mesh_llm_b200.stage import Stage

    z, layers = WIDTHS[case["size"]], []
    for kind in layer_kinds(case):
        l = capi.LayerConfig(ffn=capi.FFN_CLAMPED_GLU, n_ff=z["ff"], glu_limit=L_LIMIT, glu_alpha=L_ALPHA)
        if kind == "attention":
            l.mixer, l.n_head, l.qk_dim, l.rot_dim, l.rot_dims = capi.MIXER_LATENT_ATTN, z["heads"], L_DIM, L_ROT, L_ROT
            l.v_dim, l.kv_rank, l.window, l.rope_base, l.attn_scale = L_VDIM, L_RANK, L_WINDOW, 1e4, (L_DIM + L_ROT) ** -0.5
        else:
            l.mixer, l.rec_width, l.rec_blocks, l.conv_taps, l.rec_decay = capi.MIXER_LINEAR_REC, z["width"], z["blocks"], 4, 8.0
        layers.append(l)
    stack = capi.StackConfig(loop_times=1, precision=capi.PRECISION_BF16, embd_scale=z["width"] ** 0.5, norm_offset=1.0)
    n = case["T"] + case["steps"]
    st = Stage(stack=stack, layers=layers, n_layer=case["layers"], n_embd=z["width"], n_vocab=L_VOCAB, n_ctx=(n + 256) // 256 * 256, n_seq=1,
               n_ubatch=max(512, case["T"]))
    for name, shape in layer_tensors(case).items():
        st.set_tensor(name, BF16, make_layer_tensor(name, shape, seed).view(torch.int16).cpu().numpy())
    st.synchronize()
    dev = dict(device="cuda")
    return dict(case=case, stage=st, tokens=layer_tokens(case, seed), token=torch.empty(1, dtype=torch.int32, **dev),
                logits=torch.empty((1, L_VOCAB), **dev), next=torch.empty(1, dtype=torch.int32, **dev), every=torch.empty((1 + case["steps"], L_VOCAB), **dev))


def run(state):
    case = state["case"]
    if case["kind"] == "matmul":
        from mesh_llm_b200 import ops

        return ops.mul_mat(case["type"], state["W"], state["x"], case["N"], case["K"])
    if case["kind"] == "decoder":
        hidden, logits, tokens = state["stage"].forward(**state["call"])
        return [logits, tokens] if case["part"] == "last" else [hidden]
    # a prompt, then the following tokens one by one, as a replay feeds them: fixed buffers, logits kept after each
    st, T, every = state["stage"], case["T"], state["every"]
    st.forward(tokens=state["tokens"][:T], n_seq=1, T=T, pos0=0, logits=state["logits"], next_tokens=state["next"])
    every[0].copy_(state["logits"][0])
    for i in range(case["steps"]):
        state["token"].copy_(state["tokens"][T + i:T + i + 1])
        st.forward(tokens=state["token"], n_seq=1, T=1, pos0=T + i, logits=state["logits"], next_tokens=state["next"])
        every[1 + i].copy_(state["logits"][0])
    return [every]


# ---- floors ---------------------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "matmul":
        ty, N, K, M = (case[k] for k in ("type", "N", "K", "M"))
        return dict(bytes=N * K // 256 * BLOCK_BYTES[ty] + 4 * M * (K + N), flops=2 * M * N * K)
    if case["kind"] == "layers":
        z, T, steps = WIDTHS[case["size"]], case["T"], case["steps"]
        params = sum(math.prod(s) for n, s in layer_tensors(case).items() if n != "embed")
        head, n_att = L_VOCAB * z["width"], layer_kinds(case).count("attention")
        att = n_att * z["heads"] * 2 * (L_DIM + L_ROT + L_VDIM)
        seen = sum(i + 1 for i in range(T)) + sum(T + i + 1 for i in range(steps))
        # every weight once for the prompt and once a step, the head with each; logits; states and caches are small beside them
        return dict(bytes=(1 + steps) * (2 * (params + head) + 4 * L_VOCAB) + 2 * (T + steps) * z["width"],
                    flops=2 * (T + steps) * params + (1 + steps) * 2 * head + att * seen)
    s, _ = config(case)
    rows, L = case["n_seq"] * case["T"], case["pos0"] + case["T"]
    nbytes = flops = 0
    for name, (ty, n, k) in tensors(case).items():
        size = n * k // 256 * BLOCK_BYTES[ty] if ty != F32 else 4 * n * k
        if name == "token_embd.weight":
            nbytes += rows * size // n
        elif "_exps" in name:
            # the experts that the tokens choose: with uniform routing, E (1 - (1 - k/E)^rows) of them
            E, ku = s["n_expert"], s["n_expert_used"]
            nbytes += int(size * (1 - (1 - ku / E) ** rows))
            flops += 2 * rows * ku * (n // E) * k
        elif ty != F32 or n > 1:
            nbytes += size
            flops += 2 * (case["n_seq"] if name == "output.weight" else rows) * n * k
        else:
            nbytes += size
    row = {"f16": 4 * HEAD_DIM, "q8_0/q4_0": 34 * HEAD_DIM // 32 + 18 * HEAD_DIM // 32, "q4_0/q4_0": 36 * HEAD_DIM // 32}[case["kv"]]
    nbytes += case["layers"] * case["n_seq"] * L * s["n_head_kv"] * row  # keys and values, read or written
    seen = case["n_seq"] * sum(case["pos0"] + t + 1 for t in range(case["T"]))
    flops += case["layers"] * 4 * HEAD_DIM * s["n_head"] * seen
    nbytes += rows * (4 if case["part"] == "first" else 4 * s["n_embd"]) + (case["n_seq"] * 4 * s["n_vocab"] if case["part"] == "last" else rows * 4 * s["n_embd"])
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """A product sums int8 codes exactly and scales the sums in f32: 1e-7 off the 64-bit result, whatever the kernel.  Inside a
    stage an activation whose f32 value lies beside a rounding tie takes the neighbouring Q8 code (or f16, bf16 value) when sums
    are taken in another order, and the next layers amplify it: two kernels for the same products leave rows 2e-3 to 7e-3 apart
    (dense layers) and 5e-5 to 7e-5 (experts, whose part of the residual stream is smaller; a token between two experts is further off)."""
    if case["kind"] == "matmul":
        return {"rel": 2e-6}
    if case["kind"] == "layers":
        return {"rel": 1.7e-2}
    return {"rel": 2e-3 if case["shape"] == "moe" else 2.8e-2, "differ": 0.01}


# ---- 64 bits --------------------------------------------------------------------------------------------
def q8(x):
    """the activation quantiser of the K-quant path, whose codes are chosen in f32: blocks of 256, d = max / 127, code = rint(x (1 / d))"""
    b = x.float().reshape(-1, 256)
    d = b.abs().amax(1, keepdim=True) / 127
    return (torch.round(b * torch.where(d > 0, 1 / d, torch.zeros_like(d))).to(F64) * d.to(F64)).reshape(x.shape)


def rms(x, w, eps, offset=0.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * (w.to(F64) + offset)


def rotate(x, pos, theta, halves):
    """x [..., T, heads, d]: pairs (i, i + d/2) or (2i, 2i + 1) turned by pos * theta^(-2i/d)"""
    d = x.shape[-1]
    a = pos.to(F64)[:, None, None] * theta ** (-torch.arange(0, d, 2, device=x.device, dtype=F64) / d)
    c, s, y = torch.cos(a), torch.sin(a), torch.empty_like(x)
    i0, i1 = (slice(0, d // 2), slice(d // 2, d)) if halves else (slice(0, d, 2), slice(1, d, 2))
    y[..., i0], y[..., i1] = x[..., i0] * c - x[..., i1] * s, x[..., i0] * s + x[..., i1] * c
    return y


def stored(x, ty):
    """rows as the cache holds them: f16, or q8_0 / q4_0 blocks of 32 with an f16 scale"""
    if ty == KV_F16:
        return x.to(torch.float16).to(F64)
    b = x.float().reshape(-1, 32)
    if ty == KV_Q8_0:
        d = b.abs().amax(1, keepdim=True) / 127
        v = b * torch.where(d > 0, 1 / d, torch.zeros_like(d))
        q = torch.trunc(v + 0.5 * torch.sign(v))
    else:
        d = b.gather(1, b.abs().argmax(1, keepdim=True)) / -8
        q = torch.clamp(torch.trunc(b * torch.where(d != 0, 1 / d, torch.zeros_like(d)) + 8.5), max=15) - 8
    return (q * d.to(torch.float16).float()).to(torch.float16).to(F64).reshape(x.shape)


def attend(q, k, v, scale, first, window=None):
    """q [T, H, d] at positions first .., k, v [L, Hkv, d] -> [T, H, dv], 256 queries at a time"""
    out, rep = [], q.shape[1] // k.shape[1]
    j = torch.arange(k.shape[0], device=q.device)
    kk, vv = k.permute(1, 2, 0), v.permute(1, 0, 2)
    for lo in range(0, q.shape[0], 256):
        part = q[lo:lo + 256]
        i = torch.arange(lo, lo + part.shape[0], device=q.device)[:, None] + first
        hide = (j > i) if window is None else ((j > i) | (i - j >= window))
        s = torch.matmul(part.permute(1, 0, 2).reshape(k.shape[1], -1, q.shape[-1]), kk) * scale
        s = s.view(k.shape[1], rep, part.shape[0], -1).masked_fill(hide, -math.inf)
        p = torch.softmax(s, -1).view(k.shape[1], rep * part.shape[0], -1)
        out.append(torch.matmul(p, vv).view(q.shape[1], part.shape[0], -1).permute(1, 0, 2))
    return torch.cat(out)


def exact_decoder(case, seed):
    s, first = config(case)
    h, nh, nkv, n_seq, T, pos0 = s["n_embd"], s["n_head"], s["n_head_kv"], case["n_seq"], case["T"], case["pos0"]
    all_t, L = tensors(case), case["pos0"] + case["T"]

    def matrix(name):
        ty, rows, k = all_t[name]
        return make_f32(rows, k, seed, name).to(F64) if ty == F32 else wide(ty, rows, k, seed, name)

    def product(name, a):
        return q8(a) @ matrix(name).T

    x = inputs(case, seed)
    if case["part"] == "first":
        ty, rows, k = all_t["token_embd.weight"]
        blocks = make_blocks(ty, rows, k, seed, "token_embd.weight").view(rows, k // 256, -1)
        x = decode_blocks(ty, blocks[x.reshape(-1).long()].reshape(-1, BLOCK_BYTES[ty])).view(n_seq, L, h)
    x = x.to(F64).reshape(n_seq * L, h)
    pos, kt_vt = torch.arange(L, device="cuda"), kv_types(case)
    for l in range(first, first + case["layers"]):
        p = f"blk.{l}."
        a = rms(x, matrix(p + "attn_norm.weight"), s["rms_eps"])
        q, k, v = (product(p + f"attn_{t}.weight", a) for t in "qkv")
        if s["qkv_bias"]:
            q, k, v = (y + matrix(p + f"attn_{t}.bias") for t, y in zip("qkv", (q, k, v)))
        q, k, v = (y.view(n_seq, L, n, HEAD_DIM) for y, n in ((q, nh), (k, nkv), (v, nkv)))
        if s["qk_norm"]:
            q, k = rms(q, matrix(p + "attn_q_norm.weight"), s["rms_eps"]), rms(k, matrix(p + "attn_k_norm.weight"), s["rms_eps"])
        q, k = rotate(q, pos, s["rope_theta"], s["rope_neox"]), rotate(k, pos, s["rope_theta"], s["rope_neox"])
        k, v = stored(k, kt_vt[0]), stored(v, kt_vt[1])
        att = torch.cat([attend(q[i], k[i], v[i], HEAD_DIM ** -0.5, 0).reshape(L, nh * HEAD_DIM) for i in range(n_seq)])
        x = x + product(p + "attn_output.weight", att)
        a = rms(x, matrix(p + "ffn_norm.weight"), s["rms_eps"])
        if not s["n_expert"]:
            g = product(p + "ffn_gate.weight", a)
            x = x + product(p + "ffn_down.weight", g * torch.sigmoid(g) * product(p + "ffn_up.weight", a))
            continue
        E, ku, fe = s["n_expert"], s["n_expert_used"], s["n_ff_exp"]
        w, ids = torch.topk(torch.softmax(a @ matrix(p + "ffn_gate_inp.weight").T, -1), ku)
        w = w / w.sum(-1, keepdim=True)
        gate, up, down = (matrix(p + f"ffn_{t}_exps.weight").view(E, -1, n) for t, n in (("gate", h), ("up", h), ("down", fe)))
        a, y = q8(a), torch.zeros_like(x)
        for e in range(E):
            t, slot = torch.nonzero(ids == e, as_tuple=True)
            if len(t):
                g = a[t] @ gate[e].T
                y[t] += w[t, slot, None] * (q8(g * torch.sigmoid(g) * (a[t] @ up[e].T)) @ down[e].T)
        x = x + y
    x = x.view(n_seq, L, h)
    if case["part"] == "last":
        return [product("output.weight", rms(x[:, -1], matrix("output_norm.weight"), s["rms_eps"])), None]
    return [x[:, pos0:].reshape(n_seq * T, h)]


def exact_layers(case, seed):
    z, shapes = WIDTHS[case["size"]], layer_tensors(case)
    h, H = z["width"], z["heads"]
    t = lambda name: make_layer_tensor(name, shapes[name], seed).to(F64)
    norm = lambda x, name: rms(x, t(name), 1e-6, 1.0)
    x = t("embed")[layer_tokens(case, seed).long()] * math.sqrt(h)
    n, pos = x.shape[0], torch.arange(x.shape[0], device="cuda")
    for i, kind in enumerate(layer_kinds(case)):
        p = f"l{i}."
        a = norm(x, p + "norm1")
        if kind == "recurrence":
            y = torch.nn.functional.gelu(a @ t(p + "mix.y").T + t(p + "mix.y.b"), approximate="tanh")
            u = torch.nn.functional.pad(a @ t(p + "mix.x").T + t(p + "mix.x.b"), (0, 0, 3, 0))
            u = sum(u[k:k + n] * t(p + "mix.conv")[:, k] for k in range(4)) + t(p + "mix.conv.b")
            r, g = (torch.sigmoid(torch.einsum("bij,tbj->tbi", t(p + m), u.reshape(n, z["blocks"], -1)) + t(p + m + ".b")).reshape(n, -1) for m in ("mix.ra", "mix.ri"))
            log_a = -8 * r * torch.nn.functional.softplus(t(p + "mix.lam"))
            decay, new = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * g * u
            state, states = torch.zeros_like(new[0]), []
            for k in range(n):
                state = decay[k] * state + new[k]
                states.append(state)
            o = (torch.stack(states) * y) @ t(p + "mix.o").T
        else:
            q, c = (a @ t(p + "mix.q").T).view(n, H, L_DIM + L_ROT), a @ t(p + "mix.dkv").T
            lat, shared = rms(c[:, :L_RANK], t(p + "mix.dkv.norm"), 1e-6), rotate(c[:, None, L_RANK:], pos, 1e4, False)
            q = torch.cat([q[..., :L_DIM], rotate(q[..., L_DIM:], pos, 1e4, False)], -1)
            k = torch.cat([(lat @ t(p + "mix.uk").T).view(n, H, L_DIM), shared.expand(n, H, L_ROT)], -1)
            o = attend(q, k, (lat @ t(p + "mix.uv").T).view(n, H, L_VDIM), (L_DIM + L_ROT) ** -0.5, 0, L_WINDOW)
            o = (o * torch.sigmoid(a @ t(p + "mix.g").T)[..., None]).reshape(n, -1) @ t(p + "mix.o").T
        x = x + norm(o, p + "norm1b")
        a = norm(x, p + "norm2")
        g, u = (a @ t(p + "mlp.gate").T).clamp(max=L_LIMIT), (a @ t(p + "mlp.up").T).clamp(-L_LIMIT, L_LIMIT)
        x = x + norm((g * torch.sigmoid(L_ALPHA * g) * (u + 1)) @ t(p + "mlp.down").T, p + "norm2b")
    return [norm(x[case["T"] - 1:], "final.norm") @ t("embed").T]


def exact(case, seed):
    if case["kind"] == "matmul":
        ty, N, K, M = (case[k] for k in ("type", "N", "K", "M"))
        return q8(torch.randn((M, K), generator=_gen(seed, "x"), device="cuda").to(F64)) @ wide(ty, N, K, seed, "W").T
    return exact_decoder(case, seed) if case["kind"] == "decoder" else exact_layers(case, seed)
