"""The work that users of this framework give it, as cases that can be prepared, run and timed.

Three kinds of program stand behind the cases:

  block   a decoder that runs its own mixers and calls the MoE block layer by layer (wd_moe_forward): one token, or the
          two to four tokens of a speculative verify. A pass is one walk over the layers of the engine.
  stack   greedy decoding on the device: embedding row -> MoE stack (wd_stack_step) -> output head with arg-max. A pass
          is a few tokens; the next pass goes on from the last token, as a decode does. With every expert resident, or
          with the expert cache capped so that some picks stream in from host memory.
  dense   the plain Llama-style decoder: a prompt is read and tokens are generated (wd_dense_decoder_decode), and the
          last step's logits are fetched.

Weights and inputs are drawn from the seed on the GPU: encoded N(0, 0.02) weights where the library has an encoder,
random block bytes with scales of the same size otherwise; activations are N(0, 1), the router carries a per-expert
bias of N(0, 1), prompts are uniform token ids. Every result of this library is defined bit for bit, so the outputs of
two correct implementations are equal and the tolerance is "exact".
"""
import ctypes
import math

import numpy as np
import torch

import warpdecode_b200 as wd

BLOCK = {"q4_0": (wd.TYPE_Q4_0, 32, 18), "q8_0": (wd.TYPE_Q8_0, 32, 34), "iq4_nl": (wd.TYPE_IQ4_NL, 32, 18),
         "iq3_s": (wd.TYPE_IQ3_S, 256, 110), "iq2_s": (wd.TYPE_IQ2_S, 256, 82)}
# f16 block scale that makes weights of random block bytes about as large as N(0, 0.02) ones
SCALE = {"iq3_s": 1.4e-4, "iq2_s": 3.6e-4, "iq4_nl": 3.3e-4}
SIGMA = 0.02


def _block(name, hidden, ffn, experts, top_k, shared, layers, tokens, gate="iq3_s", down="iq3_s", router="q8_0"):
    return dict(name=name, kind="block", hidden=hidden, ffn=ffn, experts=experts, top_k=top_k, shared=shared, layers=layers,
                tokens=tokens, gate=gate, down=down, router=router)


def listed():
    return [
        # the smallest block of the tests: a call is launch and hand-over latency
        _block("block_small_1", 512, 256, 32, 4, 256, 2, 1),
        # the block of the 48-layer model, one token per call: plain decoding behind a host engine's mixers
        _block("block_model_1", 2048, 512, 512, 10, 512, 8, 1),
        # the same block with the four tokens of a speculative verify step
        _block("block_model_4", 2048, 512, 512, 10, 512, 8, 4),
        # IQ2_S experts on the power-of-two geometry, a two-token verify, no shared expert
        _block("block_iq2s_2", 1024, 512, 128, 8, 0, 6, 2, gate="iq2_s", down="iq2_s"),
        # the block shape of the reference's own model: IQ2_S gate/up, IQ4_NL down, F32 router
        _block("block_ref_1", 2560, 640, 512, 10, 640, 4, 1, gate="iq2_s", down="iq4_nl", router="f32"),
        _block("block_ref_4", 2560, 640, 512, 10, 640, 4, 4, gate="iq2_s", down="iq4_nl", router="f32"),
        # a small geometry off the powers of two, three tokens
        _block("block_ragged_3", 768, 192, 64, 6, 256, 3, 3, gate="iq3_s", down="iq4_nl"),
        # the headline: greedy decoding of the 48-layer model with the full head
        dict(name="stack_model", kind="stack", hidden=2048, ffn=512, experts=512, top_k=10, shared=512, layers=48,
             vocab=151936, tokens=8, cached=1.0),
        # the expert cache holds half of the experts; misses stream from page-locked host memory
        dict(name="stack_capped", kind="stack", hidden=2048, ffn=512, experts=512, top_k=10, shared=512, layers=4,
             vocab=32768, tokens=4, cached=0.5),
        # the dense benchmark: 8 prompt tokens, 64 generated
        dict(name="dense_generate", kind="dense", hidden=2048, heads=32, kv_heads=8, head_dim=64, ffn=8192, vocab=128256,
             layers=16, prompt=8, generate=64, style="llama"),
        # the same model reading a longer prompt (a document, a chat history) and answering briefly
        dict(name="dense_prompt", kind="dense", hidden=2048, heads=32, kv_heads=8, head_dim=64, ffn=8192, vocab=128256,
             layers=16, prompt=480, generate=32, style="llama"),
        # a small model as files carry them: Q8_0 head and down matrices, q/k/v biases, head norms, odd vocabulary
        dict(name="dense_file", kind="dense", hidden=1024, heads=16, kv_heads=4, head_dim=64, ffn=2816, vocab=32003,
             layers=8, prompt=37, generate=24, style="file"),
    ]


def _spread(rng, low, high, step=1):
    """A multiple of `step` between low and high, spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(low), math.log(high)))
    return int(min(high, max(low, round(v / step) * step)))


def draw(rng):
    kind = rng.choices(["tiled", "plain", "stack", "dense"], [4, 3, 2, 4])[0]
    if kind == "tiled":
        while True:
            c = _block(None, 256 << rng.randint(1, 3), 256 << rng.randint(0, 2), _spread(rng, 16, 512, 8), rng.randint(2, 12),
                       rng.choice([0, 128, 256, 384, 512, 640]), rng.randint(1, 4), rng.randint(1, 4))
            c["gate"] = rng.choice(["iq3_s", "iq3_s", "iq2_s"])
            c["down"] = rng.choice(["iq3_s", c["gate"]])
            if c["top_k"] * c["ffn"] * c["hidden"] <= 10 * 512 * 2048 and c["shared"] <= 2 * c["hidden"]:
                break
    elif kind == "plain":
        down = rng.choice(["iq4_nl", "iq4_nl", "iq3_s", "iq2_s"])
        ffn = 64 * rng.randint(2, 12) if down == "iq4_nl" else rng.choice([256, 512, 768])
        c = _block(None, 256 * rng.choice([3, 5, 6, 7, 9, 10, 11]), ffn, _spread(rng, 16, 512, 8), rng.randint(2, 10),
                   rng.choice([0, 128, 256, 384, 640]), rng.randint(1, 3), rng.randint(1, 4),
                   gate=rng.choice(["iq2_s", "iq3_s"]), down=down, router=rng.choice(["f32", "q8_0"]))
    elif kind == "stack":
        while True:
            c = dict(kind="stack", hidden=256 << rng.randint(1, 3), ffn=256 << rng.randint(0, 1), experts=_spread(rng, 32, 512, 8),
                     top_k=rng.randint(2, 10), shared=rng.choice([128, 256, 384, 512]), layers=_spread(rng, 2, 24),
                     vocab=_spread(rng, 4096, 151936, 32), tokens=rng.randint(1, 8), cached=1.0)
            if c["top_k"] * c["ffn"] * c["hidden"] <= 10 * 512 * 2048:
                break
    else:
        head_dim = rng.choice([32, 64, 64, 96, 128])
        kv = rng.choice([1, 2, 4, 8])
        hidden = 256 << rng.randint(1, 3)
        heads = kv * max(1, min(4, round(hidden / head_dim / kv)))
        prompt = _spread(rng, 1, 600)
        generate = _spread(rng, 1, 64)
        layers = max(2, min(_spread(rng, 2, 16), 6000 // (prompt + generate)))
        c = dict(kind="dense", hidden=hidden, heads=heads, kv_heads=kv, head_dim=head_dim, ffn=_spread(rng, 512, 8192, 32),
                 vocab=_spread(rng, 2000, 128256), layers=layers, prompt=prompt, generate=generate,
                 style=rng.choice(["llama", "llama", "file"]))
    c.pop("name", None)
    return c


# ---- sizes ----------------------------------------------------------------------------------------------------------
def _bytes(t, rows, cols):
    if t == "f32":
        return rows * cols * 4
    _, per, size = BLOCK[t]
    return rows * (cols // per) * size


def _moe_layer(c, tokens):
    """(bytes, multiply-adds) of one block call: the picked experts once each, the router and the shared expert once."""
    H, F, E, K, S = c["hidden"], c["ffn"], c["experts"], c["top_k"], c["shared"]
    gate, down = c.get("gate", "iq3_s"), c.get("down", "iq3_s")
    picked = E * (1.0 - (1.0 - K / E) ** tokens)
    b = picked * (2 * _bytes(gate, F, H) + _bytes(down, H, F)) + _bytes(c.get("router", "q8_0"), E, H)
    m = K * 3 * H * F + E * H
    if S:
        b += 3 * _bytes("q8_0", S, H) + 4 * H
        m += 3 * H * S + H
    return b + 8 * tokens * H, m * tokens


def work(c):
    if c["kind"] == "block":
        b, m = _moe_layer(c, c["tokens"])
        return {"bytes": b * c["layers"], "flops": 2.0 * m * c["layers"]}
    if c["kind"] == "stack":
        b, m = _moe_layer(c, 1)
        b, m = b * c["layers"] + _bytes("q8_0", c["vocab"], c["hidden"]), m * c["layers"] + c["vocab"] * c["hidden"]
        return {"bytes": b * c["tokens"], "flops": 2.0 * m * c["tokens"]}
    H, D, F, V = c["hidden"], c["head_dim"], c["ffn"], c["vocab"]
    q, kv, P, G = c["heads"] * D, c["kv_heads"] * D, c["prompt"], c["generate"]
    wide = "q8_0" if c["style"] == "file" else "q4_0"
    layer = _bytes("q4_0", q + 2 * kv, H) + _bytes("q4_0", H, q) + _bytes("q4_0", 2 * F, H) + _bytes(wide, H, F)
    # the prompt can be read in one pass over the weights; every further token is a pass of its own
    passes = max(1, G)
    steps = P + G - 1
    cache = c["layers"] * 2 * kv * 4 * (steps + sum(range(P, steps)))
    per_token = (q + 2 * kv) * H + H * q + 3 * F * H
    attend = c["layers"] * 2 * q * steps * (steps + 1) // 2
    return {"bytes": passes * (c["layers"] * layer + _bytes(wide, V, H)) + cache,
            "flops": 2.0 * (c["layers"] * per_token * steps + V * H * passes + attend)}


def tolerance(c):
    return "exact"


# ---- preparation ----------------------------------------------------------------------------------------------------
_streams = []


def _stream():
    """The stream a program runs its calls on (one for all of them)."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _random_blocks(t, rows, cols, gen):
    """Random bytes of a block format with scales of a sensible size, on the device."""
    _, per, size = BLOCK[t]
    n = rows * (cols // per)
    raw = torch.randint(0, 256, (n, size), dtype=torch.uint8, device="cuda", generator=gen)
    d = (torch.rand(n, device="cuda", generator=gen) + 0.5) * SCALE[t]
    raw[:, 0:2] = d.to(torch.float16).view(torch.uint8).reshape(n, 2)
    return raw


def _q8_0(rows, cols, sigma, seed, stream_id):
    w = torch.empty(_bytes("q8_0", rows, cols), dtype=torch.uint8, device="cuda")
    wd.synth_tensor_device(wd.TYPE_Q8_0, rows, cols, sigma, seed, stream_id, w.data_ptr())
    torch.cuda.synchronize()
    return w


def _ptr(a):
    return ctypes.c_void_p(a.data_ptr() if isinstance(a, torch.Tensor) else a.ctypes.data)


def _check(rc):
    if rc:
        raise RuntimeError(wd.lib().wd_last_error().decode())


def _moe_engine(c, seed, tokens, cache_mib=0):
    gate, down, router = c.get("gate", "iq3_s"), c.get("down", "iq3_s"), c.get("router", "q8_0")
    H, F, E, S = c["hidden"], c["ffn"], c["experts"], c["shared"]
    eng = wd.Engine(H, F, E, c["top_k"], S, c["layers"], expert_type=BLOCK[gate][0], down_type=BLOCK[down][0],
                    router_f32=router == "f32", max_tokens=tokens, cache_mib=cache_mib)
    tiled = all(v % 256 == 0 and (v & (v - 1)) == 0 for v in (H, F)) and router == "q8_0"
    if tiled and gate == "iq3_s" and down == "iq3_s":
        eng.synth_model(seed, SIGMA, 1.0)
        return eng
    gen, lib = _gen(seed), wd.lib()
    for l in range(c["layers"]):
        bias = np.ascontiguousarray(torch.randn(E, device="cuda", generator=gen).cpu().numpy())
        if router == "f32":
            r = (torch.randn(E, H, device="cuda", generator=gen) * SIGMA).cpu().numpy()
            _check(lib.wd_set_router_f32(eng.h, l, _ptr(r), _ptr(bias)))
        else:
            r = _q8_0(E, H, SIGMA, seed, 16 * l).cpu().numpy()
            _check(lib.wd_set_router(eng.h, l, _ptr(r), _ptr(bias)))
        if S:
            vec = (torch.randn(H, device="cuda", generator=gen) * SIGMA).cpu().numpy()
            w = [_q8_0(rows, cols, SIGMA, seed, 16 * l + i).cpu().numpy() for i, rows, cols in ((1, S, H), (2, S, H), (3, H, S))]
            _check(lib.wd_set_shared(eng.h, l, _ptr(vec), *[_ptr(a) for a in w]))
        g, u = _random_blocks(gate, E * F, H, gen), _random_blocks(gate, E * F, H, gen)
        d = _random_blocks(down, E * H, F, gen)
        torch.cuda.synchronize()
        _check(lib.wd_set_experts_device(eng.h, l, _ptr(g), _ptr(u), _ptr(d)))
        torch.cuda.synchronize()
        del g, u, d
    return eng


def _prepare_block(c, seed):
    eng = _moe_engine(c, seed, c["tokens"])
    gen = _gen(seed + 1)
    x = torch.randn(c["layers"], c["tokens"], c["hidden"], device="cuda", generator=gen)
    return dict(case=c, eng=eng, x=x, out=torch.zeros_like(x))


def _prepare_stack(c, seed):
    mib = 0
    if c["cached"] < 1.0:
        expert = 2 * _bytes("iq3_s", c["ffn"], c["hidden"]) + _bytes("iq3_s", c["hidden"], c["ffn"])
        mib = int(c["cached"] * c["layers"] * c["experts"] * expert) >> 20
    eng = _moe_engine(c, seed, 1, mib)
    H, V = c["hidden"], c["vocab"]
    table = _q8_0(V, H, 1.0, seed, 100000)
    w = _q8_0(V, H, SIGMA, seed, 100001)
    head = wd.HeadQ8_0(V, H, ggml_dev_ptr=w.data_ptr())
    torch.cuda.synchronize()
    token = torch.randint(0, V, (1,), dtype=torch.int32, device="cuda", generator=_gen(seed + 1))
    return dict(case=c, eng=eng, table=table, head=head, token=token, residual=torch.zeros(H, device="cuda"),
                logits=torch.zeros(V, device="cuda"), generated=torch.zeros(c["tokens"], dtype=torch.int32, device="cuda"))


def _prepare_dense(c, seed):
    dec = wd.DenseDecoder(c["hidden"], c["heads"], c["kv_heads"], c["head_dim"], c["ffn"], c["vocab"], c["layers"],
                          c["prompt"] + c["generate"])
    dec.synth(seed, SIGMA)
    rng = np.random.default_rng(seed)
    if c["style"] == "file":
        dec.set_tensor(0, wd.DT_OUTPUT, _q8_0(c["vocab"], c["hidden"], SIGMA, seed, 200000).cpu().numpy(), wd.TYPE_Q8_0)
        for l in range(c["layers"]):
            dec.set_tensor(l, wd.DT_W_DOWN, _q8_0(c["hidden"], c["ffn"], SIGMA, seed, 200001 + l).cpu().numpy(), wd.TYPE_Q8_0)
            for which in (wd.DT_ATTN_NORM, wd.DT_FFN_NORM, wd.DT_Q_NORM, wd.DT_K_NORM):
                dec.set_tensor(l, which, (1.0 + 0.1 * rng.standard_normal(dec.vector_len(which))).astype(np.float32))
            dec.set_tensor(l, wd.DT_BQKV, (0.1 * rng.standard_normal(dec.vector_len(wd.DT_BQKV))).astype(np.float32))
    return dict(case=c, dec=dec, prompt=rng.integers(0, c["vocab"], c["prompt"]).astype(np.int32))


def prepare(case, seed):
    seed = int(seed) & 0x7fffffff
    state = {"block": _prepare_block, "stack": _prepare_stack, "dense": _prepare_dense}[case["kind"]](case, seed)
    torch.cuda.synchronize()
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------
def _run_block(s):
    c, eng, sp = s["case"], s["eng"], _stream().cuda_stream
    for l in range(c["layers"]):
        eng.forward_device(l, s["x"][l].data_ptr(), s["out"][l].data_ptr(), sp, c["tokens"])
    return s["out"]


def _run_stack(s):
    c, sp = s["case"], _stream().cuda_stream
    H, V, n = c["hidden"], c["vocab"], c["tokens"]
    with torch.cuda.stream(_stream()):
        for i in range(n):
            wd.embed_q8_0(s["table"].data_ptr(), V, H, s["token"].data_ptr(), s["residual"].data_ptr(), sp)
            s["eng"].stack_step_device(s["residual"].data_ptr(), sp)
            s["head"].argmax(s["residual"].data_ptr(), s["token"].data_ptr(), s["logits"].data_ptr(), None, sp)
            s["generated"][i:i + 1].copy_(s["token"], non_blocking=True)
    return {"tokens": s["generated"], "residual": s["residual"], "logits": s["logits"]}


def _run_dense(s):
    tokens, _ = s["dec"].decode(s["prompt"], s["case"]["generate"])
    logits, hidden = s["dec"].read()
    return {"tokens": tokens, "logits": logits, "hidden": hidden}


def run(state):
    return {"block": _run_block, "stack": _run_stack, "dense": _run_dense}[state["case"]["kind"]](state)
