"""The work that a user of this framework has it do, as cases that can be timed and compared.

Kinds of case, each through the entry points that a program calls:

* ``token``    one sequence generates tokens: ``KhqRuntime.khq_step_fused`` (``mode="fused"``), ``khq_prestep`` +
               ``khq_step`` (``mode="prestep"``) or ``khq_capture_unroped`` + ``khq_step`` (``mode="classic"``, the
               call order of the reference host), for every attention layer of every token.
* ``serve``    many sequences generate one token each: ``BatchEngine.decode_step`` from and to pinned host buffers.
* ``prompt``   a new prompt of one sequence: ``KhqRuntime.khq_prefill`` (attention of all rows, compression of the
               full chunks, the newest tokens into the rings) for every layer.
* ``attention``  causal attention of a batch of prompts, fp16 or bf16: ``CudaOps.gqa_prefill``.
* ``compress`` rows of K and V into KHQ code words: ``CudaOps.compress``, K then V.

Values follow ``synth.py``: log-normal channel scales with four x8 outlier channels per kv-head, N(0,1) queries and gate
logits, tables fitted to a sample; the K rotor is the identity, which is what a calibration file carries, or random
(``rotor``).  A pass leaves the state where the next one finds it: positions are set back to where the case starts, and
the slots that a pass writes are not read before it has written them.
"""
import math

import numpy as np
import torch

from bonsai_mojo_1bit_optimization_t4_cuda_b200 import synth
from bonsai_mojo_1bit_optimization_t4_cuda_b200.engine import BatchEngine
from bonsai_mojo_1bit_optimization_t4_cuda_b200.ops import CudaOps
from bonsai_mojo_1bit_optimization_t4_cuda_b200.runtime import KhqRuntime

H_Q, H_KV, D = 24, 4, 256
KV = H_KV * D
CHUNK, RING = 128, 256
SCALE = 1.0 / 16.0
RINGS = ("ring_k", "ring_v", "ring_u")
CODES = ("kmask", "kpay", "knorm", "krn", "vpay", "vnorm", "vrn", "vsm")
ROW_BYTES = 220                       # code words of one (token, kv-head)
TABLE_BYTES = 2 * (2 * (D + 4 * D + 1024) + 64 * 256 * 3)


def listed():
    return [
        # one decode step of a short conversation through all 16 attention layers: launches and latency
        dict(name="token_short", kind="token", mode="fused", layers=16, tokens=1, c_len=384, win=128, rotor="identity"),
        # the same through the pre-step and the drop-in launches, some thousand tokens in
        dict(name="token_dropin", kind="token", mode="prestep", layers=16, tokens=1, c_len=2176, win=201, rotor="identity"),
        # sixteen tokens, the last of which fills the raw window and compresses its oldest half
        dict(name="token_event", kind="token", mode="fused", layers=4, tokens=16, c_len=4096, win=240, rotor="random"),
        # one very long sequence, one layer
        dict(name="token_long", kind="token", mode="fused", layers=1, tokens=1, c_len=131072, win=190, rotor="identity"),
        # a server with next to no load: three sequences of ragged length, every layer
        dict(name="serve_few", kind="serve", layers=16, seqs=3, lo=200, hi=3000, norms=0, rotor="identity"),
        # a server with some load
        dict(name="serve_some", kind="serve", layers=16, seqs=32, lo=1024, hi=16384, norms=1, rotor="random"),
        # a full server: 256 sequences of 4k to 32k tokens (two of the layers)
        dict(name="serve_full", kind="serve", layers=2, seqs=256, lo=4096, hi=32768, norms=1, rotor="identity"),
        # a prompt of one sentence through all layers
        dict(name="prompt_short", kind="prompt", layers=16, tokens=57, rotor="identity"),
        # a document as prompt, odd length
        dict(name="prompt_long", kind="prompt", layers=2, tokens=6001, rotor="random"),
        # a batch of full prompts
        dict(name="attention_fp16", kind="attention", dtype="fp16", batch=4, tokens=8192),
        # a batch of ragged middling prompts in bf16
        dict(name="attention_bf16", kind="attention", dtype="bf16", batch=9, tokens=1531),
        # the code words of a batch of long prompts (all chunks but the last)
        dict(name="compress_bulk", kind="compress", rows=129024, rotor="identity"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "token", "token", "serve", "serve", "serve", "prompt", "attention", "compress"])
    rotor = rng.choice(["identity", "identity", "random"])
    if kind == "token":
        c_len = CHUNK * _log_int(rng, 1, 1024)
        tokens = rng.choice([1, 1, rng.randint(2, 16)])
        layers = max(1, min(_log_int(rng, 1, 16), (1 << 18) // (c_len * tokens)))
        win = rng.randint(CHUNK, RING - tokens - (layers > 5))  # a compression event only where its code words are returned
        return dict(kind=kind, mode=rng.choice(["fused", "fused", "prestep", "classic"]), layers=layers, tokens=tokens,
                    c_len=c_len, win=win, rotor=rotor)
    if kind == "serve":
        seqs = _log_int(rng, 1, 256)
        lo = _log_int(rng, 128, 8192)
        hi = lo + _log_int(rng, 64, 24576)
        layers = max(1, min(_log_int(rng, 1, 16), 2 * 256 * 18432 // (seqs * (lo + hi) // 2)))
        return dict(kind=kind, layers=layers, seqs=seqs, lo=lo, hi=hi, norms=rng.randint(0, 1), rotor=rotor)
    if kind == "prompt":
        tokens = _log_int(rng, 8, 12000)
        return dict(kind=kind, layers=max(1, min(_log_int(rng, 1, 16 if tokens < RING else 5), 16000 // tokens)), tokens=tokens, rotor=rotor)
    if kind == "attention":
        tokens = _log_int(rng, 16, 16384)
        batch = max(1, min(_log_int(rng, 1, 32), 4 * 8192 * 8192 // (tokens * tokens), 65536 // tokens))
        return dict(kind=kind, dtype=rng.choice(["fp16", "bf16"]), batch=batch, tokens=tokens)
    return dict(kind="compress", rows=4 * _log_int(rng, 1, 32256), rotor=rotor)


# ------------------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _scales(g):
    """Channel scales of K and V, (2, 4, 256)."""
    s = torch.exp(0.5 * torch.randn(2, H_KV, D, generator=g, device="cuda"))
    hot = torch.rand(2, H_KV, D, generator=g, device="cuda").topk(4, dim=-1).indices
    return s.scatter(-1, hot, 8.0 * s.gather(-1, hot))


def _rows(g, scales, n):
    """n tokens of K or V, fp16 (n, 4, 256)."""
    return (torch.randn(n, H_KV, D, generator=g, device="cuda") * scales).half()


def _rope(x, pos):
    """Half-split rotation of dims 0..63 of x (tokens, heads, d) at positions pos (tokens,)."""
    f = torch.exp(torch.arange(32, device=x.device) * (-2.0 / 64.0) * math.log(synth.ROPE_THETA))
    a = pos.to(torch.float32)[:, None, None] * f
    c, s = torch.cos(a), torch.sin(a)
    y = x.float()
    lo, hi = y[..., :32].clone(), y[..., 32:64].clone()
    y[..., :32], y[..., 32:64] = lo * c - hi * s, lo * s + hi * c
    return y.to(x.dtype)


def _tables(seed, layers, rotor):
    out = []
    for layer in range(layers):
        rng = np.random.default_rng([int(seed), layer])
        k, v = synth.make_kv(rng, 64)
        out.append(synth.make_tables(rng, layer, k.reshape(-1, D), v.reshape(-1, D), vq_scale=1.0 / 16.0,
                                     k_rotor_identity=rotor == "identity"))
    return out


def _runtime(case, seed, cap):
    rt = KhqRuntime(CudaOps())
    rt.khq_activate(_tables(seed, case["layers"], case["rotor"]), cap)
    for layer in range(case["layers"]):
        rt.khq_init_layer(layer, H_Q, H_KV, D)
    return rt


def _compress(ops, t, k, v, row0=0):
    """K and V rows into a runtime layer's arrays (or any dict with the same names)."""
    n = k.numel() // D
    ops.compress(k, t["dk"], t["rk"], t["ck"], t["ck"], t["kmask"][row0 * 16:], t["knorm"][row0:], t["krn"][row0:],
                 t["kpay"][row0 * 40:], t["vsm"][row0 * 4:], n, D, t["ts_k"], t["alpha_k"], False)
    ops.compress(v, t["dv"], t["rv"], t["cv"], t["vq"], t["kmask"][row0 * 16:], t["vnorm"][row0:], t["vrn"][row0:],
                 t["vpay"][row0 * 104:], t["vsm"][row0 * 4:], n, D, t["ts_v"], t["alpha_v"], True)


def _prepare_token(case, seed):
    layers, tokens, c_len, win = case["layers"], case["tokens"], case["c_len"], case["win"]
    g = _gen(seed)
    rt = _runtime(case, seed, c_len + 2 * CHUNK)
    pos = torch.arange(c_len, c_len + win + tokens, device="cuda")
    new = {n: [] for n in ("q", "u", "k", "v")}
    for layer in range(layers):
        L = rt.layers[layer]
        sc = _scales(g)
        for t0 in range(0, c_len, 16384):
            m = min(16384, c_len - t0)
            _compress(rt.ops, dict(L.t, ts_k=L.ts_k, alpha_k=L.alpha_k, ts_v=L.ts_v, alpha_v=L.alpha_v), _rows(g, sc[0], m),
                      _rows(g, sc[1], m), t0 * H_KV)
        u, v = _rows(g, sc[0], win + tokens), _rows(g, sc[1], win + tokens)
        k = _rope(u, pos)
        slots = pos[:win] % RING
        for ring, src in (("ring_u", u), ("ring_k", k), ("ring_v", v)):
            L.t[ring].view(RING, KV)[slots] = src[:win].reshape(win, KV)
        q = torch.randn(tokens, H_Q, 2 * D, generator=g, device="cuda").half()
        if case["mode"] != "prestep":
            q[..., :D] = _rope(q[..., :D].contiguous(), pos[win:])
        for n, x in (("q", q), ("u", u[win:]), ("k", k[win:]), ("v", v[win:])):
            new[n].append(x.reshape(tokens, -1).clone())
    # (tokens, layers, ...): a token's projections of all layers
    new = {n: torch.stack(x, 1).contiguous() for n, x in new.items()}
    out = torch.empty(tokens, layers, H_Q * D, dtype=torch.float16, device="cuda")
    # the pre-step works in place: the buffers that a model's projections land in
    q_now, u_now = torch.empty_like(new["q"][0]), torch.empty_like(new["u"][0])
    split = lambda x: [list(r) for r in x]  # noqa: E731  views per token and layer, as a program's layers hold them
    return dict(case=case, rt=rt, new=new, views={n: split(x) for n, x in new.items()}, out=out, outs=split(out),
                q_now=q_now, u_now=u_now, q_nows=list(q_now), u_nows=list(u_now),
                norm=torch.exp(0.1 * torch.randn(2, layers, D, generator=g, device="cuda")))


def _run_token(s):
    case, rt, view = s["case"], s["rt"], s["views"]
    layers, start = case["layers"], case["c_len"] + case["win"]
    del rt.events[:]
    for L in rt.layers[:layers]:
        L.boundary, L.write_pos = case["c_len"], start
    for t in range(case["tokens"]):
        q, u, k, v, out = view["q"][t], view["u"][t], view["k"][t], view["v"][t], s["outs"][t]
        if case["mode"] == "fused":
            for i in range(layers):
                rt.khq_step_fused(i, q[i], u[i], k[i], v[i], out[i], SCALE)
        elif case["mode"] == "classic":
            for i in range(layers):
                rt.khq_capture_unroped(i, u[i])
                rt.khq_step(i, q[i], k[i], v[i], out[i], SCALE)
        else:
            s["q_now"].copy_(s["new"]["q"][t])
            s["u_now"].copy_(s["new"]["u"][t])
            for i in range(layers):
                rt.khq_prestep(i, s["q_nows"][i], s["u_nows"][i], v[i], start + t, s["norm"][0, i], s["norm"][1, i])
                rt.khq_step(i, s["q_nows"][i], s["u_nows"][i], v[i], out[i], SCALE, rings_written=True)
    event = case["win"] + case["tokens"] >= RING
    return [s["out"]] + [[L.t[n] for n in RINGS + (CODES if event else ())] for L in rt.layers[:layers]]


def _prepare_serve(case, seed):
    layers, B = case["layers"], case["seqs"]
    rng = np.random.default_rng([B, case["lo"], case["hi"]])  # the lengths belong to the case, the values to the seed
    ctx = rng.integers(case["lo"], case["hi"] + 1, B)
    # the state machine compresses when the window reaches 256: some sequences do in this step, where their code words are
    # among the outputs (up to five layers)
    win = rng.integers(CHUNK, RING - (layers > 5), B)
    c_len = np.maximum(ctx - win, 0) // CHUNK * CHUNK
    norms = None
    if case["norms"]:
        norms = [tuple(np.exp(0.1 * rng.standard_normal((2, D))).astype(np.float32)) for _ in range(layers)]
    eng = BatchEngine(_tables(seed, layers, case["rotor"]), c_len, win, grow_tokens=CHUNK, norm_weights=norms)
    eng.fill_synthetic(int(seed))
    g = _gen(seed + 1)
    for h in (eng.h_q, eng.h_k, eng.h_v):
        h.copy_(torch.randn(h.shape, generator=g, device="cuda").half())
    return dict(case=case, eng=eng, boundary=eng.boundary.copy(), write_pos=eng.write_pos.copy())


def _run_serve(s):
    eng = s["eng"]
    eng.boundary[:] = s["boundary"]
    eng.write_pos[:] = s["write_pos"]
    out = eng.decode_step(SCALE)
    return [out, eng.ring_k, eng.ring_v, eng.ring_u, eng.pay if eng.L <= 5 else None]


def _prepare_prompt(case, seed):
    layers, T = case["layers"], case["tokens"]
    g = _gen(seed)
    rt = _runtime(case, seed, (T + CHUNK) // CHUNK * CHUNK)
    pos = torch.arange(T, device="cuda")
    inputs = []
    for _ in range(layers):
        sc = _scales(g)
        u, v = _rows(g, sc[0], T), _rows(g, sc[1], T)
        q = torch.randn(T, H_Q, 2 * D, generator=g, device="cuda").half()
        q[..., :D] = _rope(q[..., :D].contiguous(), pos)
        inputs.append((q, u, _rope(u, pos), v, torch.empty(T, H_Q, D, dtype=torch.float16, device="cuda")))
    return dict(case=case, rt=rt, inputs=inputs)


def _run_prompt(s):
    rt, got = s["rt"], []
    del rt.events[:]
    for i, (q, u, k, v, out) in enumerate(s["inputs"]):
        L = rt.layers[i]
        L.boundary = L.write_pos = 0  # a new sequence
        rt.khq_prefill(i, q, u, k, v, out, SCALE)
        got.append([out] + [L.t[n] for n in RINGS + (CODES if L.boundary else ())])
    return got


def _prepare_attention(case, seed):
    B, T = case["batch"], case["tokens"]
    g = _gen(seed)
    dt = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
    pos = torch.arange(T, device="cuda").repeat(B)
    sc = _scales(g)
    u, v = _rows(g, sc[0], B * T), _rows(g, sc[1], B * T)
    q = torch.randn(B * T, H_Q, 2 * D, generator=g, device="cuda").to(dt)
    q[..., :D] = _rope(q[..., :D].contiguous(), pos)
    return dict(case=case, ops=CudaOps(), q=q.view(B, T, H_Q, 2 * D), k=_rope(u, pos).to(dt).view(B, T, H_KV, D),
                v=v.to(dt).view(B, T, H_KV, D), out=torch.empty(B, T, H_Q, D, dtype=dt, device="cuda"))


def _run_attention(s):
    s["ops"].gqa_prefill(s["q"], s["k"], s["v"], s["out"], s["case"]["batch"], s["case"]["tokens"], H_Q, H_KV, D, SCALE)
    return s["out"]


def _prepare_compress(case, seed):
    n = case["rows"]
    g = _gen(seed)
    tb = _tables(seed, 1, case["rotor"])[0]
    f = tb.as_f16()
    t = {a: torch.from_numpy(f[b]).cuda() for a, b in (("dk", "d_k"), ("ck", "cents_k"), ("rk", "rotor_k"), ("dv", "d_v"),
                                                         ("cv", "cents_v"), ("rv", "rotor_v"), ("vq", "vq"))}
    t.update(ts_k=tb.ts_k, alpha_k=tb.alpha_k, ts_v=tb.ts_v, alpha_v=tb.alpha_v)
    for name, per_row, dt in (("kmask", 16, torch.int32), ("kpay", 40, torch.uint8), ("knorm", 1, torch.float16),
                              ("krn", 1, torch.float16), ("vpay", 104, torch.uint8), ("vnorm", 1, torch.float16),
                              ("vrn", 1, torch.float16), ("vsm", 4, torch.uint8)):
        t[name] = torch.zeros(n * per_row, dtype=dt, device="cuda")
    sc = _scales(g)
    return dict(case=case, ops=CudaOps(), t=t, k=_rows(g, sc[0], n // H_KV), v=_rows(g, sc[1], n // H_KV))


def _run_compress(s):
    _compress(s["ops"], s["t"], s["k"], s["v"])
    return [s["t"][n] for n in CODES]


_PREPARE = dict(token=_prepare_token, serve=_prepare_serve, prompt=_prepare_prompt, attention=_prepare_attention,
                compress=_prepare_compress)
_RUN = dict(token=_run_token, serve=_run_serve, prompt=_run_prompt, attention=_run_attention, compress=_run_compress)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["case"]["kind"]](state)


# ------------------------------------------------------------------------------------------------------- costs
def _step_bytes(c_len, win):
    """One layer of one token: the two regions, the query and gate, the output, the new rows in and into three rings."""
    return H_KV * (ROW_BYTES * c_len + 4 * D * win) + 2 * (2 * H_Q * D + H_Q * D) + 6 * 2 * KV


def _compress_bytes(rows):
    return rows * (2 * 2 * D + ROW_BYTES)


def work(case):
    """Bytes read and written once, and the multiply-adds (two operations) of the attention products alone."""
    kind, layers = case["kind"], case.get("layers", 1)
    if kind == "token":
        c, w, n = case["c_len"], case["win"], case["tokens"]
        event = w + n >= RING
        nbytes = sum(_step_bytes(c, w + t + 1) for t in range(n)) + (_compress_bytes(CHUNK * H_KV) if event else 0)
        flops = sum(4 * H_Q * D * (c + w + t + 1) for t in range(n))
        return dict(bytes=layers * (nbytes + TABLE_BYTES), flops=layers * flops)
    if kind == "serve":
        w = (CHUNK + RING) // 2
        ctx = (case["lo"] + case["hi"]) / 2
        c = max(ctx - w - CHUNK / 2, 0)
        return dict(bytes=layers * (case["seqs"] * _step_bytes(c, w) + TABLE_BYTES), flops=layers * case["seqs"] * 4 * H_Q * D * (c + w))
    if kind == "prompt":
        T = case["tokens"]
        rows = max(T // CHUNK - 1, 0) * CHUNK * H_KV
        nbytes = T * 2 * (3 * H_Q * D + 2 * KV) + 12 * KV * min(T, RING) + _compress_bytes(rows) + TABLE_BYTES
        return dict(bytes=layers * nbytes, flops=layers * 2 * H_Q * D * T * (T + 1))
    if kind == "attention":
        T, B = case["tokens"], case["batch"]
        return dict(bytes=B * T * 2 * (3 * H_Q * D + 2 * KV), flops=B * 2 * H_Q * D * T * (T + 1))
    # the search of 256 codes of three dims in each of 64 patches: three subtractions and three multiply-adds a code
    return dict(bytes=_compress_bytes(case["rows"]) + TABLE_BYTES, flops=case["rows"] * 64 * 256 * 9)


def tolerance(case):
    """Code words and the rings are the same bit by bit; attention outputs are rounded to fp16 or bf16 at the end, their
    operands in between carry no less than that."""
    if case["kind"] == "compress":
        return "exact"
    if case.get("dtype") == "bf16":
        return dict(rel=1e-2, max=0.1)
    return dict(rel=2e-3, max=0.03)
