"""One decode step as one kernel (launch_khq_layer_token) against the three launches of the call-by-call sequence, at the edges of its
shapes: block and cluster remainders, the switches between its kernels, unaligned arrays, rows with any number of outliers."""
import ctypes

import numpy as np
import pytest

from bonsai_mojo_1bit_optimization_t4_cuda_b200 import synth

pytestmark = pytest.mark.gpu
D, HKV, HQ, RING, SCALE = 256, 4, 24, 256, 1.0 / 16.0
CODES = (("kmask", 64), ("kpay", 40), ("knorm", 2), ("krn", 2), ("vpay", 104), ("vnorm", 2), ("vrn", 2), ("vsm", 4))
MAX_TOKENS = 17000


@pytest.fixture(scope="module")
def state(cuda_ops):
    """A layer of a runtime and MAX_TOKENS tokens of code words drawn at random: 25 % outlier symbols, more than a row may keep."""
    import torch

    from bonsai_mojo_1bit_optimization_t4_cuda_b200.runtime import KhqRuntime

    rng = np.random.default_rng(3)
    k, v = synth.make_kv(rng, 64)
    tb = synth.make_tables(rng, 0, k.reshape(-1, D), v.reshape(-1, D), vq_scale=1.0 / 16.0)
    g = torch.Generator(device="cuda").manual_seed(4)
    rows = MAX_TOKENS * HKV
    raw = {n: torch.randint(0, 256, (rows * b,), dtype=torch.uint8, device="cuda", generator=g) for n, b in CODES}
    sparse = torch.randint(0, 256, (rows * 64,), dtype=torch.uint8, device="cuda", generator=g)  # every other row: an outlier in 16
    odd = (torch.arange(rows * 64, device="cuda") // 64) % 2 == 1
    pair = raw["kmask"] & (raw["kmask"] >> 1) & 0x55
    keep = sparse & (sparse >> 1) & 0x55
    raw["kmask"] = torch.where(odd, raw["kmask"] & ~(pair & ~keep), raw["kmask"])
    raw["kpay"].view(rows, 40)[:, :4] = torch.tensor([0xE8, 3, 0, 0], dtype=torch.uint8, device="cuda")  # multiplier 1
    u = lambda: torch.rand(rows, generator=g, device="cuda")
    for n, lo, hi in (("knorm", 0.5, 4.0), ("krn", 0.01, 0.05), ("vnorm", 0.5, 4.0), ("vrn", 0.8, 1.2)):
        raw[n] = (lo + (hi - lo) * u()).half().view(torch.uint8)
    raw["vsm"] = (0.05 * u()).view(torch.uint8)

    def layer(shift):
        rt = KhqRuntime(cuda_ops)
        rt.khq_activate([tb], MAX_TOKENS)
        rt.khq_init_layer(0, HQ, HKV, D)
        L = rt.layers[0]
        for n, b in CODES:
            buf = torch.empty(rows * b + 16, dtype=torch.uint8, device="cuda")
            buf[shift:shift + rows * b] = raw[n]
            L.t[n] = buf[shift:shift + rows * b]
        for i, n in enumerate(("ring_k", "ring_v", "ring_u")):
            L.t[n].copy_(torch.randn(L.t[n].numel(), generator=torch.Generator(device="cuda").manual_seed(i), device="cuda"))
        return L, cuda_ops.layer_ctx(L, RING, 1e7)

    new = [torch.randn(HKV * D, generator=g, device="cuda").half() for _ in range(3)]
    q = torch.randn(HQ * 2 * D, generator=g, device="cuda").half()
    return dict(plain=layer(0), shifted=layer(4), new=new, q=q)


def _separate(ops, L, q, c_len, win_len):
    import torch

    T = {n: L.t[n] for n in L.t}
    z = lambda n, dt=torch.float32: torch.zeros(n, dtype=dt, device="cuda")
    ac, aw, ap, out = z(HQ * 258), z(HQ * 258), z(HQ * 32 * 258), z(HQ * D, torch.float16)
    if c_len:
        ops.attn(q, T["kpay"], T["vpay"], T["vsm"], T["kmask"], T["knorm"], T["krn"], T["vnorm"], T["vrn"], T["ck"], T["cv"], T["vq"], T["rk"],
                 T["rv"], T["dk"], T["dv"], ac, ap, HQ, HQ, 1, c_len, c_len, 6, SCALE, L.alpha_k, L.alpha_v, 1e7, 0, 8)
    ops.window_attn(q, T["ring_k"], T["ring_v"], aw, c_len % RING, win_len, RING, HQ, HKV, D, SCALE)
    ops.merge_gate(ac, aw, q, out, HQ, D, True, c_len > 0)
    return out


@pytest.mark.parametrize("arrays", ["plain", "shifted"])
@pytest.mark.parametrize("c_len", [0, 1, 15, 16, 17, 126, 128, 129, 385, 1777, 1792, 1793, 2176, 5376, 5377, 16384, 16385, 16999])
def test_step_matches_the_separate_launches(cuda_ops, state, arrays, c_len):
    import torch

    L, ctx = state[arrays]
    k, v, u = state["new"]
    q = state["q"]
    for win_len in (1, 16, 17, 129, 255, 256) if arrays == "plain" else (130,):
        slot = (c_len + win_len - 1) % RING
        rings = {n: L.t[n].clone() for n in ("ring_k", "ring_v", "ring_u")}
        out = [torch.empty(HQ * D, dtype=torch.float16, device="cuda") for _ in range(2)]
        for o in out:
            cuda_ops.layer_step(ctx, q, k, v, u, o, c_len, win_len, False, 1, SCALE)
        for n, x in (("ring_k", k), ("ring_v", v), ("ring_u", u)):
            rings[n].view(RING, -1)[slot] = x
            assert torch.equal(rings[n], L.t[n]), n  # the token, and nothing else
        want = _separate(cuda_ops, L, q, c_len, win_len).float()
        torch.cuda.synchronize()
        assert cuda_ops.lib.khq_b200_device_status() == 0
        assert torch.equal(out[0], out[1]) and int(ctx[3].abs().sum()) == 0
        # both sides: fp32 sums in another order (some 1e-6 of the largest term), then one rounding to fp16
        err = (out[0].float() - want).abs()
        assert bool((err <= 2.0 ** -10 * want.abs() + 3e-4 * want.abs().max()).all()), (c_len, win_len, float(err.max()), float(want.abs().max()))


def test_rows_that_are_in_the_rings(cuda_ops, state):
    """Without new rows a step reads the token from the rings and leaves them alone."""
    import torch

    L, ctx = state["plain"]
    for c_len in (256, 4096):
        out, again = (torch.empty(HQ * D, dtype=torch.float16, device="cuda") for _ in range(2))
        cuda_ops.layer_step(ctx, state["q"], *state["new"], out, c_len, 140, False, 1, SCALE)
        rings = [L.t[n].clone() for n in ("ring_k", "ring_v", "ring_u")]
        cuda_ops.layer_step(ctx, state["q"], None, None, None, again, c_len, 140, False, 1, SCALE)
        assert torch.equal(out, again) and all(torch.equal(a, L.t[n]) for a, n in zip(rings, ("ring_k", "ring_v", "ring_u")))


def test_refused(cuda_ops, state):
    """Argument errors are codes, before anything is launched."""
    L, ctx = state["plain"]
    f = cuda_ops.lib.launch_khq_layer_token
    q, out, c = state["q"].data_ptr(), state["q"].data_ptr(), ctx[4]
    stream = 0
    assert f(ctx[1], c, 0, 0, 0, 0, out, 128, 10, 0, SCALE, stream) == -100
    assert f(ctx[1], 0, q, 0, 0, 0, out, 128, 10, 0, SCALE, stream) == -100
    assert f(ctx[1], c, q, 0, 0, 0, out, 128, 0, 0, SCALE, stream) == -100
    assert f(ctx[1], c, q, 0, 0, 0, out, 128, 257, 0, SCALE, stream) == -103
    assert f(ctx[1], c, q + 2, 0, 0, 0, out, 128, 10, 0, SCALE, stream) == -104
    bare = type(ctx[0])()
    ctypes.memmove(ctypes.addressof(bare), ctx[1], ctypes.sizeof(bare))
    bare.prepared = None
    assert f(ctypes.addressof(bare), c, q, 0, 0, 0, out, 128, 10, 0, SCALE, stream) == -100


@pytest.mark.parametrize("v_scale,gap", [(1.0, 0.0), (200.0, 14.3), (2000.0, 19.1), (30000.0, 24.0)])
@pytest.mark.parametrize("win_len", [17, 200, 256])
def test_window_with_one_dominant_token(cuda_ops, state, win_len, v_scale, gap):
    """The raw window against 64 bits, its first token with all but e^-gap of each other token's weight and V = 0, as the first token of a
    conversation has it: the output is the others' sum, so their small weights have to be as exact as large ones."""
    import torch

    L, ctx = state["plain"]
    g = torch.Generator(device="cuda").manual_seed(11)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    q, k, v = rnd(HQ, 2 * D), rnd(win_len, HKV, D), v_scale * rnd(win_len, HKV, D).clamp(-2.0, 2.0)
    q[:, D:] = 20.0  # open gates
    q[:, 255], k[:, :, 255] = 16.0, 0.0
    if gap:
        k[0], v[0] = 0.0, 0.0
        k[0, :, 255] = gap
    q, k, v = q.half(), k.half(), v.half()
    for ring, rows in (("ring_k", k), ("ring_v", v)):
        L.t[ring].view(RING, HKV, D)[:win_len] = rows
    out = torch.empty(HQ * D, dtype=torch.float16, device="cuda")
    cuda_ops.layer_step(ctx, q.reshape(-1), k[-1].reshape(-1), v[-1].reshape(-1), None, out, 0, win_len, False, 1, SCALE)
    qd, kd, vd = q[:, :D].double().view(HKV, 6, D), k.double(), v.double()
    w = torch.softmax(SCALE * torch.einsum("jhd,sjd->jhs", qd, kd), dim=-1)
    gate = torch.sigmoid(q[:, D:].double())
    want = torch.einsum("jhs,sjd->jhd", w, vd).reshape(HQ, D) * gate
    terms = torch.einsum("jhs,sjd->jhd", w, vd.abs()).reshape(HQ, D) * gate
    err = (out.view(HQ, D).double() - want).abs()
    # the output's own rounding, and scores of up to 32 (4e-6) and their exponentials in fp32
    assert cuda_ops.lib.khq_b200_device_status() == 0
    assert bool((err <= 2.0 ** -11 * want.abs() + 2.0 ** -25 + 1e-5 * terms).all()), (float((err / terms).max()), float(err.norm() / want.norm()))
    print(f"win {win_len} gap {gap}: {float(err.norm() / want.norm()):.2e}")


@pytest.mark.parametrize("c_len", [1792, 1793, 16999])
def test_the_last_warp_merges_every_record(cuda_ops, state, c_len):
    """A head's records are merged in their own order by whichever warp arrives last: the same bits in each of many steps back to back
    (15 records of khq_step_kernel, 9 and 31 of khq_step_wide_kernel), and the counters are left at zero."""
    import torch

    L, ctx = state["plain"]
    k, v, u = state["new"]
    outs = torch.empty(400, HQ * D, dtype=torch.float16, device="cuda")
    for o in outs:
        cuda_ops.layer_step(ctx, state["q"], k, v, u, o, c_len, 130, False, 1, SCALE)
    assert bool((outs == outs[0]).all()) and int(ctx[3].abs().sum()) == 0
    assert cuda_ops.lib.khq_b200_device_status() == 0


@pytest.mark.parametrize("c_len,splits", [(0, 1), (1, 1), (129, 8), (385, 32), (1793, 16), (5377, 33)])
def test_two_kernel_step_matches_the_separate_launches(cuda_ops, state, c_len, splits):
    """launch_khq_layer_step, the step as an attention launch and a tail (up to 32 splits: the tail merges their records)."""
    import torch

    L, ctx = state["plain"]
    k, v, u = state["new"]
    q, out = state["q"], torch.empty(HQ * D, dtype=torch.float16, device="cuda")
    c = type(ctx[0])()
    ctypes.memmove(ctypes.addressof(c), ctx[1], ctypes.sizeof(c))
    partial = torch.empty(HQ * splits * 258, dtype=torch.float32, device="cuda")
    c.attn_partial = partial.data_ptr()
    f = cuda_ops.lib.launch_khq_layer_step
    stream = torch.cuda.current_stream().cuda_stream
    for win_len in (17, 256):
        rows = [t.data_ptr() for t in (k, v, u)]
        assert f(ctypes.addressof(c), q.data_ptr(), *rows, out.data_ptr(), c_len, win_len, 0, splits, SCALE, stream) == 0
        slot = (c_len + win_len - 1) % RING
        assert all(torch.equal(L.t[n].view(RING, -1)[slot], x) for n, x in (("ring_k", k), ("ring_v", v), ("ring_u", u)))
        want = _separate(cuda_ops, L, q, c_len, win_len).float()
        again = torch.empty_like(out)  # the token is in the rings now
        assert f(ctypes.addressof(c), q.data_ptr(), 0, 0, 0, again.data_ptr(), c_len, win_len, 0, splits, SCALE, stream) == 0
        torch.cuda.synchronize()
        assert cuda_ops.lib.khq_b200_device_status() == 0 and torch.equal(out, again)
        err = (out.float() - want).abs()  # as above
        assert bool((err <= 2.0 ** -10 * want.abs() + 3e-4 * want.abs().max()).all()), (c_len, win_len, float(err.max()), float(want.abs().max()))
    assert f(ctypes.addressof(c), q.data_ptr(), 0, 0, 0, out.data_ptr(), c_len, 257, 0, splits, SCALE, stream) == -103
    assert f(ctypes.addressof(c), q.data_ptr(), rows[0], 0, 0, out.data_ptr(), c_len, 17, 0, splits, SCALE, stream) == -100
