"""Rounding of the compressed-region attention over long contexts, per rotated dim, against 64-bit sums of the same code words.

With a zero query every token has the same weight, so the wanted sums are plain sums over the tokens of what the payload
encodes: they can be had in 64 bits, and they are as long as sums over a context get.  Dims 0..2 of a patch come from the
codebook, dim 3 from a centroid bit and a residual field; the signed terms cancel, so a sum's error has to be seen against the
spread of the sums and not against the number of tokens."""
import numpy as np
import pytest

from bonsai_mojo_1bit_optimization_t4_cuda_b200 import synth

pytestmark = pytest.mark.gpu
D, HKV, HQ, NP = 256, 4, 24, 64


@pytest.fixture(scope="module", params=["centroids +-c", "centroids c/8 +-c"])
def context(cuda_ops, request):
    """131 072 tokens of compressed synthetic rows with their tables, and the 64-bit sums of the pieces [lo, hi)."""
    import torch

    n = 131072
    rng = np.random.default_rng(5)
    k, v = synth.make_kv(rng, 512)
    tb = synth.make_tables(rng, 3, k.reshape(-1, D), v.reshape(-1, D), vq_scale=1.0 / 16.0)
    f = {a: torch.from_numpy(b).cuda() for a, b in tb.as_f16().items()}
    f["cents_v"] = f["cents_v"].view(4, D)
    g = torch.Generator(device="cuda").manual_seed(11)
    rows = n * HKV
    t = dict(k_mask=torch.zeros(rows * 16, dtype=torch.int32, device="cuda"), k_payload=torch.zeros(rows * 40, dtype=torch.uint8, device="cuda"),
             v_payload=torch.zeros(rows * 104, dtype=torch.uint8, device="cuda"), v_shared_meta=torch.zeros(rows * 4, dtype=torch.uint8, device="cuda"))
    for a in ("k_norms", "k_r_norms", "v_norms", "v_r_norms"):
        t[a] = torch.zeros(rows, dtype=torch.float16, device="cuda")
    sc = torch.exp(0.5 * torch.randn(2, HKV, D, generator=g, device="cuda"))
    x = [(torch.randn(n, HKV, D, generator=g, device="cuda") * s).half() for s in sc]
    cuda_ops.compress(x[0], f["d_k"], f["rotor_k"], f["cents_k"], f["cents_k"], t["k_mask"], t["k_norms"], t["k_r_norms"], t["k_payload"],
                      t["v_shared_meta"], rows, D, tb.ts_k, tb.alpha_k, False)
    cuda_ops.compress(x[1], f["d_v"], f["rotor_v"], f["cents_v"], f["vq"], t["k_mask"], t["v_norms"], t["v_r_norms"], t["v_payload"],
                      t["v_shared_meta"], rows, D, tb.ts_v, tb.alpha_v, True)
    if "c/8" in request.param:  # the centroids' mean is not zero (only what the payload stands for changes, not the bits)
        f["cents_v"][:2] += f["cents_v"][1] / 8
    # the rotated rows that the payload encodes, in 64 bits: 12-bit fields (code bits 0..6, centroid bit, residual), high code bits
    pay = t["v_payload"].view(rows, 104).to(torch.int32)
    b = pay[:, :96].view(rows, NP // 2, 3)
    f24 = b[..., 0] | (b[..., 1] << 8) | (b[..., 2] << 16)
    fields = torch.stack([f24 & 0xFFF, f24 >> 12], -1).view(rows, NP)
    high = ((pay[:, 96:, None] >> torch.arange(8, device="cuda", dtype=torch.int32)) & 1).reshape(rows, NP)
    code = ((fields & 0x7F) | (high << 7)).long()
    vn, en = t["v_norms"].double(), t["v_r_norms"].double()
    sm = t["v_shared_meta"].view(torch.float32).double()
    cents = f["cents_v"].double()[:2].view(2, NP, 4)[..., 3]
    dims = torch.empty(rows, NP, 4, dtype=torch.float64, device="cuda")
    vq = f["vq"].double().view(NP, 256, 3)
    for p in range(NP):
        dims[:, p, :3] = vq[p][code[:, p]] * (vn * en)[:, None] * tb.alpha_v
        bit = (fields[:, p] >> 7) & 1
        dims[:, p, 3] = vn * (cents[:, p][bit] * tb.alpha_v + sm / 7.0 * ((fields[:, p] >> 8) - 8))
    sums = lambda lo, hi: dims.view(n, HKV, NP, 4)[lo:hi].sum(0).cpu().numpy()
    return n, tb, f, t, sums


def _rotated(acc, f):
    """Records' accumulators (24, 256) back into the rotated domain (24, 64, 4), in 64 bits."""
    z = acc.astype(np.float64) * 16.0 * f["d_v"].double().cpu().numpy()
    h = 1
    while h < D:
        z = z.reshape(HQ, -1, 2, h)
        z = np.stack([z[:, :, 0] + z[:, :, 1], z[:, :, 0] - z[:, :, 1]], 2).reshape(HQ, D)
        h *= 2
    r = f["rotor_v"].double().cpu().numpy().reshape(NP, 4, 4)  # the transform applies r to the accumulators of a patch
    return np.linalg.solve(r[None], z.reshape(HQ, NP, 4, 1) / 256.0)[..., 0]


def _check(acc, weight, want, f, blocks, what):
    """weight: what the record's accumulators have to be multiplied with to stand for plain sums."""
    got = _rotated(acc * weight, f).reshape(HKV, HQ // HKV, NP, 4)
    err = got - want[:, None]
    spread = want.std(axis=(0, 1))
    rel = {k: (np.sqrt((err[..., s] ** 2).mean()) / spread[s].mean(), np.abs(err[..., s]).max() / spread[s].mean())
           for k, s in (("dims 0..2", slice(0, 3)), ("dim 3", slice(3, 4)))}
    print(what, {k: "rms %.2e max %.2e" % v for k, v in rel.items()})
    # An accumulator takes two products of 16 tokens per block of a warp, each addition rounded towards zero: off by at most one unit
    # in the last place, 2^-23 of what it holds.  That is at most about 2.5 times the spread on the way (a random walk's maximum),
    # for a sum as large as the largest of 256; the pieces' errors add up at the worst.  The root mean square is half of that: the
    # mean loss of an addition is half a unit.
    bound = 2 * blocks * 2.0 ** -23
    for name, (rms, top) in rel.items():
        assert rms < 0.5 * bound + 2e-6 and top < 2.5 * bound + 1e-5, f"{what}, {name}: rms {rms:.2e}, max {top:.2e} of the spread (bound {bound:.1e})"


@pytest.mark.parametrize("tokens", [8192, 131072])
def test_one_split(cuda_ops, context, tokens):
    """launch_khq_attn_fp16 with one split: eight CTAs of three warps a kv-head share the tokens."""
    import torch

    n, tb, f, t, sums = context
    q = torch.zeros(HQ, 2 * D, dtype=torch.float16, device="cuda")
    out = torch.zeros(HQ, D + 2, dtype=torch.float32, device="cuda")
    cuda_ops.attn(q, t["k_payload"], t["v_payload"], t["v_shared_meta"], t["k_mask"], t["k_norms"], t["k_r_norms"], t["v_norms"], t["v_r_norms"],
                  f["cents_k"], f["cents_v"], f["vq"], f["rotor_k"], f["rotor_v"], f["d_k"], f["d_v"], out, None, HQ, HQ, 1, tokens, tokens, 6,
                  1 / 16, tb.alpha_k, tb.alpha_v, 1e7, 0, 1)
    r = out.cpu().numpy()
    weight = np.exp(r[:, D:D + 1].astype(np.float64))
    np.testing.assert_allclose(r[:, D + 1:] * weight, tokens, rtol=1e-6)
    _check(r[:, :D], weight, sums(0, tokens), f, tokens / (8 * 48), f"one split, {tokens} tokens")


def test_long_items(cuda_ops, context):
    """The batched entry's kernel on items of 8192 tokens, whose records are read as they are."""
    import torch

    from bonsai_mojo_1bit_optimization_t4_cuda_b200.batched import BatchedDecode

    n, tb, f, t, sums = context
    c_len = 65536
    q = torch.zeros(HQ, 2 * D, dtype=torch.float16, device="cuda")
    ring = torch.zeros(256, HKV, D, dtype=torch.float16, device="cuda")
    prob = dict(t, q_gate=q, ring_k=ring, ring_v=ring, out=torch.zeros(HQ * D, dtype=torch.float16, device="cuda"), table_id=0, c_len=c_len,
                start_pos=0, win_start=0, win_len=0)
    tab = dict(cents_k=f["cents_k"], cents_v=f["cents_v"], vq=f["vq"], k_rotor=f["rotor_k"], v_rotor=f["rotor_v"], d_k=f["d_k"], d_v=f["d_v"],
               alpha_k=tb.alpha_k, alpha_v=tb.alpha_v)
    bd = BatchedDecode([prob], [tab])
    items = np.zeros(c_len // 8192, bd.host_items.dtype)  # the planner would cut one sequence into pieces for all SMs
    items["lo"] = np.arange(0, c_len, 8192)
    items["hi"] = items["lo"] + 8192
    items["slot"] = np.arange(len(items))
    bd.host_descs["first_slot"], bd.host_descs["n_slots"] = 0, len(items)
    up = lambda a: torch.from_numpy(a.view(np.uint8).reshape(-1).copy()).cuda()
    assert len(items) <= bd.n_items  # the workspace is large enough
    bd.n_items, bd.items, bd.descs = len(items), up(items), up(bd.host_descs)
    bd.launch()
    recs = bd.workspace[256:].view(torch.float32)[:bd.n_items * HQ * (D + 2)].view(bd.n_items, HQ, D + 2).cpu().numpy()
    for w in items:
        r = recs[w["slot"]]
        _check(r[:, :D], np.exp(r[:, D:D + 1].astype(np.float64)), sums(int(w["lo"]), int(w["hi"])), f, 8192 / 48, f"item at {w['lo']}")


@pytest.mark.parametrize("norm", [7000, 20000, 50000])
def test_large_v_rows(cuda_ops, oracle, norm):
    """V rows whose norms approach the end of fp16: the weights' products with them are fp16 operands, whatever the order in which
    the scores come."""
    import torch

    import cases

    c_len = 1200
    case = cases.make_case(31 + norm, c_len, "calib")
    v = case["v"].astype(np.float32)
    v *= norm / np.sqrt((v ** 2).sum(-1, keepdims=True))
    case["v"] = v.astype(np.float16)
    kv = cases.compress_with(oracle.compress, case, c_len)
    tb, f = case["tables"], case["f16"]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    t, tab = {k: dev(a) for k, a in kv.items() if k != "near_ties"}, {k: dev(a) for k, a in f.items()}
    out = torch.zeros(HQ, D + 2, dtype=torch.float32, device="cuda")
    cuda_ops.attn(dev(case["q_gate"]), t["k_payload"], t["v_payload"], t["v_shared_meta"], t["k_mask"], t["k_norms"], t["k_r_norms"], t["v_norms"],
                  t["v_r_norms"], tab["cents_k"], tab["cents_v"], tab["vq"], tab["rotor_k"], tab["rotor_v"], tab["d_k"], tab["d_v"], out, None, HQ, HQ,
                  1, c_len, c_len, 6, 1 / 16, tb.alpha_k, tb.alpha_v, 1e7, 0, 1)
    want = oracle.attn_partial(case["q_gate"], kv, cases.tables_dict(f), HQ, 6, 1 / 16, tb.alpha_k, tb.alpha_v, 1e7, 0, 0, c_len)
    got, want = cases.normalised(out.cpu().numpy()) / norm, cases.normalised(want) / norm
    ok, mx, exc = cases.attention_close(got * 16, want * 16)  # as for rows of norm 16
    assert ok, f"max abs {mx:.3e} excess {exc:.3e}"
