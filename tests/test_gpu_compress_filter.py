"""V code search by launch size (shared by the warps of a block; large launches filtered on the tensor cores, exact where the
filter does not decide): code words bit-identical to the oracle's at the edges of the dispatch and of the row tiles, with tied and
nearly tied codes, with codebooks and rows outside the range of fp16 pieces, with a general alpha, and with codebooks and rows
of any common scale."""
import numpy as np
import pytest

from bonsai_mojo_1bit_optimization_t4_cuda_b200 import synth

pytestmark = pytest.mark.gpu
D = 256


@pytest.mark.parametrize("rows,kind", [(3, "plain"), (1184, "near"), (1185, "ties"), (8484, "plain"), (8485, "plain"), (9472, "ties"),
                                       (9473, "near"), (24641, "wide"), (25000, "odd_rows"), (28417, "ties")])
def test_v_codes_vs_oracle(cuda_ops, oracle, rows, kind):
    rng = np.random.default_rng(rows)
    alpha = 1.0 if kind in ("plain", "ties") else 0.83
    base = min(rows, 4500)  # different rows, repeated: the same row falls on different places of the tiles
    k, v = synth.make_kv(rng, (base + 3) // 4)
    tb = synth.make_tables(rng, 3, k.reshape(-1, D), v.reshape(-1, D), vq_scale=1.0 / 16.0 if kind != "wide" else 1.0).as_f16()
    vq = tb["vq"].reshape(64, 256, 3)
    if kind == "ties":
        vq[:, 128:] = vq[:, :128]  # every code twice
    elif kind == "near":
        vq[:, 1::2] = np.nextafter(vq[:, ::2], np.float16(10))  # pairs one ulp apart
    elif kind == "wide":
        vq[5] *= np.float16(3000)  # beyond the range of fp16 pieces as it stands
    x = v.reshape(-1, D)[:base].copy()
    if kind == "odd_rows":
        x[17] = 0
        x[130] = np.float16(60000)
        x[4400, 7] = np.float16("inf")
    _compare_v(cuda_ops, oracle, x, tb, vq, rows, alpha, kind)


def _compare_v(cuda_ops, oracle, x, tb, vq, rows, alpha, what):
    """The rows of x, repeated to `rows` of them: every output byte of the rows without infinities as the oracle has it."""
    import torch

    base = len(x)
    want = oracle.compress(x, tb["d_v"], tb["rotor_v"], tb["cents_v"], vq.reshape(-1), base, 1.95, alpha, True)
    x = np.resize(x, (rows, D))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    out = dict(norms=torch.zeros(rows, dtype=torch.float16, device="cuda"), r_norms=torch.zeros(rows, dtype=torch.float16, device="cuda"),
               payload=torch.zeros(rows * 104, dtype=torch.uint8, device="cuda"), shared_meta=torch.zeros(rows * 4, dtype=torch.uint8, device="cuda"))
    cuda_ops.compress(dev(x), dev(tb["d_v"]), dev(tb["rotor_v"]), dev(tb["cents_v"]), dev(vq), torch.zeros(rows * 16, dtype=torch.int32, device="cuda"),
                      out["norms"], out["r_norms"], out["payload"], out["shared_meta"], rows, D, 1.95, alpha, True)
    finite = np.isfinite(x.astype(np.float32)).all(axis=1)
    for name, got in out.items():
        g = got.cpu().numpy().view(np.uint8).reshape(rows, -1)
        w = np.ascontiguousarray(want[name]).view(np.uint8).reshape(base, -1)
        w = np.resize(w, (rows, w.shape[1]))
        bad = np.nonzero((g != w).any(axis=1) & finite)[0]
        assert len(bad) == 0, f"{what}: {name} differs in rows {bad[:8]} ({len(bad)} rows)"


@pytest.mark.parametrize("scale,alpha", [(1 / 4, 1.0), (1 / 16, 0.83), (1 / 64, 1.0), (1 / 256, 0.83), (1 / 4096, 1.0), (8.0, 1.0),
                                         (750.0, 1.0), ("patch", 1.0), ("rows", 1.0), (1.0, 1e-13), (1.0, 3e7)])
def test_v_codes_at_any_scale(cuda_ops, oracle, scale, alpha):
    """Codebook, centroids and (through the rotor) projections scaled together, from |a c| of 6e-5 to 180, where the filter's
    operands would leave the range of fp16 pieces; one patch 64 times smaller than the others ("patch"); projections 16 times the
    codebook ("rows"); alphas that put |a c| outside the filter's range (1e-13, 3e7).  8485 rows: the smallest filtered launch."""
    rng = np.random.default_rng(77)
    base = 3000
    k, v = synth.make_kv(rng, base // 4)
    tb = synth.make_tables(rng, 3, k.reshape(-1, D), v.reshape(-1, D), vq_scale=1.0 / 16.0).as_f16()
    vq, rotor, cents = tb["vq"].reshape(64, 256, 3), tb["rotor_v"].reshape(64, 16), tb["cents_v"]
    if scale == "patch":
        vq[5] *= np.float16(1 / 64)
        rotor[5] *= np.float16(1 / 64)
    elif scale == "rows":
        rotor *= np.float16(16)
    else:
        vq *= np.float16(scale)
        rotor *= np.float16(scale)
        cents *= np.float16(scale)
    _compare_v(cuda_ops, oracle, v.reshape(-1, D).copy(), tb, vq, 8485, alpha, f"scale {scale}")


@pytest.mark.parametrize("rows", [9471, 9472, 9473, 9475])
def test_k_rows_vs_oracle(cuda_ops, oracle, rows):
    """K launches on either side of the line where a warp takes four rows, and with a last group of one to three rows."""
    import torch

    rng = np.random.default_rng(rows)
    base = 1201
    k, v = synth.make_kv(rng, (base + 3) // 4)
    tb = synth.make_tables(rng, 3, k.reshape(-1, D), v.reshape(-1, D)).as_f16()
    x = k.reshape(-1, D)[:base].copy()
    x[17] = 0
    want = oracle.compress(x, tb["d_k"], tb["rotor_k"], tb["cents_k"], tb["cents_k"].reshape(-1), base, 1.95, 1.0, False)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    out = dict(mask=torch.zeros(rows * 16, dtype=torch.int32, device="cuda"), norms=torch.zeros(rows, dtype=torch.float16, device="cuda"),
               r_norms=torch.zeros(rows, dtype=torch.float16, device="cuda"), payload=torch.zeros(rows * 40, dtype=torch.uint8, device="cuda"))
    meta = torch.ones(rows * 4, dtype=torch.uint8, device="cuda")
    cuda_ops.compress(dev(np.resize(x, (rows, D))), dev(tb["d_k"]), dev(tb["rotor_k"]), dev(tb["cents_k"]), dev(tb["cents_k"]), out["mask"],
                      out["norms"], out["r_norms"], out["payload"], meta, rows, D, 1.95, 1.0, False)
    assert not meta.any()
    for name, got in out.items():
        g = got.cpu().numpy().view(np.uint8).reshape(rows, -1)
        w = np.ascontiguousarray(want[name]).view(np.uint8).reshape(base, -1)
        bad = np.nonzero((g != np.resize(w, (rows, w.shape[1]))).any(axis=1))[0]
        assert len(bad) == 0, f"{name} differs in rows {bad[:8]} ({len(bad)} rows)"
