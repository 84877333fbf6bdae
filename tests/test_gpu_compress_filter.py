"""V code search by launch size (shared by the warps of a block; large launches filtered on the tensor cores, exact where the
filter does not decide): code words bit-identical to the oracle's at the edges of the dispatch and of the row tiles, with tied and nearly tied codes, with codebooks and rows outside
the filter's range, and with a general alpha."""
import numpy as np
import pytest

from bonsai_mojo_1bit_optimization_t4_cuda_b200 import synth

pytestmark = pytest.mark.gpu
D = 256


@pytest.mark.parametrize("rows,kind", [(3, "plain"), (1184, "near"), (1185, "ties"), (8484, "plain"), (8485, "plain"), (9472, "ties"),
                                       (9473, "near"), (24641, "wide"), (25000, "odd_rows"), (28417, "ties")])
def test_v_codes_vs_oracle(cuda_ops, oracle, rows, kind):
    import torch

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
        vq[5] *= np.float16(3000)  # beyond the filter's range
    x = v.reshape(-1, D)[:base].copy()
    if kind == "odd_rows":
        x[17] = 0
        x[130] = np.float16(60000)
        x[4400, 7] = np.float16("inf")
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
        assert len(bad) == 0, f"{kind}: {name} differs in rows {bad[:8]} ({len(bad)} rows)"


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
