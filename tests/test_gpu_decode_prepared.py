"""Batched decode from prepared tables, and K rows that hold more outliers in a 16-dim word than the common path takes."""
import numpy as np
import pytest

import cases
from cases import D, H_Q, SCALE
from test_gpu_batched import oracle_step

pytestmark = pytest.mark.gpu


def dense_words(mask, rng):
    """Some rows with 9 to 16 outliers in one word (at most 50 a row), among them the first and the last row."""
    m = mask.reshape(-1, 16)
    m = np.where((m & (m >> 1)) & 0x55555555, m & ~(((m & (m >> 1)) & 0x55555555) * np.uint32(2)), m).astype(np.uint32)  # no outliers
    rows = np.unique(np.concatenate([[0, len(m) - 1], rng.integers(0, len(m), 12)]))
    for i, r in enumerate(rows):
        for w in rng.choice(16, 3, replace=False):
            m[r, w] |= np.uint32((1 << (2 * (9 + i % 8))) - 1)
    return m.reshape(mask.shape)


@pytest.mark.parametrize("variant,c_len,win_len", [("calib", 1, 0), ("calib", 47, 3), ("n01_idrot", 49, 0), ("calib", 640, 130)])
@pytest.mark.parametrize("dense", [False, True])
def test_prepared_tables_vs_oracle(cuda_ops, oracle, variant, c_len, win_len, dense):
    import torch

    from bonsai_mojo_1bit_optimization_t4_cuda_b200.batched import TABLES_DESC, BatchedDecode, prepare_tables
    from bonsai_mojo_1bit_optimization_t4_cuda_b200.lib import check, current_stream

    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    case = cases.make_case(5200 + c_len, c_len + win_len, variant, layer_id=3)
    f, tb = case["f16"], case["tables"]
    kv = cases.compress_with(oracle.compress, case, c_len)
    if dense:
        kv["k_mask"] = dense_words(kv["k_mask"], np.random.default_rng(c_len))
    ref, ring_k, ring_v = oracle_step(oracle, case, kv, c_len, c_len % 256, win_len)
    p = {k: dev(v) for k, v in kv.items() if k != "near_ties"}
    p.update(q_gate=dev(case["q_gate"]), ring_k=dev(ring_k), ring_v=dev(ring_v), table_id=0, c_len=c_len, start_pos=0,
             out=torch.zeros(H_Q * D, dtype=torch.float16, device="cuda"), win_start=c_len % 256, win_len=win_len)
    t = dict(cents_k=dev(f["cents_k"]), cents_v=dev(f["cents_v"]), vq=dev(f["vq"]), k_rotor=dev(f["rotor_k"]), v_rotor=dev(f["rotor_v"]),
             d_k=dev(f["d_k"]), d_v=dev(f["d_v"]), alpha_k=tb.alpha_k, alpha_v=tb.alpha_v)
    bd = BatchedDecode([p], [t], codebook_in_smem=2)
    bd.launch(SCALE, 1e7)
    plain = p["out"].clone()
    image = prepare_tables(bd.tables.cpu().numpy().view(TABLES_DESC), 1e7, "cuda")
    ptrs = torch.tensor([image.data_ptr()], dtype=torch.int64, device="cuda")
    p["out"].zero_()
    check("launch_khq_decode_batched_prepared_fp16", bd.lib.launch_khq_decode_batched_prepared_fp16(
        bd.descs.data_ptr(), bd.tables.data_ptr(), ptrs.data_ptr(), bd.items.data_ptr(), 1, bd.n_items, bd.workspace.data_ptr(),
        bd.ws_bytes, bd.n_items, SCALE, 1e7, 256, 2, current_stream()))
    torch.cuda.synchronize()
    assert cuda_ops.lib.khq_b200_device_status() == 0
    assert torch.equal(p["out"], plain)  # the same values, wherever the tables come from
    ok, mx, exc = cases.attention_close(plain.float().cpu().numpy().reshape(H_Q, D), ref.astype(np.float32))
    assert ok, f"max abs {mx:.3e} excess {exc:.3e}"


def test_step_right_behind_prepare(cuda_ops):
    """launch_khq_prepare_tables and a step of the layer on one stream, with nothing in between but the pre-step (which lets the attention
    start early): every step sees the image of its own tables."""
    import torch

    from bonsai_mojo_1bit_optimization_t4_cuda_b200.batched import TABLES_DESC
    from bonsai_mojo_1bit_optimization_t4_cuda_b200.lib import check, current_stream
    from bonsai_mojo_1bit_optimization_t4_cuda_b200.runtime import ROPE_BASE, KhqRuntime

    n = 300
    case = cases.make_case(612, n, "calib", layer_id=3)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    rt = KhqRuntime(cuda_ops, device="cuda")
    assert rt.khq_activate([case["tables"]], max_seq=512)
    rt.khq_init_layer(3, H_Q, cases.H_KV, D)
    L = rt.layers[3]
    rows = [dev(case[a]) for a in ("k_unroped", "k_roped", "v")]
    q = dev(case["q_gate"]).reshape(-1)
    out = torch.zeros(H_Q * D, dtype=torch.float16, device="cuda")
    for t in range(n - 1):
        assert rt.khq_step_fused(3, q, *(x[t] for x in rows), out, SCALE)
    descs = []
    for alpha_v in (1.0, 0.5):  # two sets of tables that share all but one scalar
        t = np.zeros(1, TABLES_DESC)
        for field, name in (("cents_k", "ck"), ("cents_v", "cv"), ("vq", "vq"), ("k_rotor", "rk"), ("v_rotor", "rv"), ("d_k", "dk"), ("d_v", "dv")):
            t[field] = L.t[name].data_ptr()
        t["alpha_k"], t["alpha_v"] = L.alpha_k, alpha_v
        descs.append(t)
    image, (boundary, write_pos) = L.t.ctx[2], (L.boundary, L.write_pos)
    assert boundary == 128

    def step(desc, wait):
        L.boundary, L.write_pos = boundary, write_pos
        qn, o = q.clone(), torch.zeros_like(out)
        k = rows[0][n - 1].reshape(-1).clone()
        check("launch_khq_prepare_tables", cuda_ops.lib.launch_khq_prepare_tables(desc.ctypes.data, ROPE_BASE, image.data_ptr(), current_stream()))
        if wait:
            torch.cuda.synchronize()
        assert rt.khq_prestep(3, qn, k, rows[2][n - 1], n - 1)
        assert rt.khq_step(3, qn, k, rows[2][n - 1], o, SCALE, rings_written=True)
        return o

    want = [step(d, True) for d in descs]
    assert not torch.equal(want[0], want[1])
    got = [step(descs[i % 2], False) for i in range(20)]
    torch.cuda.synchronize()
    for i, o in enumerate(got):
        assert torch.equal(o, want[i % 2]), f"step {i}"
