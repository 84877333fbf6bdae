"""The batch engine as a decode engine: eight sequences with different histories decode 300
tokens through BatchEngine.decode_step (batched pre-step, batched compression events, re-planned
batched attention) and must end in the state, and produce the outputs, of eight independent
single-sequence runtimes (KhqRuntime, the host state machine of src/khq/runtime.mojo:454-613)
fed the same projections."""
import numpy as np
import pytest

import cases
from cases import D, H_KV, H_Q, SCALE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("generation", [2, 3, 4])
def test_engine_decodes_like_independent_runtimes(cuda_ops, generation):
    import torch

    from bonsai_mojo_1bit_optimization_t4_cuda_b200.engine import BatchEngine
    from bonsai_mojo_1bit_optimization_t4_cuda_b200.runtime import KhqRuntime

    B, steps = 8, 300
    layer_ids = [3, 7]
    rng = np.random.default_rng(2027)
    sk, sv = cases.synth.channel_scales(rng), cases.synth.channel_scales(rng)
    sample_k, sample_v = cases.synth.make_kv(rng, 128, sk, sv)
    tables = [cases.synth.make_tables(rng, li, sample_k.reshape(-1, D), sample_v.reshape(-1, D), vq_scale=1.0 / 16.0)
              for li in layer_ids]
    norm_w = [((1 + 0.1 * rng.standard_normal(D)).astype(np.float32), (1 + 0.1 * rng.standard_normal(D)).astype(np.float32))
              for _ in layer_ids]
    start = [0, 17, 17, 40, 63, 90, 127, 200]  # raw tokens each sequence already holds; two share a history length

    def projections(step, seq, layer):
        g = np.random.default_rng([step + 100_000, seq, layer])
        q = g.standard_normal((H_Q, 2 * D)).astype(np.float16)
        k = (g.standard_normal((H_KV, D)) * sk).astype(np.float16)
        v = (g.standard_normal((H_KV, D)) * sv).astype(np.float16)
        return q, k, v

    # ---- reference: one runtime per sequence ------------------------------------------------------
    rts = []
    for s in range(B):
        rt = KhqRuntime(cuda_ops, device="cuda")
        assert rt.khq_activate(tables, max_seq=1024)
        for li in layer_ids:
            rt.khq_init_layer(li, H_Q, H_KV, D)
        rts.append(rt)

    def runtime_step(rt, seq, step_id, pos):
        outs = []
        for l, li in enumerate(layer_ids):
            q, k, v = projections(step_id, seq, l)
            qg, kd, vd = torch.from_numpy(q).cuda().reshape(-1), torch.from_numpy(k).cuda().reshape(-1), torch.from_numpy(v).cuda().reshape(-1)
            out = torch.zeros(H_Q * D, dtype=torch.float16, device="cuda")
            assert rt.khq_prestep(li, qg, kd, vd, pos, torch.from_numpy(norm_w[l][0]).cuda(), torch.from_numpy(norm_w[l][1]).cuda())
            assert rt.khq_step(li, qg, kd, vd, out, SCALE, rings_written=True)
            outs.append(out)
        return outs

    for s in range(B):  # histories: negative step ids so that they never collide with the common steps
        for t in range(start[s]):
            runtime_step(rts[s], s, -1 - t, t)
    # ---- the engine starts from those histories ------------------------------------------------------
    eng = BatchEngine(tables, [0] * B, start, device="cuda", codebook_in_smem=generation, grow_tokens=512, norm_weights=norm_w)
    for l, li in enumerate(layer_ids):
        for s in range(B):
            if start[s]:
                T = rts[s].layers[li].t
                n = start[s] * H_KV * D
                eng.load_window(l, s, T["ring_k"][:n], T["ring_v"][:n], T["ring_u"][:n])
    worst = 0.0
    for step in range(steps):
        for l in range(len(layer_ids)):
            for s in range(B):
                q, k, v = projections(step, s, l)
                eng.h_q[l, s].copy_(torch.from_numpy(q).reshape(-1))
                eng.h_k[l, s].copy_(torch.from_numpy(k).reshape(-1))
                eng.h_v[l, s].copy_(torch.from_numpy(v).reshape(-1))
        out = eng.decode_step(SCALE)
        torch.cuda.synchronize()
        got = out.float().numpy().reshape(len(layer_ids), B, H_Q, D).copy()
        check_outputs = step < 4 or step % 16 == 0 or step >= steps - 2 or any((start[s] + step + 1) in (255, 256, 257) for s in range(B))
        for s in range(B):
            want = runtime_step(rts[s], s, step, start[s] + step)
            if check_outputs:
                torch.cuda.synchronize()
                for l in range(len(layer_ids)):
                    ok, mx, exc = cases.attention_close(got[l, s], want[l].float().cpu().numpy().reshape(H_Q, D))
                    worst = max(worst, mx)
                    assert ok, f"step {step} sequence {s} layer {l}: max abs {mx:.3e} excess {exc:.3e}"
    assert cuda_ops.lib.khq_b200_device_status() == 0
    # ---- final state: positions, code words of every compressed token, raw rings ---------------------
    assert eng.events_fired == sum(1 for s in range(B) if start[s] + steps >= 256) + sum(1 for s in range(B) if start[s] + steps >= 384)
    per_row = dict(k_mask=("kmask", 64), k_payload=("kpay", 40), v_payload=("vpay", 104), v_shared_meta=("vsm", 4),
                   k_norms=("knorm", 2), k_r_norms=("krn", 2), v_norms=("vnorm", 2), v_r_norms=("vrn", 2))
    for s in range(B):
        for l, li in enumerate(layer_ids):
            Lr = rts[s].layers[li]
            assert int(eng.boundary[s]) == Lr.boundary and int(eng.write_pos[s]) == Lr.write_pos
            rows = Lr.boundary * H_KV
            r0 = int(eng.row_off[s])
            for key, (rkey, rb) in per_row.items():
                a = eng.pay[l][key].view(torch.uint8)[r0 * rb:(r0 + rows) * rb]
                b = Lr.t[rkey].view(torch.uint8)[:rows * rb]
                assert torch.equal(a, b), f"sequence {s} layer {l}: code words differ in {key}"
            for ring, rkey in ((eng.ring_k, "ring_k"), (eng.ring_v, "ring_v"), (eng.ring_u, "ring_u")):
                assert torch.equal(ring[l][s].reshape(-1), Lr.t[rkey].reshape(-1)), f"sequence {s} layer {l}: {rkey} differs"
    print(f"engine vs independent runtimes, generation {generation}: {eng.events_fired} events, worst output |err| {worst:.2e}")


def _small_engine(layers, seqs=2, alpha_v=1.0):
    """An engine with the same tables in every layer, on synthetic state and inputs."""
    import torch

    from bonsai_mojo_1bit_optimization_t4_cuda_b200.engine import BatchEngine

    rng = np.random.default_rng(4)
    k, v = cases.synth.make_kv(rng, 64)
    tb = cases.synth.make_tables(rng, 3, k.reshape(-1, D), v.reshape(-1, D), vq_scale=1.0 / 16.0)
    tb.alpha_v = alpha_v
    eng = BatchEngine([tb] * layers, [256, 128][:seqs], [150, 140][:seqs], grow_tokens=128)
    eng.fill_synthetic(7)
    g = torch.Generator().manual_seed(9)
    for h in (eng.h_q, eng.h_k, eng.h_v):
        h.copy_(torch.randn(h.shape, generator=g).half())
    return eng


def test_refreshed_tables(cuda_ops):
    """Tables changed behind the constructor take effect with refresh_tables."""
    import torch

    want, eng = _small_engine(2, alpha_v=0.5), _small_engine(2)
    for l in range(2):  # the same code words and raw tokens
        for n, t in eng.pay[l].items():
            want.pay[l][n].copy_(t)
        for a, b in ((want.ring_k, eng.ring_k), (want.ring_v, eng.ring_v), (want.ring_u, eng.ring_u)):
            a[l].copy_(b[l])
        want.tables[l]["vq"].mul_(0.75)
    want.refresh_tables()
    for tb in eng.tables:
        tb["vq"], tb["alpha_v"] = tb["vq"] * 0.75, 0.5
    eng.refresh_tables()
    a, b = want.decode_step(SCALE), eng.decode_step(SCALE)
    torch.cuda.synchronize()
    assert a.any() and torch.equal(a, b)


def test_engine_dropped_with_a_step_in_flight(cuda_ops):
    """An engine that goes away while its step is still queued waits for it: the outputs are complete behind that."""
    import gc

    import torch

    eng = _small_engine(3)
    want = eng.decode_step(SCALE)
    torch.cuda.synchronize()
    want = want.clone()
    del eng
    eng = _small_engine(3)
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # about a tenth of a second in front of the step
    got = eng.decode_step(SCALE)
    assert not torch.cuda.current_stream().query()
    del eng
    gc.collect()
    assert want.any() and torch.equal(got, want)
    torch.cuda.synchronize()


@pytest.mark.parametrize("layers,per_chunk", [(65, 1), (66, 0)])  # 0: as the constructor chooses
def test_more_than_64_layers(cuda_ops, layers, per_chunk):
    """The number of layers, and of the groups that are copied together, has no limit: the outputs of every layer are those that the
    attention alone gives over the state behind the step."""
    import torch

    eng = _small_engine(layers)
    if per_chunk:
        eng._args.layers_per_chunk = per_chunk
    got = eng.decode_step(SCALE)
    torch.cuda.synchronize()
    got = got.clone()
    for l in range(layers):
        eng.out[l].zero_()
        eng.attention_resident(l, SCALE)
    torch.cuda.synchronize()
    assert got.any(-1).all() and torch.equal(got, eng._out.cpu())
    assert eng.decode_step(SCALE) is eng.h_out
    torch.cuda.synchronize()


@pytest.mark.parametrize("form", ["pinned", "pageable", "fp32", "strided", "device", "list"])
def test_replaced_host_buffers(cuda_ops, form):
    """The host buffers are the attributes' at every step: other tensors of the same values give the same outputs."""
    import torch

    eng = _small_engine(3)
    start = eng.boundary.copy(), eng.write_pos.copy()

    def step():
        eng.boundary[:], eng.write_pos[:] = start
        return eng.decode_step(SCALE)

    first = step()
    torch.cuda.synchronize()
    first = first.clone()
    g = torch.Generator().manual_seed(19)
    other = [torch.randn(h.shape, generator=g).half() for h in (eng.h_q, eng.h_k, eng.h_v)]
    own = eng.h_q, eng.h_k, eng.h_v, eng.h_out
    for h, x in zip(own, other):
        h.copy_(x)
    want = step()
    torch.cuda.synchronize()
    want = want.clone()
    assert not torch.equal(want, first)
    for h in own:
        h.fill_(float("nan"))  # nothing may be read from here any more
    make = dict(pinned=lambda x: x.pin_memory(), pageable=lambda x: x.clone(), fp32=lambda x: x.float(), device=lambda x: x.cuda(),
                strided=lambda x: torch.stack([x, x], -1)[..., 0], list=lambda x: [r.clone() for r in x])[form]
    eng.h_q, eng.h_k, eng.h_v = (make(x) for x in other)
    eng.h_out = make(torch.zeros_like(want))
    got = step()
    assert got is eng.h_out
    torch.cuda.synchronize()
    got = torch.stack(list(got)) if form == "list" else got
    assert torch.equal(got.cpu().half(), want)


@pytest.mark.parametrize("c_len,win,kernel", [
    ([0, 128, 256], [1, 128, 250], 5), ([1664], [200], 5), ([1920], [130], 6), ([0, 4224, 128, 1280], [255, 129, 131, 200], 6),
    ([16000], [200], 6), ([640] * 6, [128, 140, 150, 160, 170, 180], 6), ([40064], [200], -1), ([128] * 16, [130] * 16, -1)])
def test_small_batches_through_the_step_kernels(cuda_ops, c_len, win, kernel):
    """The same step through the kernels of a single sequence (khq_b200_plan_steps), where that takes the batch, and through the
    persistent one."""
    import torch

    from bonsai_mojo_1bit_optimization_t4_cuda_b200.engine import BatchEngine

    rng = np.random.default_rng(4)
    k, v = cases.synth.make_kv(rng, 64)
    tb = cases.synth.make_tables(rng, 3, k.reshape(-1, D), v.reshape(-1, D), vq_scale=1.0 / 16.0)
    outs, engines = [], []
    for gen in (-1, 2):
        eng = BatchEngine([tb, tb], c_len, win, grow_tokens=128, codebook_in_smem=gen)
        eng.fill_synthetic(7)
        g = torch.Generator().manual_seed(9)
        steps = []
        for _ in range(3):  # the counters are left as they were
            for h in (eng.h_q, eng.h_k, eng.h_v):
                h.copy_(torch.randn(h.shape, generator=g).half())
            eng.decode_step(SCALE)
            torch.cuda.synchronize()
            steps.append(eng.h_out.float().clone())
        outs.append(torch.stack(steps))
        engines.append(eng)
    assert engines[0]._kernel == kernel and engines[1]._kernel == 2 and cuda_ops.lib.khq_b200_device_status() == 0
    # fp32 sums in another order on both sides (some 1e-6 of the largest term), then one rounding to fp16
    err, want = (outs[0] - outs[1]).abs(), outs[1].abs()
    assert bool((err <= 2.0 ** -10 * want + 3e-4 * want.max()).all()), float(err.max())
    for eng in engines:  # the resident entry, with the items of the last step
        eng.attention_resident(0, SCALE)
    torch.cuda.synchronize()
    a, b = (eng.out[0].float() for eng in engines)
    assert bool(((a - b).abs() <= 2.0 ** -10 * b.abs() + 3e-4 * b.abs().max()).all())
