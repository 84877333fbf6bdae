"""Which rows a step hands to the native call as they are, and that every other form still goes through the copying appends."""
import pytest
import torch

from cases import D, H_KV, H_Q, SCALE
from test_cpu_host import RecordingOps, _tables
from bonsai_mojo_1bit_optimization_t4_cuda_b200.lib import ptr
from bonsai_mojo_1bit_optimization_t4_cuda_b200.runtime import KhqRuntime

KV = H_KV * D


class NativeOps(RecordingOps):
    """A backend with native calls: records the addresses a step is given."""

    def layer_ctx(self, L, ring_cap, rope_base):
        return object()

    def layer_step(self, ctx, q_gate, k_roped, v_new, k_unroped, out, *rest):
        self.calls.append(("native",) + tuple(ptr(t) for t in (k_roped, v_new, k_unroped, out)))


def _rows(kind):
    """The same values in a form that a native step must not read as contiguous fp16."""
    x = (torch.arange(KV) % 251 - 125).float()  # exact in every type
    if kind == "plain":
        return x.half()
    if kind == "shaped":
        return x.half().view(H_KV, D)
    if kind == "strided":  # a slice of a fused projection
        wide = torch.full((H_KV, 3, D), float("nan"), dtype=torch.float16)
        wide[:, 1] = x.half().view(H_KV, D)
        return wide[:, 1]
    if kind == "fp32":
        return x
    if kind == "bf16":
        return x.bfloat16()
    assert kind == "unaligned"
    buf = torch.zeros(KV + 8, dtype=torch.float16)
    off = next(i for i in range(1, 8) if buf[i:].data_ptr() % 16)
    buf[off:off + KV] = x.half()
    return buf[off:off + KV]


TABLES = _tables()


def _runtime():
    rt = KhqRuntime(NativeOps(), device="cpu")
    assert rt.khq_activate([TABLES], max_seq=512)
    rt.khq_init_layer(3, H_Q, H_KV, D)
    return rt


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("at", [0, 255])  # a plain step, and one with a compression event
@pytest.mark.parametrize("kind", ["plain", "shaped", "strided", "fp32", "bf16", "unaligned"])
@pytest.mark.parametrize("which", ["k_roped", "v", "k_unroped"])
def test_rows(kind, which, at, fused):
    rt = _runtime()
    L = rt.layers[3]
    L.write_pos = at
    row = {n: _rows("plain") for n in ("k_roped", "v", "k_unroped")}
    row[which] = _rows(kind)
    q, out = torch.zeros(H_Q * 2 * D, dtype=torch.float16), torch.zeros(H_Q * D, dtype=torch.float16)
    if fused:
        assert rt.khq_step_fused(3, q, row["k_unroped"], row["k_roped"], row["v"], out, SCALE)
    else:
        rt.khq_capture_unroped(3, row["k_unroped"])
        assert rt.khq_step(3, q, row["k_roped"], row["v"], out, SCALE)
    native = [c for c in rt.ops.calls if c[0] == "native"]
    as_is = kind in ("plain", "shaped")
    assert L.write_pos == at + 1 and len(rt.events) == (at == 255)
    ring = lambda name: L.t["ring_" + name].view(256, KV)[at]
    if as_is or which == "k_unroped":  # an un-RoPE'd row is appended by itself, the rest of the step can still be native
        assert native == [("native", row["k_roped"].data_ptr(), row["v"].data_ptr(),
                           row["k_unroped"].data_ptr() if fused and as_is else 0, out.data_ptr())]
    else:
        assert not native
        assert torch.equal(ring("k"), row["k_roped"].reshape(KV).half()) and torch.equal(ring("v"), row["v"].reshape(KV).half())
    if not (fused and as_is):
        assert torch.equal(ring("u"), row["k_unroped"].reshape(KV).half())


@pytest.mark.parametrize("fused", [False, True])
def test_wrong_size_and_unaligned_output(fused):
    """A row of another size is refused as the copying append refuses it, before anything is launched; an output off 16 bytes is served."""
    rt = _runtime()
    q, out = torch.zeros(H_Q * 2 * D, dtype=torch.float16), torch.zeros(H_Q * D + 8, dtype=torch.float16)
    plain, short = _rows("plain"), _rows("plain")[:KV - 8]
    step = (lambda k, o: rt.khq_step_fused(3, q, plain, k, plain, o, SCALE)) if fused else (lambda k, o: rt.khq_step(3, q, k, plain, o, SCALE))
    with pytest.raises(RuntimeError):
        step(short, out[:H_Q * D])
    assert not [c for c in rt.ops.calls if c[0] == "native"] and rt.layers[3].write_pos == 0
    off = next(i for i in range(1, 8) if out[i:].data_ptr() % 16)
    assert step(plain, out[off:off + H_Q * D])
    assert not [c for c in rt.ops.calls if c[0] == "native"] and rt.ops.calls[-1] == ("merge", True, False)


@pytest.mark.parametrize("splits", [1, 8])
def test_native_step_has_no_split_count(monkeypatch, splits):
    """The native launch cuts the compressed region itself: the same call whatever `splits` is, and nothing computed for it."""
    rt = _runtime()
    rt.splits = splits
    monkeypatch.setattr(rt, "_khq_split_count", lambda c_len: pytest.fail("not used by the native step"))
    seen = []
    monkeypatch.setattr(rt.ops, "layer_step", lambda *args: seen.append(args[6:]))
    q, out = torch.zeros(H_Q * 2 * D, dtype=torch.float16), torch.zeros(H_Q * D, dtype=torch.float16)
    rt.layers[3].write_pos, rt.layers[3].boundary = 300, 128
    assert rt.khq_step_fused(3, q, _rows("plain"), _rows("plain"), _rows("plain"), out, SCALE)
    assert seen == [(128, 173, False, 0, SCALE)]
