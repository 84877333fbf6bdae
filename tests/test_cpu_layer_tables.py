"""What a layer's native context holds a copy of (scalars, tables in the kernels' form) follows every change of the layer."""
import pytest
import torch

from cases import D, H_KV, H_Q, SCALE
from test_cpu_step_rows import TABLES, NativeOps, _rows
from bonsai_mojo_1bit_optimization_t4_cuda_b200.runtime import KHQ_TABLES, KhqRuntime

SCALARS = ("ts_k", "alpha_k", "ts_v", "alpha_v")


class CopyingOps(NativeOps):
    """A context is a copy of all that a context may hold a copy of; a step records the one that it is given."""

    def __init__(self):
        super().__init__()
        self.made, self.used, self.finished = 0, None, 0

    def layer_ctx(self, L, ring_cap, rope_base):
        self.made += 1
        return {n: L.t[n].clone() for n in KHQ_TABLES}, {n: getattr(L, n) for n in SCALARS}, {n: t.data_ptr() for n, t in L.t.items()}

    def layer_step(self, ctx, *args):
        self.used = ctx

    def finish_device(self):
        self.finished += 1


def _set(L):
    L.t["dk"] = L.t["dk"] * 2


def _update(L):
    L.t.update(vq=L.t["vq"] * 2)


def _union(L):
    L.t |= dict(cv=L.t["cv"] * 2)


def _pop(L):
    t = L.t.pop("rk")
    L.t.setdefault("rk", t + 1)


def _delete(L):
    t = L.t["rv"]
    del L.t["rv"]
    L.t["rv"] = t + 1


def _dict(L):
    L.t = dict(L.t, ring_k=torch.zeros_like(L.t["ring_k"]))


def _in_place(L):
    L.t["dv"].neg_()


def _view(L):
    L.t["ck"].view(4, D)[2].mul_(3.0)


def _replaced_then_in_place(L):
    L.t["vq"] = L.t["vq"].clone()  # no longer a part of the layer's own buffer
    L.t["vq"].mul_(0.5)


CHANGES = [_set, _update, _union, _pop, _delete, _dict, _in_place, _view, _replaced_then_in_place, *SCALARS]


@pytest.mark.parametrize("change", CHANGES, ids=lambda c: c if isinstance(c, str) else c.__name__.strip("_"))
def test_next_step_uses_the_new_values(change):
    rt = KhqRuntime(CopyingOps(), device="cpu")
    assert rt.khq_activate([TABLES], max_seq=512)
    rt.khq_init_layer(3, H_Q, H_KV, D)
    L, row = rt.layers[3], _rows("plain")
    q, out = torch.zeros(H_Q * 2 * D, dtype=torch.float16), torch.zeros(H_Q * D, dtype=torch.float16)
    step = lambda: rt.khq_step_fused(3, q, row, row, row, out, SCALE)
    assert step() and step() and rt.ops.made == 1
    if isinstance(change, str):
        setattr(L, change, getattr(L, change) + 0.25)
    else:
        change(L)
    assert step() and step()
    assert rt.ops.made == 2 and rt.ops.finished == 1  # one new context; the device had finished with the old one
    for n in KHQ_TABLES:  # and it counts the writes into each of the tables that are there now
        made = rt.ops.made
        L.t[n].add_(1)
        assert step() and step() and rt.ops.made == made + 1, n
    tables, scalars, at = rt.ops.used
    for n in KHQ_TABLES:
        assert torch.equal(tables[n], L.t[n]), n
    assert scalars == {n: getattr(L, n) for n in SCALARS}
    assert at == {n: t.data_ptr() for n, t in L.t.items()}


def test_refresh():
    rt = KhqRuntime(CopyingOps(), device="cpu")
    assert rt.khq_activate([TABLES], max_seq=512)
    rt.khq_init_layer(3, H_Q, H_KV, D)
    L, row = rt.layers[3], _rows("plain")
    q, out = torch.zeros(H_Q * 2 * D, dtype=torch.float16), torch.zeros(H_Q * D, dtype=torch.float16)
    L.t["dk"].numpy()[:] = 7  # a write that torch does not see
    rt.khq_refresh_tables(3)
    assert rt.khq_step_fused(3, q, row, row, row, out, SCALE)
    assert torch.equal(rt.ops.used[0]["dk"], L.t["dk"]) and float(L.t["dk"][0]) == 7


def test_tables_made_in_inference_mode():
    """Their writes are not counted; everything else works, and the call that reads them anew does."""
    rt = KhqRuntime(CopyingOps(), device="cpu")
    with torch.inference_mode():
        assert rt.khq_activate([TABLES], max_seq=512)
        rt.khq_init_layer(3, H_Q, H_KV, D)
        L, row = rt.layers[3], _rows("plain")
        q, out = torch.zeros(H_Q * 2 * D, dtype=torch.float16), torch.zeros(H_Q * D, dtype=torch.float16)
        assert rt.khq_step_fused(3, q, row, row, row, out, SCALE)
        L.t["dk"].neg_()
        rt.khq_refresh_tables(3)
        assert rt.khq_step_fused(3, q, row, row, row, out, SCALE)
        assert torch.equal(rt.ops.used[0]["dk"], L.t["dk"])
