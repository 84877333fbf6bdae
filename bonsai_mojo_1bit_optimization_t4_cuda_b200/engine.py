"""Batched KHQ decode engine: B independent sequences x L attention layers resident on one GPU.

This is the public entry a serving host calls once per generated token: hand it this step's
projections for every sequence (host buffers), get the gated attention outputs back (host
buffers).  Sequences are independent, so they shard across GPUs by sequence with no collective
(one engine per rank).

Per step and sequence the engine does what the reference's ``khq_step`` does for its single
sequence (``src/khq/runtime.mojo:454-613``): the new token goes to ring slot ``write_pos % 256``
and ``write_pos`` advances; when the raw window has reached 256 tokens (and the compressed
capacity allows) the 128 oldest tokens are compressed and ``boundary`` moves on by 128; the
attention then runs over ``c_len = boundary`` compressed tokens and the ``write_pos - boundary``
raw ones.  Per layer that is one launch for the q/k head norms, K capture, RoPE and the three
ring appends of ALL sequences (``launch_khq_prestep_batched_fp16``), one K and one V compress
launch over the sequences whose event is due (``launch_khq_compress_batched_fp16``), and one
batched attention launch (``launch_khq_decode_batched_fp16``); the work items are re-planned
on the host every step and the step-dependent descriptor fields of every layer are rewritten by
one small launch (``launch_khq_update_descs``).  All of it is issued by one native call
(``launch_khq_engine_step``).

State layout: one contiguous device buffer per payload array and per layer, each sequence's
slice sized for its capacity and starting on a 128-row boundary.
"""
from __future__ import annotations

import collections
import ctypes
from typing import Optional, Sequence

import numpy as np
import torch

from . import lib as _lib
from .batched import SEQ_DESC, TABLES_DESC, WORK_ITEM, prepare_tables
from .calib import KhqLayerTables
from .lib import check, current_stream
from .synth import H_KV, H_Q

D = 256
RING = 256
CHUNK = 128
WATERMARK = 256
KV = H_KV * D  # halfs per token row group
ROTARY_DIM = 64
COPY_BYTES = 256 * 1024
SEQ_DYN = np.dtype([("c_len", "<i4"), ("start_pos", "<i4"), ("win_start", "<i4"), ("win_len", "<i4"),
                    ("first_slot", "<i4"), ("n_slots", "<i4"), ("r0", "<i4"), ("r1", "<i4")])
COMPRESS_SEG = np.dtype([("x", "<u8"), ("row0", "<i8")])
assert SEQ_DYN.itemsize == 32 and COMPRESS_SEG.itemsize == 16


def _align(n: int, a: int = 256) -> int:
    return (n + a - 1) // a * a


class BatchEngine:
    def __init__(self, tables: Sequence[KhqLayerTables], c_len: Sequence[int], win_len: Sequence[int],
                 device="cuda", tokens_per_item: int = 0, codebook_in_smem: int = -1, grow_tokens: int = 1024,
                 norm_weights: Optional[Sequence] = None, rope_theta: float = 1e7, rms_eps: float = 1e-6):
        """``c_len`` / ``win_len``: compressed and raw tokens each sequence starts with (``c_len`` a
        multiple of 128, as the state machine leaves it).  ``grow_tokens``: compressed capacity kept
        free behind every sequence's initial prefix.  ``norm_weights``: per layer ``(q_w, k_w)`` fp32
        (256,) arrays for the head RMS norms, or None for the unweighted norm.  The tables (``self.tables``) and norms
        (``self.norm_w``) are laid out for the kernels here: whoever changes one of them later calls ``refresh_tables``."""
        self.lib = _lib.load()
        self.device = torch.device(device)
        self.L = len(tables)
        self.B = len(c_len)
        self.boundary = np.asarray(c_len, np.int64).copy()
        self.write_pos = self.boundary + np.asarray(win_len, np.int64)
        assert (self.boundary % CHUNK == 0).all(), "compressed prefixes are whole 128-token chunks"
        assert ((self.write_pos - self.boundary) <= RING).all() and (np.asarray(win_len) >= 0).all()
        self.cap = self.boundary + _align(max(int(grow_tokens), 0), CHUNK)
        self.codebook_in_smem = codebook_in_smem
        self.rope_theta, self.rms_eps = float(rope_theta), float(rms_eps)
        self.host_tables = list(tables)
        dev = self.device
        z = lambda n, dt: torch.zeros(max(int(n), 1), dtype=dt, device=dev)
        # ---- tables ------------------------------------------------------------------------
        self.tables = []
        for tb in tables:
            f = tb.as_f16()
            self.tables.append(dict(
                cents_k=torch.from_numpy(f["cents_k"]).to(dev), cents_v=torch.from_numpy(f["cents_v"]).to(dev),
                vq=torch.from_numpy(f["vq"]).to(dev), k_rotor=torch.from_numpy(f["rotor_k"]).to(dev),
                v_rotor=torch.from_numpy(f["rotor_v"]).to(dev), d_k=torch.from_numpy(f["d_k"]).to(dev),
                d_v=torch.from_numpy(f["d_v"]).to(dev), alpha_k=tb.alpha_k, alpha_v=tb.alpha_v,
                ts_k=tb.ts_k, ts_v=tb.ts_v))
        t = self._tables_desc()
        self.d_tables = torch.from_numpy(t.view(np.uint8).reshape(-1).copy()).to(dev)
        self._images = prepare_tables(t, self.rope_theta, dev)
        self._d_images = torch.tensor([im.data_ptr() for im in self._images], dtype=torch.int64, device=dev)
        self.norm_w = None
        if norm_weights is not None:
            self.norm_w = [(torch.as_tensor(np.asarray(q, np.float32)).to(dev), torch.as_tensor(np.asarray(k, np.float32)).to(dev))
                           for q, k in norm_weights]
        # ---- payload arrays: per layer one buffer per array, sequences at aligned row offsets --
        rows = self.cap * H_KV
        self.row_off = np.zeros(self.B + 1, np.int64)  # in rows, multiples of 128 rows
        for i in range(self.B):
            self.row_off[i + 1] = self.row_off[i] + _align(int(rows[i]), 128)
        R = int(self.row_off[-1])
        self.pay = [dict(k_mask=z(R * 16, torch.int32), k_payload=z(R * 40, torch.uint8),
                         v_payload=z(R * 104, torch.uint8), v_shared_meta=z(R * 4, torch.uint8),
                         k_norms=z(R, torch.float16), k_r_norms=z(R, torch.float16),
                         v_norms=z(R, torch.float16), v_r_norms=z(R, torch.float16)) for _ in range(self.L)]
        ring = lambda: z(self.B * RING * KV, torch.float16).view(self.B, RING, KV)
        self.ring_k = [ring() for _ in range(self.L)]
        self.ring_v = [ring() for _ in range(self.L)]
        self.ring_u = [ring() for _ in range(self.L)]
        # inputs and outputs of all layers in one buffer each, so that a copy can take several layers
        self._q = z(self.L * self.B * H_Q * 2 * D, torch.float16).view(self.L, self.B, H_Q * 2 * D)
        self._out = z(self.L * self.B * H_Q * D, torch.float16).view(self.L, self.B, H_Q * D)
        self._k = z(self.L * self.B * KV, torch.float16).view(self.L, self.B, KV)
        self._v = z(self.L * self.B * KV, torch.float16).view(self.L, self.B, KV)
        self.q_gate, self.out = list(self._q), list(self._out)
        # ---- descriptors: layer-major, pointers fixed, the step-dependent ints rewritten per step
        d = np.zeros(self.L * self.B, SEQ_DESC)
        for l in range(self.L):
            P = self.pay[l]
            for i in range(self.B):
                r0 = int(self.row_off[i])
                e = d[l * self.B + i]
                e["q_gate"], e["out"] = self.q_gate[l][i].data_ptr(), self.out[l][i].data_ptr()
                e["ring_k"], e["ring_v"] = self.ring_k[l][i].data_ptr(), self.ring_v[l][i].data_ptr()
                e["k_mask"], e["k_payload"] = P["k_mask"][r0 * 16:].data_ptr(), P["k_payload"][r0 * 40:].data_ptr()
                e["v_payload"], e["v_shared_meta"] = P["v_payload"][r0 * 104:].data_ptr(), P["v_shared_meta"][r0 * 4:].data_ptr()
                e["k_norms"], e["k_r_norms"] = P["k_norms"][r0:].data_ptr(), P["k_r_norms"][r0:].data_ptr()
                e["v_norms"], e["v_r_norms"] = P["v_norms"][r0:].data_ptr(), P["v_r_norms"][r0:].data_ptr()
                e["table_id"] = l
        self.d_descs = torch.from_numpy(d.view(np.uint8).reshape(-1).copy()).to(dev)
        # ---- planning ----------------------------------------------------------------------
        # tokens_per_item <= 0: the library's planner chooses (it is handed 0 every step); the size it would start
        # from only bounds the buffers here
        self.tokens_per_item_arg = int(tokens_per_item) if tokens_per_item > 0 else 0
        if tokens_per_item <= 0:
            sms = torch.cuda.get_device_properties(dev).multi_processor_count if dev.type == "cuda" else 148
            tokens_per_item = int(min(max(int(self.cap.sum()) // (2 * sms), 96), 8192))
        self.tokens_per_item = (tokens_per_item + 95) // 96 * 96
        # the planner shrinks the last items of a launch (down to 48 tokens), or cuts one to three pieces per
        # SM: room for either on top of the full-size items
        sms_plan = torch.cuda.get_device_properties(dev).multi_processor_count if dev.type == "cuda" else 148
        tail_items = int(4 * sms_plan * (1.0 + np.log(self.tokens_per_item / 48.0))) + 16
        self.max_items = int(sum((int(c) + self.tokens_per_item - 1) // self.tokens_per_item + 2 for c in self.cap)) + tail_items
        # the last bytes: counters of the step kernels (khq_b200_plan_steps), zero
        self.ws_bytes = _align(int(self.lib.khq_b200_decode_workspace_bytes(self.max_items)), 256) + _align(self.B * H_Q * 4, 256)
        self.workspace = z(self.ws_bytes, torch.uint8)
        # a step's control block: per-sequence state, ring slots, positions, work items and, last, the runs that are
        # compressed this step (copied only when there are some); one copy per step, device and host laid out alike
        parts = [("dyn", self.B * SEQ_DYN.itemsize), ("slots", self.B * 4), ("pos", self.B * 4), ("items", self.max_items * WORK_ITEM.itemsize),
                 ("segs", self.L * self.B * COMPRESS_SEG.itemsize)]
        self._at, n = {}, 0
        for name, size in parts:
            self._at[name] = n
            n = _align(n + size, 128)
        self.d_control = z(n, torch.uint8)
        self.d_items = self.d_control[self._at["items"]:]
        self.d_dyn = self.d_control[self._at["dyn"]:self._at["dyn"] + self.B * SEQ_DYN.itemsize]
        # ---- pinned host staging: two parities of the control block, one set of data buffers ----
        cuda = dev.type == "cuda"
        pin = lambda *shape, dt=torch.float16: (torch.zeros(*shape, dtype=dt).pin_memory() if cuda else torch.zeros(*shape, dtype=dt))
        self.h_q = pin(self.L, self.B, H_Q * 2 * D)
        self.h_k = pin(self.L, self.B, KV)
        self.h_v = pin(self.L, self.B, KV)
        self.h_out = pin(self.L, self.B, H_Q * D)
        self._staging = dict(q=self.h_q, k=self.h_k, v=self.h_v, out=self.h_out)
        self._in_flight = collections.deque(maxlen=4)  # host buffers of the last steps (at most two are not complete)
        self._ctl = []
        for _ in range(2):
            block = pin(n, dt=torch.uint8)
            raw = block.numpy()
            part = lambda name, dt, count: raw[self._at[name]:self._at[name] + count * np.dtype(dt).itemsize].view(dt)
            self._ctl.append(dict(block=block, dyn=part("dyn", SEQ_DYN, self.B), slots=part("slots", np.int32, self.B),
                                  pos=part("pos", np.int32, self.B), items=part("items", WORK_ITEM, self.max_items),
                                  segs=part("segs", COMPRESS_SEG, self.L * self.B).reshape(self.L, self.B)))
        # ---- native side: copy streams and events, the layers' addresses, the step's arguments --------
        self._native = ctypes.c_void_p()
        if cuda:
            with torch.cuda.device(dev):
                check("khq_b200_engine_create", self.lib.khq_b200_engine_create(ctypes.byref(self._native)))
        self._layers = (_lib.EngineLayer * self.L)()
        for l in range(self.L):
            y = self._layers[l]
            for f, src in self.pay[l].items():
                setattr(y, f, src.data_ptr())
            y.ring_k, y.ring_v, y.ring_u = self.ring_k[l].data_ptr(), self.ring_v[l].data_ptr(), self.ring_u[l].data_ptr()
        self._fill_layer_tables()
        self._ring_u_at = np.array([r.data_ptr() for r in self.ring_u], np.uint64)
        a = self._args = _lib.EngineStep()
        a.d_q, a.d_k, a.d_v, a.d_out = self._q.data_ptr(), self._k.data_ptr(), self._v.data_ptr(), self._out.data_ptr()
        base = self.d_control.data_ptr()
        a.d_control = base
        for f in ("items", "dyn", "slots", "pos", "segs"):
            setattr(a, "d_" + f, base + self._at[f])
        a.descs, a.tables, a.workspace, a.workspace_bytes = (self.d_descs.data_ptr(), self.d_tables.data_ptr(), self.workspace.data_ptr(),
                                                             self.ws_bytes)
        a.images = self._d_images.data_ptr()
        a.n_layers, a.n_seq, a.ring_cap, a.rotary_dim = self.L, self.B, RING, ROTARY_DIM
        self._laid_out_theta = a.rope_theta = self.rope_theta
        # A copy of a few tens of KB takes as long as one of 256 KB (3-4 us): layers are copied in groups of about that
        # much, at most half of them at once so that copies and kernels still overlap.
        a.layers_per_chunk = int(min(max(COPY_BYTES // (self.B * (H_Q * 2 * D + 2 * KV) * 2), 1), max(self.L // 2, 1)))
        self._step = 0
        self.n_items = 0
        self.events_fired = 0
        self._plan(self._ctl[0])
        if cuda:
            nb = self._control_bytes(0)
            self.d_control[:nb].copy_(self._ctl[0]["block"][:nb])
            check("launch_khq_update_descs", self.lib.launch_khq_update_descs(self.d_descs.data_ptr(), self.d_dyn.data_ptr(), self.B,
                                                                              self.L, current_stream()))

    def __del__(self):  # the buffers go after this, which waits for the copies of a step in flight
        native = getattr(self, "_native", None)
        if native:
            self.lib.khq_b200_engine_destroy(native)
            self._native = None

    # ---------------------------------------------------------------------------------- tables
    def _tables_desc(self) -> np.ndarray:
        t = np.zeros(self.L, TABLES_DESC)
        for i, tb in enumerate(self.tables):
            for k in ("cents_k", "cents_v", "vq", "k_rotor", "v_rotor", "d_k", "d_v"):
                t[k][i] = tb[k].data_ptr()
            t["alpha_k"][i], t["alpha_v"][i] = tb["alpha_k"], tb["alpha_v"]
        return t

    def _fill_layer_tables(self) -> None:
        for l, (y, tb) in enumerate(zip(self._layers, self.tables)):
            if self.norm_w is not None:
                y.q_norm, y.k_norm = self.norm_w[l][0].data_ptr(), self.norm_w[l][1].data_ptr()
            for f, src in (("d_k", "d_k"), ("cents_k", "cents_k"), ("rotor_k", "k_rotor"), ("d_v", "d_v"), ("cents_v", "cents_v"),
                           ("rotor_v", "v_rotor"), ("vq", "vq")):
                setattr(y, f, tb[src].data_ptr())
            y.ts_k, y.alpha_k, y.ts_v, y.alpha_v = tb["ts_k"], tb["alpha_k"], tb["ts_v"], tb["alpha_v"]

    def refresh_tables(self) -> None:
        """Entries of ``self.tables`` have been replaced or written into, or ones of ``self.norm_w`` replaced: the steps behind this
        call use the new values.  Waits for the device."""
        with torch.cuda.device(self.device):
            torch.cuda.synchronize()  # steps in flight read the old tables; writes into the new ones have to be complete
            t = self._tables_desc()
            self.d_tables.copy_(torch.from_numpy(t.view(np.uint8).reshape(-1).copy()))
            self._images.copy_(prepare_tables(t, self.rope_theta, self.device))
            self._fill_layer_tables()
            self._laid_out_theta = self._args.rope_theta = self.rope_theta
            torch.cuda.synchronize()

    # ---------------------------------------------------------------------------------- sizes
    @property
    def c_len(self) -> np.ndarray:
        return self.boundary

    @property
    def win_len(self) -> np.ndarray:
        return self.write_pos - self.boundary

    @property
    def win_start(self) -> np.ndarray:
        return self.boundary % RING

    @property
    def algorithmic_bytes_per_layer(self) -> int:
        return int(H_KV * (220 * self.boundary + 1024 * (self.write_pos - self.boundary)).sum())

    @property
    def h2d_bytes_per_step(self) -> int:
        """Projections of one step for every layer and sequence plus the step's control block
        (work items, per-sequence state, ring slots, positions)."""
        return self.L * self.B * (H_Q * 2 * D + 2 * KV) * 2 + self._control_bytes(0)

    @property
    def d2h_bytes_per_step(self) -> int:
        return self.L * self.B * H_Q * D * 2

    # ---------------------------------------------------------------------------------- planning
    def _control_bytes(self, n_events: int) -> int:
        """Bytes of the control block that a step with n_events compression events copies."""
        if n_events:
            return self._at["segs"] + self.L * self.B * COMPRESS_SEG.itemsize
        return self._at["items"] + self.n_items * WORK_ITEM.itemsize

    def _plan(self, ctl) -> None:
        """Cut the current compressed prefixes and windows into work items (host planner of the
        library) and write items and per-sequence state into the host control block; one launch then
        rewrites the step-dependent fields of all L x B descriptors from it."""
        dyn = ctl["dyn"]
        c = self.boundary.astype(np.int32)
        w = (self.write_pos - self.boundary).astype(np.int32)
        first = np.empty(self.B, np.int32)
        cnt = np.empty(self.B, np.int32)
        items = ctl["block"].data_ptr() + self._at["items"]
        # a small batch: the kernels of a single sequence's step
        self._kernel, steps = int(self.codebook_in_smem), ctypes.c_int(0)
        mode = 0
        if self._kernel < 0 and self.tokens_per_item_arg == 0:
            mode = self.lib.khq_b200_plan_steps(c.ctypes.data, w.ctypes.data, self.B, items, self.max_items, ctypes.addressof(steps),
                                                first.ctypes.data, cnt.ctypes.data)
        if mode > 0:
            self._kernel, n = mode, steps.value
        else:
            n = self.lib.khq_b200_plan_decode(c.ctypes.data, w.ctypes.data, self.B, self.tokens_per_item_arg, items, self.max_items,
                                              first.ctypes.data, cnt.ctypes.data)
            if n < 0 or n > self.max_items:
                raise _lib.KhqLaunchError("khq_b200_plan_decode", n)
        self.n_items = int(n)
        dyn["c_len"], dyn["start_pos"], dyn["win_start"], dyn["win_len"] = c, 0, c % RING, w
        dyn["first_slot"], dyn["n_slots"] = first, cnt

    # ---------------------------------------------------------------------------------- loading
    def compress_into(self, layer: int, seq: int, k_unroped: torch.Tensor, v: torch.Tensor, tok0: int = 0) -> None:
        """Compress tokens [tok0, tok0+n) of one sequence-layer from fp16 (n, 4, 256) device tensors
        (two launch_khq_compress_fp16 calls, K then V)."""
        n = k_unroped.shape[0]
        rows = n * H_KV
        tb, P = self.tables[layer], self.pay[layer]
        r0 = int(self.row_off[seq]) + tok0 * H_KV
        st = current_stream()
        rc = self.lib.launch_khq_compress_fp16(
            k_unroped.data_ptr(), tb["d_k"].data_ptr(), tb["k_rotor"].data_ptr(), tb["cents_k"].data_ptr(),
            tb["cents_k"].data_ptr(), P["k_mask"][r0 * 16:].data_ptr(), P["k_norms"][r0:].data_ptr(),
            P["k_r_norms"][r0:].data_ptr(), P["k_payload"][r0 * 40:].data_ptr(), P["v_shared_meta"][r0 * 4:].data_ptr(),
            rows, D, float(tb["ts_k"]), float(tb["alpha_k"]), 0, st)
        check("launch_khq_compress_fp16", rc)
        rc = self.lib.launch_khq_compress_fp16(
            v.data_ptr(), tb["d_v"].data_ptr(), tb["v_rotor"].data_ptr(), tb["cents_v"].data_ptr(),
            tb["vq"].data_ptr(), P["k_mask"][r0 * 16:].data_ptr(), P["v_norms"][r0:].data_ptr(),
            P["v_r_norms"][r0:].data_ptr(), P["v_payload"][r0 * 104:].data_ptr(), P["v_shared_meta"][r0 * 4:].data_ptr(),
            rows, D, float(tb["ts_v"]), float(tb["alpha_v"]), 1, st)
        check("launch_khq_compress_fp16", rc)

    def load_window(self, layer: int, seq: int, k_roped: torch.Tensor, v: torch.Tensor, k_unroped: Optional[torch.Tensor] = None) -> None:
        """Place the sequence's raw tokens (fp16 (win_len, 4, 256)) into the ring slots of its window."""
        ws, wl = int(self.boundary[seq] % RING), int(self.write_pos[seq] - self.boundary[seq])
        slots = (ws + torch.arange(wl, device=self.device)) % RING
        self.ring_k[layer][seq, slots] = k_roped.reshape(wl, KV)
        self.ring_v[layer][seq, slots] = v.reshape(wl, KV)
        self.ring_u[layer][seq, slots] = (k_unroped if k_unroped is not None else k_roped).reshape(wl, KV)

    def fill_synthetic(self, seed: int, chunk_tokens: int = 16384) -> None:
        """Seeded synthetic state: per layer and kv-head channel scales exp(0.5 N(0,1)) with four x8
        outlier channels; K/V ~ N(0, s_c); compressed with the library's own compress kernel."""
        g = torch.Generator(device=self.device)
        for l in range(self.L):
            g.manual_seed(seed + 17 * l)
            sc = torch.exp(0.5 * torch.randn(2, H_KV, D, generator=g, device=self.device))
            for h in range(H_KV):
                for kv in range(2):
                    idx = torch.randperm(D, generator=g, device=self.device)[:4]
                    sc[kv, h, idx] *= 8.0
            for i in range(self.B):
                n = int(self.boundary[i])
                for t0 in range(0, n, chunk_tokens):
                    m = min(chunk_tokens, n - t0)
                    k = (torch.randn(m, H_KV, D, generator=g, device=self.device) * sc[0]).half()
                    v = (torch.randn(m, H_KV, D, generator=g, device=self.device) * sc[1]).half()
                    self.compress_into(l, i, k, v, t0)
                wl = int(self.write_pos[i] - self.boundary[i])
                if wl:
                    k = (torch.randn(wl, H_KV, D, generator=g, device=self.device) * sc[0]).half()
                    v = (torch.randn(wl, H_KV, D, generator=g, device=self.device) * sc[1]).half()
                    self.load_window(l, i, k, v)
            self.q_gate[l].copy_(torch.randn(self.B, H_Q * 2 * D, generator=g, device=self.device).half())

    # ---------------------------------------------------------------------------------- stepping
    def attention_resident(self, layer: int, scale: float = 1.0 / 16.0) -> None:
        """The hot path alone: one batched attention launch for `layer` over the current state,
        inputs already in HBM."""
        rc = self.lib.launch_khq_decode_batched_prepared_fp16(
            self.d_descs.data_ptr() + layer * self.B * SEQ_DESC.itemsize, self.d_tables.data_ptr(), self._d_images.data_ptr(), self.d_items.data_ptr(),
            self.B, self.n_items, self.workspace.data_ptr(), self.ws_bytes, self.n_items, float(scale), self.rope_theta, RING,
            self._kernel if self._kernel >= 5 else int(self.codebook_in_smem), current_stream())  # the items' kernel
        check("launch_khq_decode_batched_prepared_fp16", rc)

    def _host_buffer(self, t, name: str):
        """``t`` if the native step can copy from or to it as it is, else the engine's own buffer of that name."""
        own = self._staging[name]
        plain = isinstance(t, torch.Tensor) and t.is_cpu and t.dtype is torch.float16 and t.numel() == own.numel() and t.is_contiguous()
        return t if plain else own

    def decode_step(self, scale: float = 1.0 / 16.0) -> torch.Tensor:
        """End-to-end token step from HOST buffers.  ``h_q`` (L, B, 24*512: query and gate halves, the
        query not yet normed or rotated), ``h_k`` and ``h_v`` (L, B, 4*256) hold this step's projections
        in pinned host memory.  Every sequence advances by one token: append, compression event if
        due, attention.  The gated outputs land in ``h_out`` (returned; valid once the stream has
        synchronised).  Any of the four may be replaced by another tensor between steps; what is not contiguous
        fp16 in host memory costs a wait and a copy."""
        parity = self._step & 1
        ctl, a, lib = self._ctl[parity], self._args, self.lib
        # the copy that last read this parity's host block has finished
        check("khq_b200_engine_wait_control", lib.khq_b200_engine_wait_control(self._native, parity))
        # ---- host state machine (src/khq/runtime.mojo:486-553, for every sequence) -----------------
        window = self.write_pos + 1 - self.boundary
        due = (window >= WATERMARK) & (self.boundary + CHUNK <= self.cap)
        n_ev = int(np.count_nonzero(due))
        if window.max() > RING and (window[~due] > RING).any():
            raise RuntimeError("a sequence's compressed capacity is exhausted (raise grow_tokens)")
        self._step += 1
        ctl["slots"][:] = self.write_pos % RING
        ctl["pos"][:] = self.write_pos
        self.write_pos += 1
        if n_ev:
            idx = np.nonzero(due)[0]
            at = self.boundary[idx]
            # the V launch reads ring_v at the same offsets from its own base
            ctl["segs"]["x"][:, :n_ev] = self._ring_u_at[:, None] + ((idx * RING + at % RING) * KV * 2).astype(np.uint64)
            ctl["segs"]["row0"][:, :n_ev] = self.row_off[idx] + at * H_KV
            self.boundary[idx] += CHUNK
            self.events_fired += n_ev
        self._plan(ctl)
        a.h_control, a.control_bytes, a.parity = ctl["block"].data_ptr(), self._control_bytes(n_ev), parity
        a.n_items, a.n_events, a.scale = self.n_items, n_ev, float(scale)
        a.codebook_in_smem, a.rms_eps = self._kernel, self.rms_eps
        if self.rope_theta != self._laid_out_theta:
            self.refresh_tables()
        given = dict(q=self.h_q, k=self.h_k, v=self.h_v, out=self.h_out)
        host = {n: self._host_buffer(t, n) for n, t in given.items()}
        for n in ("q", "k", "v"):
            if host[n] is not given[n]:
                torch.cuda.current_stream().synchronize()  # the step before has copied from the engine's buffer
                for l in range(self.L):
                    host[n][l].copy_(given[n][l])
        a.h_q, a.h_k, a.h_v, a.h_out = host["q"].data_ptr(), host["k"].data_ptr(), host["v"].data_ptr(), host["out"].data_ptr()
        self._in_flight.append(host)
        check("launch_khq_engine_step", lib.launch_khq_engine_step(self._native, self._layers, ctypes.addressof(a), current_stream()))
        if host["out"] is not given["out"]:
            torch.cuda.current_stream().synchronize()
            for l in range(self.L):
                given["out"][l].copy_(host["out"][l])
        return self.h_out
