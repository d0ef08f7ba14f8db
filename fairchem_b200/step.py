"""Whole-model evaluation from native code (csrc/model_step.cu): what the backbone and the energy head run by default.

One call issues every launch of the forward pass and one every launch of the backward pass; Python lays the weights out
once per model (``ModelPlan``), hands over the graph arrays and two memory blocks, and ties the result into autograd
(``BackboneStep``).  ``ModelPlan.of`` returns None for configurations the native path does not cover (other channel
counts, another contraction mode, a partitioned system); those run the per-op path of backbone.py.
"""

from __future__ import annotations

import ctypes
from ctypes import POINTER, Structure, byref, c_float, c_int32, c_int64, c_void_p

import torch

from . import _lib, ops

C = 128


class Weight(Structure):
    _fields_ = [("hi", c_void_p), ("lo", c_void_p), ("scale", c_float), ("rows", c_int32), ("cols", c_int32)]


class LayerStruct(Structure):
    _fields_ = ([(n, Weight * 3) for n in ("conv1", "conv1_t", "conv2", "conv2_t")]
                + [(n, Weight) for n in ("radial_out", "radial_out_t", "ffn_in", "ffn_in_t0", "ffn_in_t", "ffn_out", "ffn_out_t")]
                + [(n, c_void_p) for n in ("conv1_bias", "conv2_bias", "radial_out_bias", "ffn_in_bias", "ffn_out_bias", "norm1_w",
                                           "norm1_b", "norm2_w", "norm2_b")]
                + [("eps1", c_float), ("eps2", c_float)])


class ModelStruct(Structure):
    _fields_ = ([(n, c_int32) for n in ("lmax", "num_layers", "num_basis", "num_elements")]
                + [(n, c_float) for n in ("cutoff", "basis_start", "basis_stop", "basis_width", "rescale", "radial_eps", "norm_eps")]
                + [("layers", POINTER(LayerStruct))]
                + [(n, Weight) for n in ("rad_w0", "rad_w1", "rad_w1_t", "rad_w0_t")]
                + [(n, c_void_p) for n in ("rad_b0", "rad_b1", "ln1_w", "ln1_b", "ln2_w", "ln2_b", "table_src", "table_tgt")]
                + [(n, Weight) for n in ("degree_out", "degree_out_t")]
                + [(n, c_void_p) for n in ("degree_out_bias", "element_emb", "norm_w", "norm_b", "charge_emb", "spin_emb",
                                           "dataset_emb", "csd_w_t", "csd_b")]
                + [(n, Weight) for n in ("head_w1", "head_w1_t", "head_w2", "head_w2_t")]
                + [(n, c_void_p) for n in ("head_b1", "head_b2", "head_w3", "head_b3", "head_scale")])


class EvalStruct(Structure):
    _fields_ = ([("num_nodes", c_int64), ("num_edges", c_int64)]
                + [(n, c_int32) for n in ("num_systems", "num_chunks", "want_grad", "keep_radial")]
                + [(n, c_void_p) for n in ("pos", "shift", "gamma", "src", "tgt", "row_ptr", "src_ptr", "src_perm", "chunk_src", "z",
                                           "batch", "dataset", "charge", "spin", "chunk_node", "chunk_edge", "keep", "scratch", "x_out",
                                           "energy", "grad_x", "grad_pos")]
                + [("grad_sign", c_float), ("virial", c_void_p), ("status", c_void_p)])


def _versions(params) -> tuple:
    return tuple([p._version for p in params] + [p.data_ptr() for p in params])


class _Weights:
    """Half-split device copies of a module's matrices; keeps every tensor whose address is handed out alive."""

    def __init__(self):
        self.alive = []

    def ptr(self, t: torch.Tensor) -> int:
        t = t.detach().float().contiguous()
        self.alive.append(t)
        return t.data_ptr()

    def split(self, w: torch.Tensor) -> Weight:
        hi, lo, scale = ops.split_f16(w)
        self.alive += [hi, lo]
        return Weight(hi.data_ptr(), lo.data_ptr(), scale, w.shape[0], w.shape[1])


def _radial_nets(bb):
    return [b.edge_wise.so2_conv_1.rad_func for b in bb.blocks] + [bb.edge_degree_embedding.rad_func]


class ModelPlan:
    """Weights of one backbone in the layout of csrc/model_step.cu, rebuilt when a parameter changes."""

    def __init__(self, bb, params):
        from .backbone import _conv_weights

        self.params, self.versions = params, _versions(params)
        w = self.w = _Weights()
        self.device = params[0].device
        lmax, nb = bb.lmax, bb.num_distance_basis
        self.layers = (LayerStruct * bb.num_layers)()
        for s, blk in zip(self.layers, bb.blocks):
            ew, ff = blk.edge_wise, blk.atom_wise
            for name, conv in (("conv1", ew.so2_conv_1), ("conv2", ew.so2_conv_2)):
                mats = [m.detach() for m in _conv_weights(conv)]
                getattr(s, name)[:] = [w.split(m) for m in mats]
                getattr(s, name + "_t")[:] = [w.split(m.t().contiguous()) for m in mats]
                setattr(s, name + "_bias", w.ptr(conv.fc_m0.bias))
            out = ew.so2_conv_1.rad_func.net[6]
            s.radial_out, s.radial_out_t, s.radial_out_bias = w.split(out.weight), w.split(out.weight.t().contiguous()), w.ptr(out.bias)
            gate, w1, w2 = ff.scalar_mlp[0], ff.so3_linear_1, ff.so3_linear_2
            zeros = torch.zeros(lmax * C, device=self.device)
            s.ffn_in = w.split(torch.cat([gate.weight.detach(), *w1.weight.detach()]))
            s.ffn_in_bias = w.ptr(torch.cat([gate.bias.detach(), w1.bias.detach(), zeros]))
            s.ffn_in_t0 = w.split(torch.cat([gate.weight.detach(), w1.weight.detach()[0]]).t().contiguous())
            s.ffn_in_t = w.split(torch.cat([m.t() for m in w1.weight.detach()[1:]]))
            s.ffn_out = w.split(torch.cat([*w2.weight.detach()]))
            s.ffn_out_t = w.split(torch.cat([m.t() for m in w2.weight.detach()]))
            s.ffn_out_bias = w.ptr(torch.cat([w2.bias.detach(), zeros]))
            s.norm1_w, s.norm1_b = w.ptr(blk.norm_1.affine_weight), w.ptr(blk.norm_1.affine_bias)
            s.norm2_w, s.norm2_b = w.ptr(blk.norm_2.affine_weight), w.ptr(blk.norm_2.affine_bias)
            s.eps1, s.eps2 = blk.norm_1.eps, blk.norm_2.eps
        m = self.model = ModelStruct()
        m.lmax, m.num_layers, m.num_basis, m.num_elements = lmax, bb.num_layers, nb, bb.max_num_elements
        m.cutoff, m.basis_start, m.basis_stop, m.basis_width = bb.cutoff, 0.0, bb.cutoff, 2.0
        m.rescale, m.norm_eps = bb.rescale_factor, bb.norm.eps
        m.layers = self.layers
        nets = _radial_nets(bb)
        m.radial_eps = nets[0].net[1].eps
        w0 = torch.cat([n.net[0].weight.detach()[:, :nb] for n in nets])
        m.rad_w0, m.rad_w0_t = w.split(w0), w.split(w0.t().contiguous())
        m.rad_w1 = w.split(torch.cat([n.net[3].weight.detach() for n in nets]))
        m.rad_w1_t = w.split(torch.cat([n.net[3].weight.detach().t() for n in nets]))
        for name, mod, attr in (("rad_b0", 0, "bias"), ("rad_b1", 3, "bias"), ("ln1_w", 1, "weight"), ("ln1_b", 1, "bias"),
                                ("ln2_w", 4, "weight"), ("ln2_b", 4, "bias")):
            setattr(m, name, w.ptr(torch.cat([getattr(n.net[mod], attr).detach() for n in nets])))
        tables = [bb._tables(n) for n in nets]
        m.table_src, m.table_tgt = w.ptr(torch.cat([t[0] for t in tables], 1)), w.ptr(torch.cat([t[1] for t in tables], 1))
        out = nets[-1].net[6]
        m.degree_out, m.degree_out_t, m.degree_out_bias = w.split(out.weight), w.split(out.weight.t().contiguous()), w.ptr(out.bias)
        m.element_emb, m.norm_w, m.norm_b = w.ptr(bb.sphere_embedding.weight), w.ptr(bb.norm.affine_weight), w.ptr(bb.norm.affine_bias)
        m.charge_emb, m.spin_emb = w.ptr(bb.charge_embedding.rand_emb.weight), w.ptr(bb.spin_embedding.rand_emb.weight)
        emb = bb.dataset_embedding.dataset_emb_dict
        self.dataset_row = {name: i for i, name in enumerate(emb)}
        m.dataset_emb = w.ptr(torch.cat([e.weight for e in emb.values()]))
        m.csd_w_t, m.csd_b = w.ptr(bb.mix_csd.weight.t()), w.ptr(bb.mix_csd.bias)
        self.dataset_ids = {}  # (names) -> int32 device tensor of their rows, for batches of one dataset

    @staticmethod
    def supported(bb) -> bool:
        from .backbone import _GemmState

        nets = _radial_nets(bb)
        return (_GemmState.precision == 2 and _GemmState.fused_conv and _GemmState.native and not ops.generic_kernels()
                and ops.CONV_VARIANT == -1 and bb.keep_level is None and bb.sphere_channels == C and bb.hidden_channels == C
                and bb.edge_channels == C and bb.num_distance_basis % 32 == 0 and 1 <= bb.num_layers < 40
                and all(len(n.net) == 7 and n.net[1].eps == n.net[4].eps == nets[0].net[1].eps for n in nets))

    @classmethod
    def of(cls, bb):
        """The backbone's plan, or None when the native path does not apply."""
        if not cls.supported(bb):
            return None
        plan = getattr(bb, "_step_plan", None)
        if plan is not None and plan.versions == _versions(plan.params):
            return plan
        params = list(bb.parameters())
        if not params[0].is_cuda or any(p.dtype != torch.float32 for p in params):
            return None
        bb._step_plan = plan = cls(bb, params)
        return plan

    def with_head(self, head):
        """The model struct with the energy head's weights filled in (cached on the head), or None."""
        eb = head.energy_block
        params = list(eb.parameters())
        key = (id(self), _versions(params))
        hit = getattr(head, "_step_model", None)
        if hit is not None and hit[0] == key:
            return hit[1]
        if eb[0].weight.shape != (C, C) or eb[2].weight.shape != (C, C) or eb[4].weight.shape != (1, C):
            return None
        w, m = _Weights(), ModelStruct()
        ctypes.pointer(m)[0] = self.model
        m.head_w1, m.head_w1_t = w.split(eb[0].weight), w.split(eb[0].weight.detach().t().contiguous())
        m.head_w2, m.head_w2_t = w.split(eb[2].weight), w.split(eb[2].weight.detach().t().contiguous())
        m.head_b1, m.head_b2, m.head_w3, m.head_b3 = w.ptr(eb[0].bias), w.ptr(eb[2].bias), w.ptr(eb[4].weight), w.ptr(eb[4].bias)
        from .backbone import _pow2_scale

        m.head_scale = w.ptr(_pow2_scale(eb[4].weight.detach().abs().max() * 1.1))  # |d silu| <= 1.1
        head._step_model = (key, m, w, self)
        return m

    def dataset_index(self, bb, names) -> torch.Tensor:
        key = names[0] if all(n == names[0] for n in names) else None
        if key is not None:
            hit = self.dataset_ids.get((key, len(names)))
            if hit is not None:
                return hit
        idx = torch.tensor([self.dataset_row[bb.dataset_embedding.mapping[n]] for n in names], dtype=torch.int32, device=self.device)
        if key is not None and len(self.dataset_ids) < 64:
            self.dataset_ids[(key, len(names))] = idx
        return idx


def _stream():
    return c_void_p(torch.cuda.current_stream().cuda_stream)


class BackboneStep:
    """One evaluation: graph arrays, outputs and the memory that the backward pass reads."""

    def __init__(self, plan: ModelPlan, pos, graph, z, batch, dataset, charge, spin, shift, gamma, num_systems: int, want_grad: bool,
                 want_virial: bool, status):
        self.plan, self.model = plan, plan.model
        dev = pos.device
        self.nodes, self.systems = pos.shape[0], num_systems
        e = self.ev = EvalStruct()
        e.num_nodes, e.num_edges, e.num_systems = self.nodes, graph.num_edges, num_systems
        e.num_chunks, e.want_grad = graph.num_chunks, int(want_grad)
        self.refs = [pos, graph, z, batch, dataset, charge, spin, shift, gamma, status]
        e.pos, e.z, e.batch, e.dataset = pos.data_ptr(), z.data_ptr(), batch.data_ptr(), dataset.data_ptr()
        e.charge, e.spin, e.status = charge.data_ptr(), spin.data_ptr(), status.data_ptr()
        e.shift = None if shift is None else shift.data_ptr()
        e.gamma = None if gamma is None else gamma.data_ptr()
        e.src, e.tgt, e.row_ptr = graph.src.data_ptr(), graph.tgt.data_ptr(), graph.row_ptr.data_ptr()
        e.src_ptr, e.src_perm = graph.src_ptr.data_ptr(), graph.src_perm.data_ptr()
        e.chunk_src = None if graph.chunk_src is None else graph.chunk_src.data_ptr()
        e.chunk_node, e.chunk_edge = ctypes.cast(graph.chunk_node, c_void_p), ctypes.cast(graph.chunk_edge, c_void_p)
        self.want_virial = want_virial
        self.virial = None
        self.device = dev
        self.sizes = (c_int64 * 3)()
        self.keep = self.scratch = None

    def plan_memory(self) -> bool:
        """Decide whether the radial weights are kept too; False when the kept tensors do not fit the free memory."""
        e, sizes = self.ev, self.sizes
        for keep_radial in (1, 0) if e.want_grad else (0,):
            e.keep_radial = keep_radial
            _lib.call("fcb200_model_sizes", byref(self.model), byref(e), sizes)
            need = sizes[0] + max(sizes[1], sizes[2] if e.want_grad else 0)
            if need < (1 << 30):  # what any free GPU has; spares the memory query of small systems
                return True
            if not hasattr(self, "avail"):
                free, self.total = torch.cuda.mem_get_info(self.device)
                self.avail = free + torch.cuda.memory_reserved(self.device) - torch.cuda.memory_allocated(self.device)
            # the largest kept set only with room to spare
            if need * (1.15 if keep_radial else 1.0) + 0.03 * self.total < self.avail:
                return True
        return False

    def _block(self, nbytes: int) -> torch.Tensor:
        return torch.empty(nbytes, dtype=torch.uint8, device=self.device)

    def forward(self) -> torch.Tensor:
        e = self.ev
        self.keep = self._block(self.sizes[0])
        scratch = self._block(self.sizes[1])
        nl = (self.model.lmax + 1) ** 2
        x = torch.empty(self.nodes, nl, C, dtype=torch.float32, device=self.device)
        e.keep, e.scratch, e.x_out = self.keep.data_ptr(), scratch.data_ptr(), x.data_ptr()
        _lib.call("fcb200_model_forward", byref(self.model), byref(e), _stream())
        return x

    def energy(self, model: ModelStruct) -> torch.Tensor:
        out = torch.zeros(self.systems, dtype=torch.float64, device=self.device)
        self.ev.energy = out.data_ptr()
        _lib.call("fcb200_model_energy", byref(model), byref(self.ev), _stream())
        return out

    def backward(self, model: ModelStruct, grad_x, sign: float) -> torch.Tensor:
        """sign * gradient of the energy sum (grad_x None) or of <grad_x, node embedding> with respect to the positions."""
        if self.keep is None:
            raise RuntimeError("fairchem_b200: this evaluation's buffers were released by an earlier backward pass")
        e = self.ev
        scratch = self._block(self.sizes[2])
        grad = torch.empty(self.nodes, 3, dtype=torch.float32, device=self.device)
        e.scratch, e.grad_pos, e.grad_sign = scratch.data_ptr(), grad.data_ptr(), sign
        e.grad_x = None if grad_x is None else grad_x.data_ptr()
        if self.want_virial:
            v = torch.zeros(self.systems, 3, 3, dtype=torch.float64, device=self.device)
            e.virial = v.data_ptr()
            self.virial["virial"] = v
        _lib.call("fcb200_model_backward", byref(model), byref(e), _stream())
        self.keep = None
        return grad


class BackboneFn(torch.autograd.Function):
    """Node embedding as a function of the positions."""

    @staticmethod
    def forward(ctx, pos, step: BackboneStep):
        ctx.step = step
        return step.forward()

    @staticmethod
    def backward(ctx, grad_x):
        return ctx.step.backward(ctx.step.model, grad_x.contiguous(), 1.0), None


class StepGraph:
    """Index arrays of one edge list (sorted by target) for the native evaluation."""

    @classmethod
    def from_edges(cls, src, tgt, num_nodes: int, chunk_edges: int):
        g = ops.EdgeGraph(src, tgt, num_nodes)
        self = cls()
        self.src, self.tgt, self.row_ptr, self.src_ptr, self.src_perm = g.src, g.tgt, g.row_ptr, g.src_ptr, g.src_perm
        e = self.num_edges = g.num_edges
        n = self.num_chunks = max(1, (e + chunk_edges // 2) // chunk_edges)
        cut = torch.searchsorted(g.row_ptr, torch.arange(1, n, device=src.device, dtype=torch.int32) * (e // n)) if n > 1 else None
        nodes = [0] + ([] if cut is None else cut.tolist()) + [num_nodes]
        nodes = sorted(set(nodes))
        n = self.num_chunks = len(nodes) - 1
        edges = [0] + ([] if n == 1 else g.row_ptr[torch.tensor(nodes[1:-1], device=src.device)].tolist()) + [e]
        self.chunk_node, self.chunk_edge = (c_int64 * (n + 1))(*nodes), (c_int64 * (n + 1))(*edges)
        self.chunk_src = None
        if n > 1:
            key = g.src.long()[g.src_perm.long()] * e + g.src_perm.long()
            want = torch.arange(num_nodes, device=src.device)[None] * e + torch.tensor(edges, device=src.device)[:, None]
            self.chunk_src = torch.searchsorted(key, want).to(torch.int32).contiguous()
        return self
