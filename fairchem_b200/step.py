"""Whole-model evaluation from native code (csrc/model_step.cu): what the backbone and the energy head run by default.

One call issues every launch of the forward pass and one every launch of the backward pass; Python lays the weights out
once per model (``ModelPlan``), hands over the graph arrays and two memory blocks, and ties the result into autograd
(``BackboneStep``).  ``ModelPlan.of`` returns None for configurations the native path does not cover (other channel
counts, another contraction mode, a partitioned system); those run the per-op path of backbone.py.
"""

from __future__ import annotations

import ctypes
import operator
from ctypes import POINTER, Structure, byref, c_float, c_int32, c_int64, c_void_p
from itertools import chain
from typing import Optional

import torch
import torch.nn.modules.module as _nn_module

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
                + [(n, c_int32) for n in ("num_systems", "num_chunks", "want_grad", "keep_radial", "drop_layers")]
                + [(n, c_void_p) for n in ("pos", "shift", "gamma", "src", "tgt", "row_ptr", "src_ptr", "src_perm", "chunk_src", "z",
                                           "batch", "dataset", "charge", "spin", "chunk_node", "chunk_edge", "keep", "scratch", "x_out",
                                           "energy", "grad_x", "grad_pos")]
                + [("grad_sign", c_float), ("virial", c_void_p), ("status", c_void_p)])


_VERSION = operator.attrgetter("_version")
_EPS = operator.attrgetter("eps")
_SCALARS = operator.attrgetter("lmax", "num_distance_basis", "max_num_elements", "cutoff", "rescale_factor", "sphere_channels",
                               "hidden_channels", "edge_channels", "charge_embedding.offset", "spin_embedding.offset")


def _versions(params) -> list:
    return [*map(_VERSION, params), *map(torch.Tensor.data_ptr, params)]


class _Origin:
    """What a plan was laid out from: every submodule and parameter a backbone holds, the parameters' versions and
    addresses, and the plain numbers that went into the plan.  The objects are looked up again on each call, because an
    assigned parameter (``load_state_dict(assign=True)``, ``functional_call``, ``module.weight = ...``) leaves the old
    one as it was.  45 us for four layers with the hooks below, spent while the launches of the forward pass run (in front of
    them a molecule of 21 atoms took 1366 us, so 1314)."""

    def __init__(self, bb):
        mods = list(bb.modules())
        self.views = [m._modules.values() for m in mods if m._modules] + [m._parameters.values() for m in mods if m._parameters]
        self.eps_of = [m for m in mods if hasattr(m, "eps")]
        self.objects = self._objects()
        self.params = [o for o in self.objects if isinstance(o, torch.Tensor)]
        self.versions, self.scalars = _versions(self.params), self._scalars(bb)

    def _objects(self) -> list:
        return [*chain.from_iterable(self.views)]

    def _scalars(self, bb) -> list:
        return [*_SCALARS(bb), *map(_EPS, self.eps_of)]

    def unchanged(self, bb) -> bool:
        now = self._objects()
        return (len(now) == len(self.objects) and all(map(operator.is_, now, self.objects))
                and self.versions == _versions(self.params) and self.scalars == self._scalars(bb))


def structure_of(bb) -> tuple:
    """Module types and parameter shapes by name."""
    return ({n: type(m) for n, m in bb.named_modules(remove_duplicate=False) if n},
            {n: p.shape for n, p in bb.named_parameters(remove_duplicate=False)})


_METHODS = ("csd_embedding", "_tables", "_graph")  # what the native evaluation does in their place
_HOOK_DICTS = ("_forward_hooks", "_forward_pre_hooks", "_backward_hooks", "_backward_pre_hooks")
_GLOBAL_HOOKS = [getattr(_nn_module, "_global" + n) for n in _HOOK_DICTS]


class _Calls:
    """The submodules that the per-op path calls as modules, and the hooks it would run.  A hook, or a forward of an
    instance's own, sends an evaluation down that path."""

    def __init__(self, bb):
        mods = [bb.norm, bb.sphere_embedding, bb.charge_embedding, bb.charge_embedding.rand_emb, bb.spin_embedding,
                bb.spin_embedding.rand_emb, bb.dataset_embedding, bb.mix_csd]
        for blk in bb.blocks:
            mods += [blk.norm_1, blk.norm_2, blk.atom_wise, blk.atom_wise.so3_linear_1, blk.atom_wise.so3_linear_2]
        self.hooks = [*_GLOBAL_HOOKS, *(getattr(m, n) for m in mods for n in _HOOK_DICTS)]
        self.attributes = [m.__dict__ for m in mods]

    def watched(self, bb) -> bool:  # the backbone is passed in: held here it would be a cycle through its own plan
        return any(map(len, self.hooks)) or any("forward" in d for d in self.attributes) or any(n in bb.__dict__ for n in _METHODS)


class _Weights:
    """Half-split device copies of a module's matrices; keeps every tensor whose address is handed out alive.

    They are written on the stream that was current then.  Another stream waits for that before its first use, and the
    memory goes back only behind what other streams were still doing with it."""

    def __init__(self, device):
        self.alive = []
        self.device, self.home, self.ready, self.last_use = device, torch.cuda.current_stream(device), None, {}

    def laid_out(self):
        self.ready = self.home.record_event()

    def before_use(self, stream):
        if stream.cuda_stream not in self.last_use:
            stream.wait_event(self.ready)

    def after_use(self, stream):
        self.last_use[stream.cuda_stream] = stream.record_event(self.last_use.get(stream.cuda_stream))

    def __del__(self):
        for event in self.last_use.values():
            self.home.wait_event(event)

    def ptr(self, t: torch.Tensor) -> int:
        t = t.detach().float().contiguous()
        self.alive.append(t)
        return t.data_ptr()

    def split(self, w: torch.Tensor) -> Weight:
        hi, lo, scale = ops.split_f16(w)
        self.alive += [hi, lo]
        return Weight(hi.data_ptr(), lo.data_ptr(), scale, w.shape[0], w.shape[1])


class HoldsPlan:
    """Mixin of the modules that keep a plan (``_step_plan``): device addresses of their own weights, which neither a copy nor
    a file of the module may carry.  Both lay out their own when they are first used."""

    def __getstate__(self):
        return {k: v for k, v in self.__dict__.items() if k != "_step_plan"}


def _radial_nets(bb):
    return [b.edge_wise.so2_conv_1.rad_func for b in bb.blocks] + [bb.edge_degree_embedding.rad_func]


class ModelPlan:
    """Weights of one backbone in the layout of csrc/model_step.cu, rebuilt when anything they were read from changes."""

    def __init__(self, bb, origin: _Origin):
        from .backbone import _conv_weights

        self.origin, self.calls, self.in_doubt = origin, _Calls(bb), False
        self.device = origin.params[0].device
        w = self.w = _Weights(self.device)
        lmax, nb = bb.lmax, bb.num_distance_basis
        self.layers = (LayerStruct * len(bb.blocks))()
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
        m.lmax, m.num_layers, m.num_basis, m.num_elements = lmax, len(bb.blocks), nb, bb.max_num_elements
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
        self.datasets = list(emb)
        self.dataset_row = {name: i for i, name in enumerate(emb)}
        m.dataset_emb = w.ptr(torch.cat([e.weight for e in emb.values()]))
        m.csd_w_t, m.csd_b = w.ptr(bb.mix_csd.weight.t()), w.ptr(bb.mix_csd.bias)
        w.laid_out()
        self.dataset_ids = {}  # (row, systems) -> int32 device tensor, for batches of one dataset

    @staticmethod
    def supported(bb) -> bool:
        """Shapes that csrc/model_step.cu is written for, of the modules and methods that it stands for."""
        from .backbone import eSCNMDBackboneB200 as plain

        if not (bb.sphere_channels == C and bb.hidden_channels == C and bb.edge_channels == C and bb.num_distance_basis % 32 == 0
                and (bb.charge_embedding.offset, bb.spin_embedding.offset) == (100, 0)  # as csrc/node_step.cuh indexes the tables
                and 1 <= len(bb.blocks) < 40 and all(getattr(type(bb), n) is getattr(plain, n) for n in _METHODS)):
            return False
        nets = _radial_nets(bb)
        return (bb.__dict__.get("_built_as") in (None, structure_of(bb))
                and all(n.net[1].eps == n.net[4].eps == nets[0].net[1].eps for n in nets))

    @staticmethod
    def wanted(bb) -> bool:
        from .backbone import _GemmState as mode

        return (mode.precision == 2 and mode.fused_conv and mode.native and bb.keep_level is None
                and not ops.generic_kernels())

    @classmethod
    def likely(cls, bb, device):
        """The plan of the last evaluation, for the caller to begin with: ``of`` says afterwards whether it still holds.  One
        that did not hold the last time, or that could not even be launched with these inputs, is checked at once."""
        if not cls.wanted(bb):
            return None
        plan = bb.__dict__.get("_step_plan")
        if plan is None or plan.in_doubt or plan.device != device or plan.datasets != list(bb.dataset_embedding.dataset_emb_dict):
            return cls.of(bb)
        return plan

    @classmethod
    def of(cls, bb):
        """The backbone's plan, or None when the native path does not apply."""
        if not cls.wanted(bb):
            return None
        plan = bb.__dict__.get("_step_plan")
        if plan is None or not plan.origin.unchanged(bb):
            if plan is not None:
                plan.in_doubt = True
            origin = _Origin(bb)
            if not cls.supported(bb) or not origin.params[0].is_cuda or any(p.dtype != torch.float32 for p in origin.params):
                return None
            bb._step_plan = plan = cls(bb, origin)
        plan.in_doubt = plan.calls.watched(bb)
        return None if plan.in_doubt else plan

    def with_head(self, head) -> Optional["HeadPlan"]:
        """This plan with the energy head's weights (cached on the head), or None."""
        eb = head.energy_block
        params = [p for i in (0, 2, 4) for p in (eb[i].weight, eb[i].bias)]
        if any(p is None for p in params):
            return None
        key = _versions(params)
        hit = getattr(head, "_step_plan", None)
        if hit is not None and hit.backbone is self and hit.key == key:
            return hit
        if eb[0].weight.shape != (C, C) or eb[2].weight.shape != (C, C) or eb[4].weight.shape != (1, C):
            return None
        if any(p.device != self.device or p.dtype != torch.float32 for p in params):
            return None
        head._step_plan = hit = HeadPlan(self, eb, key)
        return hit

    def dataset_index(self, bb, names) -> torch.Tensor:
        mapping, key = bb.dataset_embedding.mapping, None
        if all(n == names[0] for n in names):
            rows = [self.dataset_row[mapping[names[0]]]] * len(names)
            key = (rows[0], len(names))
        else:
            rows = [self.dataset_row[mapping[n]] for n in names]
        idx = self.dataset_ids.get(key)
        if idx is None:
            idx = torch.tensor(rows, dtype=torch.int32, device=self.device)
            if key is not None and len(self.dataset_ids) < 64:
                self.dataset_ids[key] = idx
                self.w.alive.append(idx)
        return idx


class HeadPlan:
    """A backbone's plan with an energy head's weights filled in."""

    def __init__(self, backbone: ModelPlan, eb, key):
        from .backbone import _pow2_scale

        self.backbone, self.key = backbone, key
        w, m = self.w, self.model = _Weights(backbone.device), ModelStruct()
        ctypes.pointer(m)[0] = backbone.model
        m.head_w1, m.head_w1_t = w.split(eb[0].weight), w.split(eb[0].weight.detach().t().contiguous())
        m.head_w2, m.head_w2_t = w.split(eb[2].weight), w.split(eb[2].weight.detach().t().contiguous())
        m.head_b1, m.head_b2, m.head_w3, m.head_b3 = w.ptr(eb[0].bias), w.ptr(eb[2].bias), w.ptr(eb[4].weight), w.ptr(eb[4].bias)
        m.head_scale = w.ptr(_pow2_scale(eb[4].weight.detach().abs().max() * 1.1))  # |d silu| <= 1.1
        w.laid_out()


def _stream():
    return c_void_p(torch.cuda.current_stream(torch.cuda.current_device()).cuda_stream)  # an index: 2 us, no argument 18


ALWAYS_THERE = 1 << 28  # bytes that any GPU in use has; more: what the allocator already holds, or the driver is asked


class BackboneStep:
    """One evaluation: graph arrays, outputs and the memory that the backward pass reads."""

    def __init__(self, plan: ModelPlan, graph: "StepGraph", dataset, gamma, want_virial: bool, status):
        self.plan, self.model = plan, plan.model
        self.nodes, self.systems, self.device = graph.nodes, graph.systems, graph.device
        e, g = EvalStruct(), graph.g
        self.ev = e
        e.num_nodes, e.num_systems, e.want_grad = self.nodes, self.systems, int(graph.want_grad)
        if dataset.numel() != self.systems:
            raise ValueError(f"dataset has {dataset.numel()} entries, expected {self.systems}")
        gamma = None if gamma is None or gamma.numel() == 0 else gamma.contiguous()
        ops._chk(gamma)
        ops._f32(gamma)
        self.gamma = gamma
        self.leaf, self.graph = graph.leaf, graph
        self.refs = [t for t in (dataset, gamma, status, *graph.alive) if t is not None]
        self.watched = [t for t in (graph.pos, graph.charge, graph.spin, gamma) if t is not None]  # may be the caller's own memory
        for name in ("pos", "z", "batch", "src", "tgt", "row_ptr", "src_ptr", "src_perm"):
            setattr(e, name, getattr(g, name))
        e.shift, e.dataset, e.charge, e.spin = graph.shift, dataset.data_ptr(), g.charge, g.spin
        e.gamma = None if gamma is None else gamma.data_ptr()
        e.status = status.data_ptr()
        self.want_virial, self.virial = want_virial, None
        self.sizes = (c_int64 * 3)()
        self.keep = self.home = None
        self.spent = False  # the head has computed the forces

    def set_edges(self, graph: "StepGraph"):
        e = self.ev
        if self.gamma is not None and self.gamma.numel() != graph.num_edges:
            raise ValueError(f"gamma has {self.gamma.numel()} entries for {graph.num_edges} edges")
        e.num_edges, e.num_chunks = graph.num_edges, graph.num_chunks
        e.chunk_src = graph.g.chunk_src if graph.num_chunks > 1 else None
        e.chunk_node, e.chunk_edge = ctypes.addressof(graph.chunk_node), ctypes.addressof(graph.chunk_edge)

    def plan_memory(self) -> bool:
        """Decide what is kept for the backward pass: everything with the gated rows as half planes (1), everything with them
        in float32 (2), all but the radial weights (0), or, layer by layer, no conv-1 output and messages either.  False when not even the smallest set fits the free memory.

        All but the first give the same bits; in the first the gate's gradient is made from half planes, and forces differ by
        some 2e-7 of their norm from those.  So near the limit of the first set two calls on one system
        agree to that, not bit for bit, when other allocations come or go between them."""
        e, sizes, layers = self.ev, self.sizes, self.model.num_layers
        for keep_radial, drop in chain(((1, 0), (2, 0)), ((0, n) for n in range(layers + 1))) if e.want_grad else ((0, 0),):
            e.keep_radial, e.drop_layers = keep_radial, drop
            _lib.call("fcb200_model_sizes", byref(self.model), byref(e), sizes)
            need = sizes[0] + max(sizes[1], sizes[2] if e.want_grad else 0)
            if need < ALWAYS_THERE or need < self._cached():
                return True
            if not hasattr(self, "avail"):
                free, self.total = torch.cuda.mem_get_info(self.device)
                self.avail = free + self._cached()
            # the radial weights only with room to spare
            if need * (1.15 if keep_radial else 1.0) + 0.03 * self.total < self.avail:
                return True
        return False

    def _cached(self) -> int:
        """Bytes the caching allocator holds and does not use.  Asking the driver for free memory instead takes
        10-40 ms now and then, so that is left to evaluations that need more than this."""
        stats = torch._C._cuda_memoryStats(self.device.index)
        return stats["reserved_bytes"]["all"]["current"] - stats["allocated_bytes"]["all"]["current"]

    def _block(self, nbytes: int) -> torch.Tensor:
        return torch.empty(nbytes, dtype=torch.uint8, device=self.device)

    def forward(self) -> torch.Tensor:
        if self.ev.want_grad:  # tensors of inference mode have no versions, and no second backward pass either
            self.inputs = [(t, t._version) for t in self.watched if not t.is_inference()]
        return self._forward()

    def _launch(self, name: str, *plans):
        """One native call on the current stream, which need not be the one that the evaluation began on."""
        stream = torch.cuda.current_stream(self.device.index)
        if self.home is None:
            self.home = stream
        elif stream.cuda_stream != self.home.cuda_stream:
            stream.wait_stream(self.home)
            for t in (self.keep, self.graph.a.block, self.graph.b.block, *self.refs):
                t.record_stream(stream)
        foreign = [p.w for p in plans if p.w.home.cuda_stream != stream.cuda_stream]
        for w in foreign:
            w.before_use(stream)
        _lib.call(name, byref(plans[-1].model), byref(self.ev), c_void_p(stream.cuda_stream))
        for w in foreign:
            w.after_use(stream)

    def _forward(self) -> torch.Tensor:
        e = self.ev
        self.keep = self._block(self.sizes[0])
        scratch = self._block(self.sizes[1])
        nl = (self.model.lmax + 1) ** 2
        x = torch.empty(self.nodes, nl, C, dtype=torch.float32, device=self.device)
        e.keep, e.scratch, e.x_out = self.keep.data_ptr(), scratch.data_ptr(), x.data_ptr()
        self._launch("fcb200_model_forward", self.plan)
        return x

    def energy(self, head: HeadPlan) -> torch.Tensor:
        out = torch.zeros(self.systems, dtype=torch.float64, device=self.device)
        self.ev.energy = out.data_ptr()
        self._launch("fcb200_model_energy", self.plan, head)
        return out

    def backward(self, head: Optional[HeadPlan], grad_x, sign: float) -> torch.Tensor:
        """sign * gradient of the energy sum (grad_x None) or of <grad_x, node embedding> with respect to the positions."""
        if self.keep is None:  # released by an earlier backward pass over a retained graph: computed again
            if any(t._version != v for t, v in self.inputs):
                raise RuntimeError("fairchem_b200: an input of this evaluation was modified in place after its first backward pass")
            self._forward()
        e = self.ev
        scratch = self._block(self.sizes[2])
        grad = torch.empty(self.nodes, 3, dtype=torch.float32, device=self.device)
        e.scratch, e.grad_pos, e.grad_sign = scratch.data_ptr(), grad.data_ptr(), sign
        e.grad_x = None if grad_x is None else grad_x.data_ptr()
        if self.want_virial:
            v = torch.zeros(self.systems, 3, 3, dtype=torch.float64, device=self.device)
            e.virial = v.data_ptr()
            self.virial["virial"] = v
        self._launch("fcb200_model_backward", self.plan, *([] if head is None else [head]))
        self.keep = None
        return grad


class BackboneFn(torch.autograd.Function):
    """Node embedding as a function of the positions."""

    @staticmethod
    def forward(ctx, pos, step: BackboneStep):
        ctx.step = step
        ctx.save_for_backward(pos)
        return step.forward()

    @staticmethod
    def backward(ctx, grad_x):
        ctx.saved_tensors  # raises autograd's own error for a graph that was not retained, or positions modified since
        step = ctx.step
        if step.spent:  # the head took its gradient from this evaluation without autograd and did not retain it
            raise RuntimeError("fairchem_b200: the forces of this evaluation were computed already; its graph was not retained")
        return step.backward(None, grad_x.contiguous(), 1.0), None


class GraphStruct(Structure):
    _fields_ = ([("num_nodes", c_int64)]
                + [(n, c_int32) for n in ("num_systems", "num_elements", "max_neighbors", "stride", "chunk_edges", "want_totals")]
                + [("radius", c_float), ("radius_sq", c_float)]
                + [(n, c_void_p) for n in ("pos", "cell", "pbc", "natoms", "batch64", "z64", "charge", "spin", "sys", "bbox", "z", "batch",
                                           "rows", "count", "row_ptr", "info")]
                + [("num_sources", c_int64), ("num_cells", c_int64)]
                + [(n, c_void_p) for n in ("cell_count", "source_cell", "cell_ptr", "cell_fill", "bucket", "cand_ptr", "cand_id",
                                           "cand_sys", "pos0", "cell0", "pbc0", "natoms0")]
                + [("limit_sq", c_float), ("num_chunks", c_int32), ("num_edges", c_int64)]
                + [(n, c_void_p) for n in ("src", "tgt", "shift", "edge_index", "cell_offsets", "src_count", "src_ptr", "src_tmp",
                                           "src_perm", "chunk_src")])


INFO_WORDS, INFO_INPUT, INFO_NODES, INFO_EDGES = 1040, 7, 8, 8 + 513
INPUT_ERRORS = ((1, "atomic number outside the embedding table"), (2, "system index (batch) outside the batch"),
                (4, "charge outside [-100, 100]"), (8, "spin outside [0, 100]"))
STRIDE_MAX = 512     # kept neighbours of one target that graph_select_kernel can hold
BRUTE_NODES = 8192   # below: every periodic image in reach is tried, no grid and no host read to size one
BRUTE_PAIRS = 4e9    # above that, still the faster way while the systems of a batch are small


class _Carve:
    """Sub-arrays of one int32 allocation, 256-byte aligned."""

    def __init__(self, device, **sizes):
        offsets, total = {}, 0
        for name, n in sizes.items():
            offsets[name] = total
            total += (n + 63) // 64 * 64
        self.block = torch.empty(total, dtype=torch.int32, device=device)
        base = self.block.data_ptr()
        self.ptr = {name: base + 4 * o for name, o in offsets.items()}
        self.offsets = offsets

    def view(self, name: str, n: int) -> torch.Tensor:
        return self.block[self.offsets[name]:self.offsets[name] + n]


class StepGraph:
    """Index arrays of one evaluation for csrc/model_step.cu (edges sorted by target; ``None`` from ``build`` when the
    general path has to decide: too many neighbours, a degenerate cell)."""

    def __init__(self, bb, data, want_grad: bool):
        self.bb, self.data, self.want_grad = bb, data, want_grad
        pos = self.pos = data["pos"].detach().contiguous()
        self.leaf = data["pos"]
        self.device, self.nodes, self.systems = pos.device, pos.shape[0], len(data["natoms"])
        n, b = self.nodes, self.systems
        if pos.dim() != 2 or pos.shape[1] != 3:
            raise ValueError(f"positions of shape {tuple(pos.shape)}, expected [atoms, 3]")
        for key, want in (("batch", n), ("atomic_numbers", n), ("cell", 9 * b), ("charge", b), ("spin", b)):
            if data[key].numel() != want:  # the kernels read as many
                raise ValueError(f"{key} has {data[key].numel()} entries, expected {want} for {n} atoms in {b} systems")
        self.a = _Carve(self.device, sys=b * 24, bbox=b * 6, z=n, batch=n, count=n, row_ptr=n + 1, info=INFO_WORDS)
        g = self.g = GraphStruct()
        g.num_nodes, g.num_systems, g.num_elements = n, b, bb.max_num_elements
        g.max_neighbors, g.chunk_edges = int(bb.max_neighbors), bb.edge_chunk_size
        g.radius, g.radius_sq = bb.cutoff, bb.cutoff * bb.cutoff
        pbc = data["pbc"] if data["pbc"].dtype == torch.bool else data["pbc"].bool()
        cell = data["cell"].detach().to(torch.float32)
        self.alive = [cell.contiguous(), pbc.contiguous(),
                      *(data[k].long().contiguous() for k in ("natoms", "batch", "atomic_numbers", "charge", "spin"))]
        if any(t.device != self.device for t in self.alive):  # small host tensors next to device positions
            self.alive = [t.to(self.device) for t in self.alive]
        if self.alive[1].numel() != 3 * b:
            self.alive[1] = self.alive[1].reshape(-1, 3).expand(b, 3).contiguous()
        g.pos = pos.data_ptr()
        g.cell, g.pbc, g.natoms, g.batch64, g.z64, g.charge, g.spin = (t.data_ptr() for t in self.alive)
        self.charge, self.spin = self.alive[-2:]
        for name, p in self.a.ptr.items():
            setattr(g, name, p)
        self.chunk_src = self.edge_index = self.cell_offsets = self.shift = None
        self.pending = False

    def _call(self, name):
        _lib.call(name, byref(self.g), _stream())

    def _info(self, words: int = INFO_WORDS):
        """The info block on the host, in which the kernels have noted inputs that the model has no embedding for."""
        info = self.a.view("info", words).cpu()
        self._refuse(int(info[INFO_INPUT]))
        return info

    @staticmethod
    def _refuse(bits: int):
        if bits:
            raise ValueError(", ".join(what for bit, what in INPUT_ERRORS if bits & bit))

    def check_inputs(self):
        """Before other code indexes by them: raise for inputs outside the tables."""
        self._call("fcb200_graph_systems")
        self._info(8)

    def _set_chunks(self, edges: int, node_cut: list, edge_cut: list):
        self.num_edges, n = edges, len(node_cut) - 1
        self.num_chunks = n
        self.chunk_node, self.chunk_edge = (c_int64 * (n + 1))(*node_cut), (c_int64 * (n + 1))(*edge_cut)

    def _finish_info(self, info):
        n = int(info[2])
        nodes, edges = info[INFO_NODES:INFO_NODES + n + 1].tolist(), info[INFO_EDGES:INFO_EDGES + n + 1].tolist()
        if any(b <= a for a, b in zip(edges, edges[1:])):  # a target with more edges than a chunk: do not cut
            nodes, edges = [0, self.nodes], [0, int(info[0])]
        self._set_chunks(int(info[0]), nodes, edges)

    def build(self) -> bool:
        """Search, selection and tables from the positions.  False: not for this path."""
        g, bb = self.g, self.bb
        nl = bb.neighbor_list
        k = g.max_neighbors
        g.stride = min(STRIDE_MAX, 2 * k + 8) if k > 0 else STRIDE_MAX
        g.want_totals = int(self.nodes > BRUTE_NODES and nl is None)
        self._call("fcb200_graph_systems")
        capacity = self.nodes * g.stride
        rows = torch.empty(capacity * 2, dtype=torch.int32, device=self.device)
        g.rows = rows.data_ptr()
        # Few nodes: the edge arrays are sized for every kept-neighbour slot, so that they are filled before the host learns
        # the edge count instead of after it; finish() reads it once the host has nothing else left to prepare.
        if nl is None and self.nodes <= BRUTE_NODES and 2 * capacity < 3 * g.chunk_edges:
            self._call("fcb200_graph_select")
            self._fill(capacity, 1)
            self.pending = True
            return True
        if nl is not None:
            info = self._select_kept(nl)
        else:
            if g.want_totals:
                head = self._info(8)
                if int(head[1]):
                    return False
                g.num_sources, g.num_cells = int(head[4]), int(head[5])
                if float(head.view(torch.float32)[6]) > BRUTE_PAIRS:
                    c = _Carve(self.device, cell_count=g.num_cells + 1, cell_ptr=g.num_cells + 1, cell_fill=g.num_cells + 1,
                               source_cell=g.num_sources, bucket=4 * g.num_sources)
                    for name, p in c.ptr.items():
                        setattr(g, name, p)
            self._call("fcb200_graph_select")
            info = self._info()
        if info is None or int(info[1]) or int(info[0]) == 0:
            return False
        self._finish_info(info)
        self._fill(self.num_edges, self.num_chunks)
        return True

    def finish(self) -> bool:
        """After build: the number of edges where it is not known yet.  False: not for this path."""
        if self.pending:
            self.pending = False
            info = self.a.view("info", 8).tolist()
            self._refuse(info[INFO_INPUT])
            if info[1] or info[0] == 0:
                return False
            self._set_chunks(info[0], [0, self.nodes], [0, info[0]])
            self.edge_index, self.cell_offsets = self.edge_index[:, :info[0]], self.cell_offsets[:info[0]]
        return True

    def _fill(self, capacity: int, chunks: int):
        self._edges(capacity, chunks)
        self.edge_index = torch.empty(2, capacity, dtype=torch.int64, device=self.device)
        self.cell_offsets = torch.empty(capacity, 3, dtype=torch.float32, device=self.device)
        self.g.edge_index, self.g.cell_offsets = self.edge_index.data_ptr(), self.cell_offsets.data_ptr()
        self._call("fcb200_graph_fill")

    def _select_kept(self, nl):
        """Selection from a SkinNeighborList's candidates, refreshed by a new search when they have expired."""
        g, data = self.g, self.data
        key = (self.nodes, tuple(data["natoms"].shape), self.device, None)
        if nl.skin > 0.0 and nl._cand is not None and nl._key == key and nl.origin is not None:
            pos0, cell0, pbc0, natoms0 = nl.origin
            g.pos0, g.cell0, g.pbc0, g.natoms0 = pos0.data_ptr(), cell0.data_ptr(), pbc0.data_ptr(), natoms0.data_ptr()
            g.limit_sq = (0.5 * nl.skin) ** 2
            self._candidates(nl)
            self._call("fcb200_graph_select")
            info = self._info()
            if not int(info[3]):
                nl.refreshes += 1
                return info
        self._info(8)  # the search indexes by the batch
        nl.search(data, data["pbc"])
        nl.origin = (nl._pos0, self.alive[0].clone(), self.alive[1].clone(), self.alive[2].clone())
        g.pos0 = None
        self._candidates(nl)
        self._call("fcb200_graph_select")
        return self._info()

    def _candidates(self, nl):
        c = nl._cand
        self.g.cand_ptr, self.g.cand_id, self.g.cand_sys = c.cand_ptr.data_ptr(), c.cand_id.data_ptr(), c.sys_t.data_ptr()
        self.candidates = c

    def _edges(self, e: int, chunks: int):
        n = self.nodes
        sizes = dict(src=e, tgt=e, shift=3 * e)
        if self.want_grad:
            sizes.update(src_count=n, src_ptr=n + 1, src_tmp=e, src_perm=e)
            if chunks > 1:
                sizes["chunk_src"] = (chunks + 1) * n
        self.b = _Carve(self.device, **sizes)
        for name, p in self.b.ptr.items():
            setattr(self.g, name, p)
        self.g.num_edges, self.g.num_chunks = e, chunks
        self.shift = self.g.shift

    def from_edges(self, src, tgt, shift):
        """Tables for a given edge list (int64, sorted by target) and its shift vectors."""
        g = self.g
        self._call("fcb200_graph_systems")
        g.rows, g.cand_sys = None, None
        e = src.shape[0]
        self._edges(e, max(1, min(512, (e + g.chunk_edges // 2) // g.chunk_edges)))
        self.b.view("src", e).copy_(src)
        self.b.view("tgt", e).copy_(tgt)
        self.alive.append(shift)
        self.shift = shift.data_ptr()
        self._call("fcb200_graph_fill")
        self._finish_info(self._info())
        return self
