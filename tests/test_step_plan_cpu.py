"""Host side of the whole-model evaluation (fairchem_b200/step.py) that needs no GPU: when a plan is still good, what a
copy of a used model carries."""

import copy
import ctypes
import gc
import pickle
import weakref
from types import SimpleNamespace as NS

import pytest
import torch
import torch.nn as nn

from fairchem_b200 import _lib, step, synthetic, weights
from fairchem_b200.backbone import MLP_EFS_HeadB200, RMSNormSH, eSCNMDBackboneB200
from fairchem_b200.graph import build_system_table


@pytest.fixture()
def bb():
    return eSCNMDBackboneB200(**weights.UMA_S)


def _assign_state(bb):
    bb.load_state_dict({k: v.clone() for k, v in bb.state_dict().items()}, assign=True)


def _new_parameter(bb):
    lin = bb.blocks[1].edge_wise.so2_conv_2.fc_m0
    lin.weight = nn.Parameter(lin.weight.detach() * 2)


def _new_module(bb):
    bb.blocks[3].atom_wise.so3_linear_1 = type(bb.blocks[3].atom_wise.so3_linear_1)(128, 128, 2)


def _in_place(bb):
    with torch.no_grad():
        bb.mix_csd.bias.add_(1.0)


def _moved_storage(bb):
    bb.norm.affine_weight.data = bb.norm.affine_weight.data.clone()


def _swap(bb):
    bb.blocks[0], bb.blocks[1] = bb.blocks[1], bb.blocks[0]


CHANGES = {
    "load_state_dict_assign": _assign_state, "parameter": _new_parameter, "module": _new_module, "in_place": _in_place, "storage": _moved_storage,
    "block_order": _swap, "fewer_blocks": lambda bb: bb.blocks.__delitem__(3),
    "cutoff": lambda bb: setattr(bb, "cutoff", 5.0), "rescale": lambda bb: setattr(bb, "rescale_factor", 4.0),
    "charge_offset": lambda bb: setattr(bb.charge_embedding, "offset", 90),
    "norm_eps": lambda bb: setattr(bb.blocks[2].norm_2, "eps", 1e-4),
    "radial_eps": lambda bb: setattr(bb.edge_degree_embedding.rad_func.net[4], "eps", 1e-3),
}


@pytest.mark.parametrize("change", list(CHANGES))
def test_plan_is_given_up_when_what_it_was_read_from_changes(bb, change):
    origin = step._Origin(bb)
    assert origin.unchanged(bb)
    CHANGES[change](bb)
    assert not origin.unchanged(bb)
    assert step._Origin(bb).unchanged(bb)


def test_plan_is_given_up_inside_functional_call(bb):
    origin, seen = step._Origin(bb), []
    bb.forward = lambda: seen.append(origin.unchanged(bb))
    torch.func.functional_call(bb, {"blocks.0.norm_1.affine_weight": torch.zeros(3, 128)}, ())
    assert seen == [False] and origin.unchanged(bb)


def _used_model():
    """A model as an evaluation leaves it: plans with device addresses on the backbone and the head."""
    bb = eSCNMDBackboneB200(**dict(weights.UMA_S, num_layers=1))
    head = MLP_EFS_HeadB200(bb)
    bb._step_plan, head._step_plan = step.ModelStruct(), (1, step.ModelStruct())
    bb._step_plan.layers = ctypes.pointer(step.LayerStruct())
    return nn.ModuleDict({"bb": bb, "head": head})


@pytest.mark.parametrize("how", ["deepcopy", "pickle", "save", "copy"])
def test_a_used_model_can_be_copied_and_saved_whole(how, tmp_path):
    model = _used_model()
    if how == "deepcopy":
        other = copy.deepcopy(model)
    elif how == "copy":
        other = nn.ModuleDict({k: copy.copy(m) for k, m in model.items()})
    elif how == "pickle":
        other = pickle.loads(pickle.dumps(model))
    else:
        torch.save(model, tmp_path / "model.pt")
        other = torch.load(tmp_path / "model.pt", weights_only=False)
    assert model["bb"]._step_plan is not None and model["head"]._step_plan is not None
    for m in other.values():
        assert not hasattr(m, "_step_plan")
    for (n, p), (_, q) in zip(model.named_parameters(), other.named_parameters()):
        assert torch.equal(p, q), n


class _OtherNorm(RMSNormSH):
    pass


def _foreign_module(bb):
    bb.blocks[1].norm_2 = _OtherNorm(2, 128)


def _other_shape(bb):
    bb.blocks[0].edge_wise.so2_conv_1.fc_m0 = nn.Linear(768, 512)


def test_other_modules_are_not_for_the_native_path(bb):
    assert step.ModelPlan.supported(bb)
    for change in (_foreign_module, _other_shape, CHANGES["charge_offset"]):
        other = copy.deepcopy(bb)
        change(other)
        assert step.ModelPlan.supported(bb) and not step.ModelPlan.supported(other)

    class Sub(eSCNMDBackboneB200):
        def csd_embedding(self, charge, spin, dataset):
            return super().csd_embedding(charge, spin, dataset)

    assert not step.ModelPlan.supported(Sub(**dict(weights.UMA_S, num_layers=1)))


@pytest.mark.parametrize("kind", ["forward_hook", "pre_hook", "backward_hook", "global_hook", "own_forward", "own_method"])
def test_hooks_send_an_evaluation_down_the_per_op_path(bb, kind):
    calls, undo = step._Calls(bb), None
    assert not calls.watched(bb)
    mod = bb.blocks[2].atom_wise.so3_linear_2
    if kind == "forward_hook":
        undo = mod.register_forward_hook(lambda *a: None).remove
    elif kind == "pre_hook":
        undo = bb.norm.register_forward_pre_hook(lambda *a: None).remove
    elif kind == "backward_hook":
        undo = bb.blocks[0].norm_1.register_full_backward_hook(lambda *a: None).remove
    elif kind == "global_hook":
        undo = nn.modules.module.register_module_forward_hook(lambda *a: None).remove
    elif kind == "own_forward":
        mod.forward = lambda x: x
        undo = lambda: delattr(mod, "forward")  # noqa: E731
    else:
        bb.csd_embedding = lambda *a: None
        undo = lambda: delattr(bb, "csd_embedding")  # noqa: E731
    assert calls.watched(bb)
    undo()
    assert not calls.watched(bb)


@pytest.mark.parametrize("cfg", ["UMA_S", "ESCN_MD_L4"])
def test_what_is_kept_follows_the_free_memory_layer_by_layer(cfg, monkeypatch):
    """The 100 000-atom box and beyond: less free memory, fewer layers with per-edge tensors, and only then no evaluation."""
    cfg = getattr(weights, cfg)
    run = object.__new__(step.BackboneStep)
    layers = (step.LayerStruct * cfg["num_layers"])()
    run.model = m = step.ModelStruct()
    m.lmax, m.num_layers, m.num_basis, m.layers = cfg["lmax"], cfg["num_layers"], cfg["num_distance_basis"], layers
    run.ev = e = step.EvalStruct()
    nodes, edges, chunks = 100_000, 3_100_000, 24
    node, edge = ((ctypes.c_int64 * (chunks + 1))(*(n * i // chunks for i in range(chunks + 1))) for n in (nodes, edges))
    e.num_nodes, e.num_edges, e.num_systems, e.num_chunks, e.want_grad = nodes, edges, 1, chunks, 1
    e.chunk_node, e.chunk_edge = ctypes.addressof(node), ctypes.addressof(edge)
    run.sizes, run.device = (ctypes.c_int64 * 3)(), torch.device("cuda", 0)
    total = 183 * 2 ** 30
    monkeypatch.setattr(step.BackboneStep, "_cached", lambda self: 0)

    def kept(avail):
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (avail, total))
        run.__dict__.pop("avail", None)
        if not run.plan_memory():
            return None
        need = run.sizes[0] + max(run.sizes[1], run.sizes[2])
        return e.keep_radial, e.drop_layers, need

    seen, avail = [], 10 ** 13
    while (got := kept(int(avail))) is not None:
        seen.append(got)
        avail = got[2] + 0.03 * total  # what this choice needs: the next one has to do with less
    want = [(1, 0), *((0, n) for n in range(cfg["num_layers"] + 1))]
    assert [s[:2] for s in seen] == want
    lmax = cfg["lmax"]
    rows = 5 * lmax - 1  # of a message
    per_layer = edges * (lmax + 2 * rows) * 512  # conv-1 output and messages
    no_radial = [s[2] for s in seen if s[0] == 0]
    for a, b in zip(no_radial, no_radial[1:]):
        # the row counts are rounded up by at most 1/32; the first dropped layer adds two chunk-sized buffers
        assert a - b < per_layer * 33 / 32 + 4096 and a - b > 0.75 * per_layer
    e.want_grad = 0
    assert kept(10 ** 12)[:2] == (0, 0)


@pytest.mark.parametrize("cfg", ["UMA_S", "ESCN_MD_L4"])
def test_radial_weights_stay_where_only_the_planes_do_not_fit(cfg, monkeypatch):
    """Planes cost 512 bytes an edge and layer more than float32 rows; where that is too much the rows go, not the radial weights."""
    cfg = getattr(weights, cfg)
    run = object.__new__(step.BackboneStep)
    layers = (step.LayerStruct * cfg["num_layers"])()
    run.model = m = step.ModelStruct()
    m.lmax, m.num_layers, m.num_basis, m.layers = cfg["lmax"], cfg["num_layers"], cfg["num_distance_basis"], layers
    run.ev = e = step.EvalStruct()
    nodes, edges, chunks = 60_000, 1_860_000, 15
    node, edge = ((ctypes.c_int64 * (chunks + 1))(*(n * i // chunks for i in range(chunks + 1))) for n in (nodes, edges))
    e.num_nodes, e.num_edges, e.num_systems, e.num_chunks, e.want_grad = nodes, edges, 1, chunks, 1
    e.chunk_node, e.chunk_edge = ctypes.addressof(node), ctypes.addressof(edge)
    run.sizes, run.device = (ctypes.c_int64 * 3)(), torch.device("cuda", 0)
    total = 10 ** 12
    monkeypatch.setattr(step.BackboneStep, "_cached", lambda self: 0)

    def kept(avail):
        monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (int(avail), total))
        run.__dict__.pop("avail", None)
        assert run.plan_memory()
        return e.keep_radial, e.drop_layers, run.sizes[0] + max(run.sizes[1], run.sizes[2])

    planes = kept(10 ** 13)
    assert planes[:2] == (1, 0)
    rows = kept(1.15 * planes[2] + 0.03 * total)  # not enough, by a byte
    assert rows[:2] == (2, 0)
    extra = edges * cfg["num_layers"] * 512
    rounding = 33 / 32
    assert 0 < planes[2] - rows[2] <= extra * rounding
    assert kept(1.15 * rows[2] + 0.03 * total + 1)[:2] == (2, 0)
    assert kept(1.15 * rows[2] + 0.03 * total)[:2] == (0, 0)


class _Stream:
    def __init__(self, handle, log):
        self.cuda_stream, self.log = handle, log

    def wait_stream(self, other):
        self.log.append((self.cuda_stream, "waits for", other.cuda_stream))

    def wait_event(self, event):
        self.log.append((self.cuda_stream, "waits for", event))

    def record_event(self, event=None):
        return f"event of {self.cuda_stream}"


def test_memory_and_weights_used_on_another_stream_are_tied_to_it(monkeypatch):
    log, used = [], []
    one, two = _Stream(1, log), _Stream(2, log)
    now = [one]
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: now[0])
    monkeypatch.setattr(step._lib, "call", lambda name, *args: log.append((args[-1].value, name)))
    tensor = lambda name: NS(record_stream=lambda s: used.append((name, s.cuda_stream)))  # noqa: E731
    plan, head = NS(w=step._Weights(0), model=step.ModelStruct()), NS(w=step._Weights(0), model=step.ModelStruct())
    plan.w.laid_out(), head.w.laid_out()
    run = object.__new__(step.BackboneStep)
    run.device, run.ev, run.home, run.plan = torch.device("cuda", 0), step.EvalStruct(), None, plan
    run.keep, run.graph, run.refs = tensor("keep"), NS(a=NS(block=tensor("a")), b=NS(block=tensor("b"))), [tensor("charge")]
    run._launch("forward", plan)
    run._launch("energy", plan, head)
    assert log == [(1, "forward"), (1, "energy")] and not used
    now[0] = two
    run._launch("backward", plan, head)
    assert log[2:] == [(2, "waits for", 1), *2 * [(2, "waits for", "event of 1")], (2, "backward")]
    assert sorted(used) == [("a", 2), ("b", 2), ("charge", 2), ("keep", 2)]
    del log[:], plan, run
    head.w.__del__()  # both blocks of weights go back behind what the second stream did with them
    assert log == 2 * [(1, "waits for", "event of 2")]
    head.w.last_use.clear()


def test_inputs_of_another_length_than_the_kernels_read_are_refused(bb):
    data = synthetic.molecule_batch(3, 5, 8, seed=1)
    step.StepGraph(bb, data, True)
    for key in ("batch", "atomic_numbers", "cell", "charge", "spin"):
        for wrong in (data[key][:-1], torch.cat([data[key], data[key]])):
            d = data.clone()
            d[key] = wrong
            with pytest.raises(ValueError, match=key):
                step.StepGraph(bb, d, True)
    d = data.clone()
    d["pos"] = d["pos"][:, :2]
    with pytest.raises(ValueError, match="positions"):
        step.StepGraph(bb, d, True)
    with pytest.raises(_lib.FairchemB200Error, match="positions"):
        build_system_table(data.pos, data.cell, data.pbc, data.natoms + 1, 6.0)


def test_a_given_graph_that_names_other_atoms_is_refused(bb):
    bb.otf_graph = False
    data = synthetic.molecule_batch(1, 5, 5, seed=1)
    good = dict(edge_index=torch.tensor([[0, 4], [1, 0]]), cell_offsets=torch.zeros(2, 3))
    data.update(good)
    bb._graph(data)
    for key, wrong in (("edge_index", torch.tensor([[0, 5], [1, 0]])), ("edge_index", torch.tensor([[0, 4], [-1, 0]])),
                       ("cell_offsets", torch.zeros(1, 3)), ("edge_index", torch.zeros(3, 2, dtype=torch.long))):
        data.update({**good, key: wrong})
        with pytest.raises(ValueError, match="edge_index"):
            bb._graph(data)


def test_a_model_and_its_plan_go_without_the_garbage_collector():
    """Their device memory has to come back when the last reference goes, not at some later collection."""
    gc.disable()
    try:
        other = eSCNMDBackboneB200(**dict(weights.UMA_S, num_layers=1))
        other._step_plan = NS(origin=step._Origin(other), calls=step._Calls(other))
        inner = weakref.ref(other.norm)
        del other
        assert inner() is None
    finally:
        gc.enable()
