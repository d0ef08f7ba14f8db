"""Whole-model native evaluation (csrc/model_step.cu) against the per-op path, at the sizes where its dispatch changes:
one atom without neighbours, ragged row tiles, node counts for each way of sharing a node's edges among warps (8, 4, 1), several chunks."""

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = {
    "one_atom": (lambda s: s.molecule_batch(1, 1, 1, seed=1), {}),
    "molecule_9": (lambda s: s.molecule_batch(1, 9, 9, seed=2), {}),
    "molecules_7": (lambda s: s.molecule_batch(7, 3, 31, seed=3), {}),
    "fcc_32_chunks": (lambda s: s.fcc_cu((2, 2, 2), seed=4), {"edge_chunk_size": 257}),
    "alloy_stress": (lambda s: s.bcc_alloy((3, 4, 5), seed=5), {"regress_stress": True}),
    "water_2200": (lambda s: s.water_box(2200, seed=6), {"edge_chunk_size": 30000}),
    "water_1201": (lambda s: s.water_box(1201, seed=7), {}),
    "alloy_1440": (lambda s: s.bcc_alloy((12, 12, 5), seed=8), {}),
    "batch_stress": (lambda s: s.merge([s.fcc_cu((2, 2, 2), seed=1), s.bcc_alloy((2, 3, 2), seed=2)]), {"regress_stress": True}),
}


def _model(B, cfg_name, **kw):
    from fairchem_b200 import weights

    cfg = getattr(weights, cfg_name)
    if cfg_name == "ESCN_MD_L4":
        cfg = dict(cfg, num_layers=2)
    return B.build_model(cfg, weights.random_init_state_dict(cfg, 0), device="cuda", **kw)


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-12))


@pytest.mark.parametrize("cfg", ["UMA_S", "ESCN_MD_L4"])
@pytest.mark.parametrize("name", list(CASES))
def test_native_evaluation_matches_per_op_path(cfg, name, monkeypatch):
    from fairchem_b200 import backbone as B
    from fairchem_b200 import step, synthetic

    general = []
    from_edges = step.StepGraph.from_edges
    monkeypatch.setattr(step.StepGraph, "from_edges", lambda self, *a: general.append(1) or from_edges(self, *a))
    make, kw = CASES[name]
    bb, head = _model(B, cfg, **kw)
    data = make(synthetic).to("cuda")
    out = {}
    for native in (True, False):
        B._GemmState.native = native
        try:
            d = data.clone()
            emb = bb(d)
            assert ("step" in emb) == native
            out[native] = head(d, emb)
        finally:
            B._GemmState.native = True
    assert len(general) == (name == "one_atom")  # the evaluation's own graph, but for the atom without neighbours
    assert set(out[True]) == set(out[False])
    # energies are sums of per-atom terms of order 0.1 that may cancel
    e, ref = out[True]["energy"], out[False]["energy"]
    assert bool(((e - ref).abs() < 5e-6 * ref.abs().clamp_min(0.1 * len(data.pos))).all())
    f = out[False]["forces"]
    if float(f.abs().max()) > 1e-6:
        assert _rel(out[True]["forces"], f) < 2e-5
    if "stress" in out[True]:
        assert _rel(out[True]["stress"], out[False]["stress"]) < 5e-5


def test_gradient_of_the_node_embedding_and_repeated_use():
    """The embedding is differentiable on its own, an energy-only model keeps nothing, and a released evaluation says so."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S")
    data = synthetic.molecule_batch(3, 5, 12, seed=9).to("cuda")
    grads = []
    weight = None
    for native in (True, False):
        B._GemmState.native = native
        try:
            d = data.clone()
            x = bb(d)["node_embedding"]
            weight = torch.randn(x.shape, generator=torch.Generator("cuda").manual_seed(1), device="cuda") if weight is None else weight
            grads.append(torch.autograd.grad((x * weight).sum(), d["pos"])[0])
        finally:
            B._GemmState.native = True
    assert _rel(grads[0], grads[1]) < 2e-5
    d = data.clone()
    emb = bb(d)
    first = head(d, emb)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(emb["node_embedding"].sum(), d["pos"])
    bb2, head2 = _model(B, "UMA_S", regress_forces=False)
    d = data.clone()
    out = head2(d, bb2(d))
    assert set(out) == {"energy"} and _rel(out["energy"], first["energy"]) < 1e-6


def test_out_of_table_charge_is_an_error():
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S")
    d = synthetic.molecule_batch(2, 5, 5, seed=1).to("cuda")
    d["charge"] = torch.tensor([0, 400], device="cuda")
    with pytest.raises(ValueError):
        head(d, bb(d))


@pytest.mark.parametrize("how", ["assign", "functional_call", "scalars"])
def test_replaced_parameters_and_settings_are_used(how):
    """After an evaluation, other parameter objects and other plain settings: the next one uses them."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S")
    data = synthetic.molecule_batch(2, 6, 9, seed=3).to("cuda")
    before = head(data.clone(), bb(data.clone()))["energy"]
    sd = {k: v.clone() for k, v in bb.state_dict().items()}
    sd["blocks.2.edge_wise.so2_conv_1.fc_m0.weight"] *= 3.0
    call = bb
    if how == "assign":
        bb.load_state_dict(sd, assign=True)
    elif how == "functional_call":
        call = lambda d: torch.func.functional_call(bb, sd, (d,))  # noqa: E731
    else:
        bb.cutoff, bb.rescale_factor, bb.blocks[1].norm_2.eps = 4.5, 3.0, 0.1
    out = []
    for native in (True, False):
        B._GemmState.native = native
        try:
            d = data.clone()
            emb = call(d)
            assert ("step" in emb) == native
            out.append(emb["node_embedding"].detach())
            if how != "functional_call":
                out.append(head(d, emb)["forces"])
        finally:
            B._GemmState.native = True
    half = len(out) // 2
    for got, ref in zip(out[:half], out[half:]):
        assert _rel(got, ref) < 2e-5
    if how == "functional_call":  # and the module's own parameters afterwards
        d = data.clone()
        after = head(d, bb(d))["energy"]
        assert _rel(after, before) < 1e-6


def test_copies_of_a_used_model_evaluate_on_their_own_weights():
    import copy

    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S")
    data = synthetic.molecule_batch(2, 6, 9, seed=4).to("cuda")
    run = lambda b, h: (lambda d: h(d, b(d))["forces"])(data.clone())  # noqa: E731
    first = run(bb, head)
    bb2, head2 = copy.deepcopy((bb, head))
    with torch.no_grad():
        bb2.blocks[0].norm_1.affine_weight.mul_(2.0)
    assert _rel(run(bb2, head2), first) > 1e-3
    assert _rel(run(bb, head), first) < 1e-6


@pytest.mark.parametrize("wants", ["forces", "stress"])
def test_repeated_backward_over_a_retained_graph(wants):
    """Several vector-Jacobian products of one node embedding, then the head's forces, as autograd allows them."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S", regress_stress=wants == "stress")
    data = synthetic.bcc_alloy((2, 2, 3), seed=5).to("cuda")
    out = {}
    for native in (True, False):
        B._GemmState.native = native
        try:
            d = data.clone()
            emb = bb(d)
            x = emb["node_embedding"]
            gen = torch.Generator("cuda").manual_seed(2)
            grads = [torch.autograd.grad((x * torch.randn(x.shape, generator=gen, device="cuda")).sum(), d["pos"], retain_graph=True)[0]
                     for _ in range(3)]
            res = head(d, emb)
            out[native] = grads + [res[k] for k in sorted(res)]
            with pytest.raises(RuntimeError):  # the head did not retain the graph
                torch.autograd.grad(x.sum(), d["pos"])
        finally:
            B._GemmState.native = True
    for got, ref in zip(out[True], out[False]):
        assert _rel(got, ref) < 2e-5


def test_backward_again_without_a_retained_graph_or_after_a_change_is_an_error():
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, _ = _model(B, "UMA_S")
    data = synthetic.molecule_batch(2, 5, 8, seed=6).to("cuda")
    d = data.clone()
    x = bb(d)["node_embedding"]
    torch.autograd.grad(x.sum(), d["pos"])
    with pytest.raises(RuntimeError):
        torch.autograd.grad(x.sum(), d["pos"])
    for key in ("pos", "charge"):
        d = data.clone()
        x = bb(d)["node_embedding"]
        torch.autograd.grad(x.sum(), d["pos"], retain_graph=True)
        with torch.no_grad():
            d[key].add_(1)
        with pytest.raises(RuntimeError):
            torch.autograd.grad(x.sum(), d["pos"])


@pytest.mark.parametrize("what", ["module_hook", "foreign_module", "tensor_hook", "position_hook", "retain_grad"])
def test_hooks_and_foreign_modules_take_part(what):
    """What the per-op path calls and autograd runs is called and run, and the model goes back to the native path after."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S")
    data = synthetic.molecule_batch(2, 5, 8, seed=7).to("cuda")
    plain = head(data.clone(), bb(data.clone()))["energy"]
    d = data.clone()
    ref = head(d, bb(d))["forces"]
    d, seen = data.clone(), []
    if what == "module_hook":
        handle = bb.blocks[1].norm_2.register_forward_hook(lambda m, i, o: seen.append(o) or 2.0 * o)
    elif what == "foreign_module":
        class Doubled(B.RMSNormSH):
            def forward(self, x, extra=None):
                seen.append(x)
                return 2.0 * super().forward(x, extra)

        old = bb.blocks[1].norm_2
        bb.blocks[1].norm_2 = new = Doubled(2, 128).cuda()
        new.load_state_dict(old.state_dict())
    emb = bb(d)
    if what == "tensor_hook":
        emb["node_embedding"].register_hook(lambda g: seen.append(g) or 2.0 * g)
    elif what == "position_hook":
        d["pos"].register_hook(lambda g: seen.append(g) or 2.0 * g)
    elif what == "retain_grad":
        emb["node_embedding"].retain_grad()
    out = head(d, emb)
    if what == "retain_grad":
        assert emb["node_embedding"].grad is not None
        assert _rel(out["forces"], ref) < 2e-5
    else:
        assert len(seen) == 1
        if what in ("tensor_hook", "position_hook"):
            assert _rel(out["forces"], 2.0 * ref) < 2e-5
        else:
            assert _rel(out["energy"], plain) > 1e-4
            if what == "module_hook":
                handle.remove()
            else:
                bb.blocks[1].norm_2 = old
    d = data.clone()
    emb = bb(d)
    assert "step" in emb and _rel(head(d, emb)["forces"], ref) < 1e-6


@pytest.mark.parametrize("cfg,drop", [("UMA_S", 1), ("UMA_S", 4), ("ESCN_MD_L4", 1), ("ESCN_MD_L4", 2)])
@pytest.mark.parametrize("wants", ["forces", "stress"])
def test_layers_that_keep_nothing_per_edge_give_the_same_result(cfg, drop, wants, monkeypatch):
    """Less free memory: some layers are computed again in the backward pass, with the same kernels on the same inputs."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import step, synthetic

    bb, head = _model(B, cfg, regress_stress=wants == "stress", edge_chunk_size=700)
    data = synthetic.merge([synthetic.fcc_cu((2, 2, 3), seed=8), synthetic.molecule_batch(2, 5, 30, seed=9)]).to("cuda")
    d = data.clone()
    ref = head(d, bb(d))
    runs = []

    def short(run):
        run.ev.keep_radial, run.ev.drop_layers = 0, drop
        step._lib.call("fcb200_model_sizes", step.byref(run.model), step.byref(run.ev), run.sizes)
        runs.append(run)
        return True

    monkeypatch.setattr(step.BackboneStep, "plan_memory", short)
    d = data.clone()
    emb = bb(d)
    got = head(d, emb)
    assert len(runs) == 1 and runs[0].ev.num_chunks > 1
    for k in ref:
        assert _rel(got[k], ref[k]) < 1e-6, k


@pytest.mark.parametrize("cfg", ["UMA_S", "ESCN_MD_L4"])
@pytest.mark.parametrize("chunk", [129, 700, 131072])  # items of 32, 64 and 128 columns, rows past the last full tile
def test_gate_gradients_from_kept_planes_and_from_kept_rows_agree(cfg, chunk, monkeypatch):
    """With everything kept the gate's backward reads the gated rows as half planes (22 bits: 2.4e-7 of each term), with the
    radial weights dropped the raw rows in float32."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import step, synthetic

    bb, head = _model(B, cfg, edge_chunk_size=chunk)
    data = synthetic.merge([synthetic.fcc_cu((3, 3, 4), seed=8), synthetic.molecule_batch(2, 5, 30, seed=9)]).to("cuda")
    d = data.clone()
    ref = head(d, bb(d))

    def no_radial(run):
        run.ev.keep_radial, run.ev.drop_layers = 0, 0
        step._lib.call("fcb200_model_sizes", step.byref(run.model), step.byref(run.ev), run.sizes)
        return True

    monkeypatch.setattr(step.BackboneStep, "plan_memory", no_radial)
    d = data.clone()
    got = head(d, bb(d))
    assert torch.equal(got["energy"], ref["energy"])
    assert _rel(got["forces"], ref["forces"]) < 1e-6


@pytest.mark.parametrize("skin", [0.0, 0.5])
def test_without_the_memory_the_per_op_path_takes_over_the_graph(skin, monkeypatch):
    from fairchem_b200 import backbone as B
    from fairchem_b200 import graph, step, synthetic

    bb, head = _model(B, "UMA_S")
    data = synthetic.water_box(300, seed=1).to("cuda")
    d = data.clone()
    ref = head(d, bb(d))
    if skin:
        bb.neighbor_list = graph.SkinNeighborList(bb.cutoff, bb.max_neighbors, skin)
    monkeypatch.setattr(step.BackboneStep, "plan_memory", lambda run: False)
    monkeypatch.setattr(B.eSCNMDBackboneB200, "_graph", lambda *a: pytest.fail("the graph was built a second time"))
    d = data.clone()
    emb = bb(d)
    assert "step" not in emb
    got = head(d, emb)
    for k in ref:
        assert _rel(got[k], ref[k]) < 2e-5
    if skin:
        assert (bb.neighbor_list.searches, bb.neighbor_list.refreshes) == (1, 0)


def test_head_on_another_stream_and_memory_reused_on_the_first():
    """The evaluation's memory is allocated on the backbone's stream; a head on another one frees it there while its kernels
    are still queued, and the first stream's next allocations must not get it before they are done."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S", regress_stress=True)
    data = synthetic.bcc_alloy((6, 6, 6), seed=2).to("cuda")
    d = data.clone()
    ref = head(d, bb(d))
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    junk, got = [], []
    for _ in range(4):
        with torch.cuda.stream(first):
            d = data.clone()
            emb = bb(d)
            nbytes = emb["step"].keep.numel()
        with torch.cuda.stream(second):
            got.append(head(d, emb, check_status=False))
        del emb, d
        with torch.cuda.stream(first):
            junk = [torch.full((nbytes // 2,), 255, dtype=torch.uint8, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    assert len(junk) == 2
    for out in got:
        for k in ref:
            assert _rel(out[k], ref[k]) < 1e-6, k


def test_threads_with_streams_of_their_own_share_a_model():
    import threading

    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S")
    systems = [synthetic.molecule_batch(3, 10, 20, seed=20 + i).to("cuda") for i in range(3)]
    refs = [head(d, bb(d))["forces"] for d in (s.clone() for s in systems)]
    del bb._step_plan, head._step_plan
    torch.cuda.synchronize()
    worst = [1.0] * len(systems)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            rel = []
            for _ in range(10):
                d = systems[i].clone()
                rel.append(_rel(head(d, bb(d))["forces"], refs[i]))
            worst[i] = max(rel)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(systems))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert max(worst) < 1e-6


@pytest.mark.parametrize("what", ["atomic number", "batch", "charge", "spin"])
@pytest.mark.parametrize("graph", ["own", "own_chunked", "own_counted", "kept_list", "given", "all_periodic"])
def test_inputs_outside_the_tables_are_reported_by_the_backbone(what, graph, monkeypatch):
    """The backbone's own call raises and names them; nothing is left behind for the next evaluation."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import step, synthetic
    from fairchem_b200.graph import SkinNeighborList

    kw = {"own_chunked": {"edge_chunk_size": 40}, "all_periodic": {"always_use_pbc": True}}.get(graph, {})
    bb, head = _model(B, "UMA_S", **kw)
    data = synthetic.merge([synthetic.fcc_cu((2, 2, 2), seed=i) for i in range(3)]).to("cuda")
    if graph == "own_counted":
        monkeypatch.setattr(step, "BRUTE_NODES", 0)
    if graph == "kept_list":
        bb.neighbor_list = SkinNeighborList(bb.cutoff, bb.max_neighbors, 0.5)
    if graph == "given":
        bb(data.clone())
        bb.otf_graph = False
        data["edge_index"], data["cell_offsets"] = bb.last_graph["edge_index"].clone(), bb.last_graph["cell_offsets"].clone()
    d = data.clone()
    ref = head(d, bb(d))["forces"]
    key = "atomic_numbers" if what == "atomic number" else what
    for value in (-101, 1000):
        d = data.clone()
        d[key] = d[key].clone()
        d[key][-1] = value
        with pytest.raises(ValueError, match=what):
            bb(d)
        assert B.read_gemm_status() == 0
    d = data.clone()
    assert _rel(head(d, bb(d))["forces"], ref) < 1e-6
    if graph == "kept_list":  # a list that has expired is searched for again, by code that indexes by the batch
        bb.neighbor_list = SkinNeighborList(bb.cutoff, bb.max_neighbors, 0.5)
        d[key] = d[key].clone()
        d[key][0] = 1000
        with pytest.raises(ValueError, match=what):
            bb(d)


def test_kept_list_of_another_split_is_not_used():
    """The same atoms and the same number of systems, divided differently: the kept candidates name periodic sources that a
    target's new system does not have, and the list is searched for again."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic
    from fairchem_b200.graph import SkinNeighborList

    bb, head = _model(B, "UMA_S")
    bb.neighbor_list = SkinNeighborList(bb.cutoff, bb.max_neighbors, 0.5)
    mol, cu = synthetic.molecule_batch(1, 20, 20, seed=2), synthetic.fcc_cu((2, 2, 2), seed=1)
    a, b = synthetic.merge([mol, cu]), synthetic.merge([cu, mol])  # 20 + 32 atoms, images 1 and 27; then the other way round
    for data in (a, b, a):
        d = data.to("cuda")
        emb = bb(d)
        got, kept = head(d, emb), bb.neighbor_list
        bb.neighbor_list = None
        d = data.to("cuda")
        ref = head(d, bb(d))
        bb.neighbor_list = kept
        assert _rel(got["forces"], ref["forces"]) < 1e-6
    assert (kept.searches, kept.refreshes) == (3, 0)


@pytest.mark.parametrize("forces", [False, True])
@pytest.mark.parametrize("mode", ["inference_mode", "no_grad"])
def test_evaluation_inside_inference_mode(forces, mode):
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, "UMA_S", regress_forces=forces)
    data = synthetic.molecule_batch(2, 6, 9, seed=8).to("cuda")
    d = data.clone()
    ref = head(d, bb(d))
    with getattr(torch, mode)():
        d = data.clone() if not (forces and mode == "inference_mode") else data
        out = head(d, bb(d))
    assert set(out) == set(ref)
    for k in ref:
        assert _rel(out[k], ref[k]) < 1e-6


def _close_gates(bb, value):
    """The gates of every edge block near sigmoid(value)."""
    for block in bb.blocks:
        with torch.no_grad():
            block.edge_wise.so2_conv_1.fc_m0.bias[: bb.lmax * 128] = value


def _force_kept_set(monkeypatch, kept):
    """Evaluations are planned with (keep_radial, drop_layers) = kept[-1]; returns what they were planned with."""
    from fairchem_b200 import step

    runs = []

    def forced(run):
        run.ev.keep_radial, run.ev.drop_layers = kept[-1]
        step._lib.call("fcb200_model_sizes", step.byref(run.model), step.byref(run.ev), run.sizes)
        runs.append((int(run.ev.keep_radial), int(run.ev.drop_layers)))
        return True

    monkeypatch.setattr(step.BackboneStep, "plan_memory", forced)
    return runs


@pytest.mark.parametrize("cfg", ["UMA_S", "ESCN_MD_L4"])
@pytest.mark.parametrize("chunk", [129, 700, 131072])
@pytest.mark.parametrize("gates", [0.0, -12.0])
def test_what_the_free_memory_decides(cfg, chunk, gates, monkeypatch):
    """Kept sets differ in what is computed again, by the same kernels on the same inputs: the same bits, but for the first,
    where the gate's gradient is made from half planes (2.4e-7 of a term): forces to 1e-6 of the norm."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, cfg, edge_chunk_size=chunk)
    if gates:
        _close_gates(bb, gates)
    data = synthetic.merge([synthetic.fcc_cu((3, 3, 4), seed=8), synthetic.bcc_alloy((2, 2, 3), seed=9)]).to("cuda")
    kept, forces = [], []
    runs = _force_kept_set(monkeypatch, kept)
    for k in [(1, 0), (2, 0), (0, 0), (0, 1), (0, len(bb.blocks))]:
        kept.append(k)
        d = data.clone()
        forces.append(head(d, bb(d))["forces"])
    assert runs == kept
    assert all(torch.equal(f, forces[1]) for f in forces[2:])
    assert _rel(forces[0], forces[1]) < 1e-6


@pytest.mark.parametrize("cfg", ["UMA_S", "ESCN_MD_L4"])
@pytest.mark.parametrize("gates", [-6.0, -12.0, -20.0])
@pytest.mark.parametrize("kept", [(1, 0), (0, 0)])
def test_closed_gates_against_float64(cfg, gates, kept, monkeypatch):
    """Gates closed to sigmoid = 2.5e-3, 6e-6 and 2e-9: the planes of the gated rows hold 1.5e-11 absolute, not 22 bits, there,
    and what such gates carry is as small."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic, weights
    from oracle import escn_md_oracle as O

    bb, head = _model(B, cfg)
    _close_gates(bb, gates)
    data = synthetic.fcc_cu((2, 3, 3), seed=12)
    runs = _force_kept_set(monkeypatch, [kept])
    d = data.to("cuda")
    forces = head(d, bb(d))["forces"].cpu()
    assert runs == [kept]
    shape = dict(getattr(weights, cfg), num_layers=len(bb.blocks))
    sd = weights.random_init_state_dict(shape, 0)
    for i in range(len(bb.blocks)):
        sd[f"blocks.{i}.edge_wise.so2_conv_1.fc_m0.bias"][: bb.lmax * 128] = gates
    sd = {k: v.double() if v.is_floating_point() else v for k, v in sd.items()}
    graph = bb.last_graph
    _, ref = O.energy_and_forces(sd, shape, data, graph["edge_index"].cpu(), graph["cell_offsets"].cpu())
    assert _rel(forces, ref) < 2e-5


@pytest.mark.parametrize("cfg", ["UMA_S", "ESCN_MD_L4"])
@pytest.mark.parametrize("cells", [(3, 3, 4), (3, 4, 4), (4, 5, 5), (5, 5, 5), (5, 5, 6)])  # one to five rounds of 148 nodes
def test_every_way_of_sharing_a_nodes_edges_among_warps(cfg, cells):
    """Eight or four warps to a node, by node count, lmax and kernel, against the per-op path's one warp."""
    from fairchem_b200 import backbone as B
    from fairchem_b200 import synthetic

    bb, head = _model(B, cfg)
    data = synthetic.fcc_cu(cells, seed=11).to("cuda")
    out = {}
    for native in (True, False):
        B._GemmState.native = native
        try:
            d = data.clone()
            emb = bb(d)
            assert ("step" in emb) == native
            out[native] = head(d, emb)
        finally:
            B._GemmState.native = True
    e, ref = out[True]["energy"], out[False]["energy"]
    assert bool(((e - ref).abs() < 5e-6 * ref.abs().clamp_min(0.1 * len(data.pos))).all())
    assert _rel(out[True]["forces"], out[False]["forces"]) < 2e-5
