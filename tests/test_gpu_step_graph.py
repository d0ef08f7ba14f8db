"""Graph of a whole-model evaluation (csrc/graph_step.cu): each way of searching against the stand-alone search, which
tests/test_gpu_graph.py holds to the oracle, and each case that it leaves to that search."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _bb(**kw):
    from fairchem_b200 import backbone as B
    from fairchem_b200 import weights

    cfg = dict(weights.UMA_S, num_layers=1)
    return B.build_model(cfg, weights.random_init_state_dict(cfg, 0), device="cuda", **kw)


def _edges(index, offsets):
    """Rows (target, source, image) in order."""
    rows = torch.cat([index.flip(0).t(), offsets.long()], 1).cpu().tolist()
    return sorted(map(tuple, rows))


def _skewed(synthetic):
    d = synthetic.bcc_alloy((4, 3, 5), seed=3)
    shear = torch.tensor([[1.0, 0.0, 0.0], [0.35, 1.0, 0.0], [-0.3, 0.25, 1.0]])
    d["cell"], d["pos"] = d["cell"] @ shear, d["pos"] @ shear
    return d


def _slab(synthetic):
    d = synthetic.fcc_cu((3, 3, 2), seed=4)
    d["pbc"] = torch.tensor([[True, True, False]])
    return d


SYSTEMS = {
    "molecules": lambda s: s.molecule_batch(9, 2, 40, seed=1),
    "small_cell": lambda s: s.fcc_cu((1, 1, 1), seed=2),
    "skewed_cell": _skewed,
    "slab": _slab,
    "mixed_batch": lambda s: s.merge([s.fcc_cu((2, 2, 3), seed=5), s.molecule_batch(3, 5, 20, seed=6), _skewed(s)]),
    "water": lambda s: s.water_box(1201, seed=7),
}


@pytest.mark.parametrize("name", list(SYSTEMS))
@pytest.mark.parametrize("search", ["images", "images_counted", "grid", "kept_list", "chunked"])
def test_searches_find_the_edges_of_the_stand_alone_search(name, search, monkeypatch):
    from fairchem_b200 import step, synthetic
    from fairchem_b200.graph import SkinNeighborList, radius_graph_pbc_b200

    bb, _ = _bb(**({"edge_chunk_size": 300} if search == "chunked" else {}))
    d = SYSTEMS[name](synthetic).to("cuda")
    if search in ("images_counted", "grid"):
        monkeypatch.setattr(step, "BRUTE_NODES", 0)
    if search == "grid":
        monkeypatch.setattr(step, "BRUTE_PAIRS", 0)
    if search == "kept_list":
        bb.neighbor_list = SkinNeighborList(bb.cutoff, bb.max_neighbors, 0.6)
        bb(d.clone())
        with torch.no_grad():
            d["pos"] = d["pos"] + 0.05 * torch.randn(d["pos"].shape, generator=torch.Generator("cuda").manual_seed(1), device="cuda").clamp(-2, 2)
    graph = step.StepGraph(bb, d, True)
    assert graph.build() and graph.finish()
    assert bool(graph.g.cell_ptr) == (search == "grid") and bool(graph.g.cand_ptr) == (search == "kept_list")
    if search == "kept_list":
        assert (bb.neighbor_list.searches, bb.neighbor_list.refreshes) == (1, 1)
    if search == "chunked":
        assert graph.num_chunks == max(1, (graph.num_edges + 150) // 300)
    index, offsets, _ = radius_graph_pbc_b200(d, bb.cutoff, bb.max_neighbors, False, d["pbc"])
    assert graph.num_edges == index.shape[1] and graph.edge_index.shape == index.shape
    assert bool((graph.edge_index[1][1:] >= graph.edge_index[1][:-1]).all())
    assert _edges(graph.edge_index, graph.cell_offsets) == _edges(index, offsets)
    # the tables of the backward pass: edges by source, in edge order
    n, e = graph.nodes, graph.num_edges
    src = graph.edge_index[0]
    ptr, perm = graph.b.view("src_ptr", n + 1).long(), graph.b.view("src_perm", e).long()
    assert torch.equal(ptr[1:] - ptr[:-1], torch.bincount(src, minlength=n)) and int(ptr[0]) == 0
    assert torch.equal(perm, torch.sort(src, stable=True).indices)


def test_a_box_that_is_searched_by_grid_by_itself():
    from fairchem_b200 import step, synthetic
    from fairchem_b200.graph import radius_graph_pbc_b200

    bb, _ = _bb()
    d = synthetic.water_box(13001, seed=2).to("cuda")
    graph = step.StepGraph(bb, d, True)
    assert graph.build() and graph.finish() and graph.g.cell_ptr and graph.num_chunks > 1
    index, offsets, _ = radius_graph_pbc_b200(d, bb.cutoff, bb.max_neighbors, False, d["pbc"])
    assert _edges(graph.edge_index, graph.cell_offsets) == _edges(index, offsets)


def _perfect_fcc(synthetic):
    d = synthetic.fcc_cu((3, 3, 3), seed=0)
    a = float(d["cell"][0, 0, 0]) / 3
    frac = torch.tensor([[0.0, 0.0, 0.0], [0.0, 0.5, 0.5], [0.5, 0.0, 0.5], [0.5, 0.5, 0.0]])
    grid = torch.cartesian_prod(*[torch.arange(3.0)] * 3)
    d["pos"] = ((grid[:, None] + frac[None]).reshape(-1, 3) * a).float()
    return d


def _dense(synthetic):
    d = synthetic.molecule_batch(1, 600, 600, seed=1)
    g = torch.cartesian_prod(*[torch.arange(9.0)] * 3)[:600]  # 0.6 A apart: every atom has some 600 within 6 A
    d["pos"] = 0.6 * g + 0.01 * torch.randn(600, 3, generator=torch.Generator().manual_seed(1))
    return d


# more kept neighbours than a row holds (12 at one distance, limit 1); more candidates than shared memory holds
LEFT = {"kept_neighbours": (_perfect_fcc, {"max_neighbors": 1}), "candidates": (_dense, {}),
        "no_edges": (lambda s: s.molecule_batch(2, 1, 1, seed=1), {})}


@pytest.mark.parametrize("name", list(LEFT))
@pytest.mark.parametrize("when", ["after_the_edge_arrays", "before"])
def test_what_the_native_graph_leaves_to_the_stand_alone_search(name, when, monkeypatch):
    from fairchem_b200 import backbone as B
    from fairchem_b200 import step, synthetic

    make, over = LEFT[name]
    bb, head = _bb(**({"edge_chunk_size": 50} if when == "before" else {}))
    for key, value in over.items():
        setattr(bb, key, value)
    data = make(synthetic).to("cuda")
    graph = step.StepGraph(bb, data.clone(), True)
    if when == "before":
        assert not graph.build()
    else:
        assert graph.build() and graph.pending and not graph.finish()
    out = {}
    for native in (True, False):
        monkeypatch.setattr(B._GemmState, "native", native)
        d = data.clone()
        emb = bb(d)
        assert ("step" in emb) == native
        out[native] = (bb.last_graph, head(d, emb))
    (g1, r1), (g0, r0) = out[True], out[False]
    assert _edges(g1["edge_index"], g1["cell_offsets"]) == _edges(g0["edge_index"], g0["cell_offsets"])
    for k in r0:
        assert float((r1[k].double() - r0[k].double()).norm()) <= 2e-5 * float(r0[k].double().norm()) + 1e-6 * len(data.pos), k


def test_a_cell_of_no_volume_is_left_to_the_stand_alone_search():
    from fairchem_b200 import step, synthetic

    bb, _ = _bb()
    d = synthetic.fcc_cu((2, 2, 2), seed=1).to("cuda")
    d["cell"] = d["cell"].clone()
    d["cell"][0, 2] = d["cell"][0, 1]
    graph = step.StepGraph(bb, d, True)
    assert graph.build() and not graph.finish()
    with pytest.raises((ValueError, OverflowError)):  # which refuses it: no image count comes of a volume of zero
        bb(d)
