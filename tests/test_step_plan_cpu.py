"""Host side of the whole-model evaluation (fairchem_b200/step.py) that needs no GPU: when a plan is still good."""

import pytest
import torch
import torch.nn as nn

from fairchem_b200 import step, weights
from fairchem_b200.backbone import eSCNMDBackboneB200


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
