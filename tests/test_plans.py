"""The plans that calls of one geometry share (lattice_filter.py): host code, no GPU needed."""
import sys

import numpy as np
import torch

import permutohedral_lattice_b200 as plb   # noqa: F401 - loads the module below

lf = sys.modules["permutohedral_lattice_b200.lattice_filter"]


def test_thetas_of_any_type_are_taken_by_value():
    x, ref = torch.zeros((1, 8, 9, 3)), torch.zeros((1, 8, 9, 2))
    plain = lf._plan_of(x, ref, True, 8.0, 0.5, 1.0)
    assert lf._plan_of(x, ref, True, np.array(8.0), np.float32(0.5), torch.tensor(1)) is plain
    theta = torch.tensor(8.0)
    assert lf._plan_of(x, ref, True, theta, 0.5, 1.0) is plain
    theta.mul_(2.0)
    changed = lf._plan_of(x, ref, True, theta, 0.5, 1.0)
    assert changed is not plain and changed.call.theta == (16.0, 0.5, 1.0) and plain.call.theta == (8.0, 0.5, 1.0)


def test_number_of_plans_is_bounded():
    for n in range(1, lf.MOST_PLANS + 20):
        lf._plan_of(torch.zeros((1, 1, n, 1)), None, False, 1.0, 1.0, 1.0)
    assert len(lf._plans) <= lf.MOST_PLANS
