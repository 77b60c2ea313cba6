"""The articulation's descent in the space of its constraint rows against the one in its coordinates."""
import os

import numpy as np
import pytest

from nuka import Field as F, templates as T
from test_gpu_merged_tree import star
from test_gpu_variants import assert_same, create, outputs

pytestmark = pytest.mark.gpu


def scene(name, E):
    rng = np.random.Generator(np.random.PCG64(len(name)))
    if name == "quadruped":
        return T.quadruped(0), T.quadruped_state(E, 0)
    limbs, depth, floating, joint = {"limits": (2, 2, True, dict(limits=(-0.1, 0.1), frictionloss=0.02)),       # 12 rows of joints, with a contact the 15 that fit
                                     "fixed": (4, 2, False, {}), "deep": (3, 5, True, {}),
                                     "locking": (4, 7, True, {}),
                                     "wide": (5, 6, True, {})}[name]                                              # these two with two coordinates per lane
    n = limbs * depth
    q = np.zeros((E, n + 1), np.float32)
    q[:, 1:] = 0.25 * rng.standard_normal((E, n))
    state = {"q": q, "qdot": np.zeros_like(q)}
    state["qdot"][:, 1:] = rng.standard_normal((E, n))
    if floating:
        state["base_pose"] = np.zeros((E, 7), np.float32)
        state["base_pose"][:, 2:4] = 1.0
    return star(limbs, depth, floating, **joint), state


# Every row that fits; 14 and 4 rows at most, no multiples of the three that a contact has (envs with more take the coordinates);
# split steps.  The bars of one step's velocities against the reference: 1e-5 of max(|v|, 1).  A sweep ends an env's solve where its
# rows' residual falls below 1e-5 m/s, so two roundings can end it a sweep apart, which moves a light joint at the end of a limb by
# that residual over its lever of 0.04 m: up to 3e-4 rad/s per row, of which a tip has three.
@pytest.mark.parametrize("name", ["quadruped", "limits", "fixed", "deep", "wide"])
@pytest.mark.parametrize("forced", [{}, {"ROWS": 14}, {"ROWS": 4}, {"SPLIT": 1}], ids=["all", "14", "4", "split"])
def test_rows_equal_coordinates(device, name, forced):
    E = 96
    tb, state = scene(name, E)
    rows = outputs(create(device, tb, state, E, **forced), (1,))
    coordinates = outputs(create(device, tb, state, E, ROWS=0), (1,))
    assert rows["CONTACT_COUNT"].sum() > 0 and rows["ENV_STATUS"].max() == 0 and coordinates["ENV_STATUS"].max() == 0
    got, want = rows["JOINT_VELOCITY"].astype(np.float64), coordinates["JOINT_VELOCITY"].astype(np.float64)
    assert np.array_equal(got, want) == (name != "wide")          # the other route, which up to 32 coordinates do not take
    error = np.abs(got - want).max(axis=1) / np.maximum(np.abs(want).max(axis=1), 1.0)
    assert np.percentile(error, 95) < 1e-5 and error.max() < 1e-3, (float(np.percentile(error, 95)), float(error.max()))
    assert (rows["SOLVER_SWEEPS"] == coordinates["SOLVER_SWEEPS"]).mean() > 0.95


# One step against a 64-bit evaluation of the same inputs (golden/wide_exact.npz: the oracle's sources with double for float).  The descent by
# rows may be no less exact than the one in coordinates.  The envs are the same, so what a mean over 512 of them can differ by is a few per cent.
def test_rows_are_as_exact_as_coordinates(device):
    E = 512
    tb, state = scene("wide", E)
    want = np.load(os.path.join(os.path.dirname(__file__), "golden", "wide_exact.npz"))["qdot"]
    errors = []
    for forced in ({}, {"ROWS": 0}):
        out = outputs(create(device, tb, state, E, **forced), (1,))
        touched = (out["CONTACT_COUNT"].reshape(E, -1) > 0).any(axis=1)
        error = np.abs(out["JOINT_VELOCITY"].reshape(E, -1).astype(np.float64) - want).max(axis=1) / np.maximum(np.abs(want).max(axis=1), 1.0)
        errors.append(np.exp(np.log(error[touched] + 1e-12).mean()))
    assert errors[0] != errors[1] and errors[0] < 1.05 * errors[1], errors


# The last residual is the momentum balance at the velocity found, whichever space the descent took: no 32-bit velocity is in exact balance
# with contacts, so it is zero only where the descent in coordinates finds zero as well
@pytest.mark.parametrize("name", ["wide", "locking"])
def test_balance_of_descents_by_rows_is_measured(device, name):
    E = 96
    tb, state = scene(name, E)
    rows, coordinates = (outputs(create(device, tb, state, E, **forced), (1,)) for forced in ({}, {"ROWS": 0}))
    touched = (rows["CONTACT_COUNT"].reshape(E, -1) > 0).any(axis=1)
    got, want = rows["SOLVER_RESIDUAL"].reshape(E, 4)[touched, 3], coordinates["SOLVER_RESIDUAL"].reshape(E, 4)[touched, 3]
    assert (want > 0).sum() > 20 and not ((got == 0) & (want > 0)).any(), (int(((got == 0) & (want > 0)).sum()), float(want.max()))


# Solves in two slices against one, and against whole steps: the same bits.  With four rows the small slice holds one contact, so that both
# slices have envs to solve; with free bodies one that touches nothing counts as well
@pytest.mark.parametrize("name", ["quadruped", "boxes", "wide"])
@pytest.mark.parametrize("rows", [4, 64])
def test_small_and_large_slices_equal_whole_steps(device, name, rows):
    E = 300
    if name == "boxes":
        tb, state = T.quadruped(0, boxes=2), T.quadruped_state(E, 0)
    else:
        tb, state = scene(name, E)
    whole, one, two = (outputs(create(device, tb, state, E, ROWS=rows, **forced), (2, 1))
                       for forced in (dict(SPLIT=0), dict(SPLIT=1, ONE_TIER=1), dict(SPLIT=1, TWO_TIERS=1)))
    assert two["CONTACT_COUNT"].sum() > 0
    assert_same(whole, one)
    assert_same(one, two)


# The same with the shapes read from the printed layout.  A small slice with room for one contact of the articulation
# leaves both slices envs to solve (with free bodies one that touches nothing counts as well); the usual one; with four rows in the rows' space
@pytest.mark.parametrize("name", ["quadruped", "boxes", "wide"])
@pytest.mark.parametrize("small", [{"SMALL_REACH": 1}, {}, {"ROWS": 4}], ids=["one", "usual", "rows"])
def test_envs_on_both_sides_of_the_small_slice(device, capfd, name, small):
    E = 300
    if name == "boxes":
        tb, state = T.quadruped(0, boxes=2), T.quadruped_state(E, 0)
    else:
        tb, state = scene(name, E)
    whole, one, two = (outputs(create(device, tb, state, E, **small, **forced), (2, 1))
                       for forced in (dict(SPLIT=0), dict(SPLIT=1, ONE_TIER=1), dict(SPLIT=1, TWO_TIERS=1)))
    shapes = [line for line in capfd.readouterr().err.splitlines() if "split: stages" in line]
    assert [int(line.split("small ")[1].split()[0]) != 0 for line in shapes] == [False, True]              # whole steps have no slices
    touched = (two["CONTACT_COUNT"] > 0).sum(axis=1)
    if small == {"SMALL_REACH": 1} and name != "boxes":
        assert (touched > 1).any() and (touched <= 1).any()                                                # envs on both sides
    assert_same(whole, one)
    assert_same(one, two)
