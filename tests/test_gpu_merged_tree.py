"""Contacts between two branches of an articulation's tree: the Newton systems on the tree with those branches joined against the
dense ones, over the depths a joined tree can have."""
import numpy as np
import pytest

from nuka import Field as F, templates as T
from test_gpu_variants import assert_same, create, outputs

pytestmark = pytest.mark.gpu


def star(limbs, depth, floating, **joint):
    """Limbs of `depth` joints around a small hub, each with a sphere at its tip; the tips of all limbs can touch.  `joint`: more of every joint."""
    tb = T.TemplateBuilder(1.0 / 200.0, 8, max_contacts=32)
    hub = tb.add_link(None, T.FLOATING if floating else T.FIXED, mass=2.0, inertia_diag=(0.02, 0.02, 0.02))
    for k in range(limbs):
        angle = 2.0 * np.pi * k / limbs
        parent, offset = hub, (0.06 * np.cos(angle), 0.06 * np.sin(angle), 0.0)
        for d in range(depth):
            axis = ((np.cos(angle), np.sin(angle), 0.0), (-np.sin(angle), np.cos(angle), 0.0), (0.0, 0.0, 1.0))[(d + k) % 3]
            tip = d == depth - 1
            parent = tb.add_link(parent, T.REVOLUTE, axis=axis, offset=offset, mass=0.3, inertia_diag=(0.001, 0.001, 0.001), com=(0.0, 0.0, 0.03),
                                 kp=5.0, kd=0.2, armature=0.005, shape=(T.SPHERE, 0.05) if tip else None, conaffinity=1, **joint)
            offset = (0.0, 0.0, 0.25 / depth)
    return tb


# one coordinate per lane: two limbs, with and without a floating base; as deep as the solve's levels; deeper where five limbs touch.
# Two coordinates per lane: joins of 18 of 24 levels and of 27; of 14, 21 and 28; of up to exactly 24 and of 28
@pytest.mark.parametrize("limbs,depth,floating", [(2, 3, True), (2, 3, False), (4, 3, True), (5, 3, True), (3, 9, True), (4, 7, True), (7, 4, True)])
def test_joined_branches_equal_dense_systems(device, limbs, depth, floating):
    E, n = 96, limbs * depth
    tb, rng = star(limbs, depth, floating), np.random.Generator(np.random.PCG64(limbs * depth))
    q = np.zeros((E, n + 1), np.float32)
    q[:, 1:] = 0.25 * rng.standard_normal((E, n))
    qd = np.zeros_like(q)
    qd[:, 1:] = rng.standard_normal((E, n))
    state = {"q": q, "qdot": qd}
    if floating:
        base = np.zeros((E, 7), np.float32)
        base[:, 2], base[:, 3] = 1.0, 1.0
        state["base_pose"] = base
    for steps, bar95, worst in ((1, 1e-5, 1e-4), (3, 1e-4, 5e-3)):
        joined, dense = (outputs(create(device, tb, state, E, **forced), (steps,)) for forced in ({"ROWS": 0}, {"DENSE": 1}))
        assert (joined["CONTACT_COUNT"].sum(axis=1) > 0).mean() > 0.25         # two limbs meet in three envs of ten, seven in all
        assert joined["ENV_STATUS"].max() == 0 and dense["ENV_STATUS"].max() == 0
        got, want = joined["JOINT_VELOCITY"].astype(np.float64), dense["JOINT_VELOCITY"].astype(np.float64)
        assert not np.array_equal(got, want)                  # some envs took the other route
        # the bars of the reference comparisons: velocities against max(|v|, 1), an unconverged solve amplifies last-bit differences
        error = np.abs(got - want).max(axis=1) / np.maximum(np.abs(want).max(axis=1), 1.0)
        assert np.percentile(error, 95) < bar95 and error.max() < worst, (steps, float(np.percentile(error, 95)), float(error.max()))
    assert_same(outputs(create(device, tb, state, E, SPLIT=0), (2, 1)), outputs(create(device, tb, state, E, SPLIT=1), (1, 2), True))


# Beside the limbs' contacts: rows of free bodies on the tips, of joints past their limits, of dry friction.  One coordinate per lane and
# two, whole steps and split ones (two coordinates with free bodies have no split form)
@pytest.mark.parametrize("limbs,depth,floating", [(4, 3, True), (3, 3, False), (7, 4, True)])
@pytest.mark.parametrize("bodies", [0, 3])
def test_joined_branches_beside_bodies_limits_and_friction(device, limbs, depth, floating, bodies):
    E, n = 96, limbs * depth
    tb, rng = star(limbs, depth, floating, limits=(-0.2, 0.2), frictionloss=0.02), np.random.Generator(np.random.PCG64(n))
    tb.cfg["max_contacts"] = 64
    height = 0.25 * (depth - 1) / depth
    links = len(tb.bodies)
    for k in range(bodies):
        tb.add_free_body((T.SPHERE, 0.05), 1.0, (0.001, 0.001, 0.001), (0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0))
    q = np.zeros((E, n + 1), np.float32)
    q[:, 1:] = 0.2 * rng.standard_normal((E, n))
    state = {"q": q, "qdot": np.zeros_like(q)}
    state["qdot"][:, 1:] = rng.standard_normal((E, n))
    base = np.zeros((E, 7), np.float32)
    base[:, 3] = 1.0
    if floating:
        base[:, 2] = 1.0
        state["base_pose"] = base
    if bodies:
        pose = np.zeros((E, links + bodies, 7), np.float32)
        pose[..., 3] = 1.0
        for k in range(bodies):                               # over the tips, about to be pushed aside
            angle = 2.0 * np.pi * k / bodies
            pose[:, links + k, :3] = np.array([0.08 * np.cos(angle), 0.08 * np.sin(angle), height + 0.085], np.float32) + base[:, :3]
        state["body_pose"] = pose.reshape(E, -1)
    # one step with free bodies: in later ones the force on a body that nothing touches can underflow, which ends the env's sweeps (the
    # reference's rule), and with it single envs of any two roundings
    for steps, bar95, worst in ((1, 1e-5, 1e-4), (3, 1e-4, 5e-3))[:1 if bodies else 2]:
        joined, dense = (outputs(create(device, tb, state, E, **forced), (steps,)) for forced in ({}, {"DENSE": 1}))
        assert (joined["CONTACT_COUNT"].sum(axis=1) > 0).mean() > 0.25
        assert joined["ENV_STATUS"].max() == 0 and dense["ENV_STATUS"].max() == 0
        assert not np.array_equal(joined["JOINT_VELOCITY"], dense["JOINT_VELOCITY"])
        for field in ("JOINT_VELOCITY",) + (("BODY_LINEAR_VELOCITY",) if bodies else ()):
            got, want = (x[field].reshape(E, -1).astype(np.float64) for x in (joined, dense))
            error = np.abs(got - want).max(axis=1) / np.maximum(np.abs(want).max(axis=1), 1.0)
            assert np.percentile(error, 95) < bar95 and error.max() < worst, (field, steps, float(np.percentile(error, 95)), float(error.max()))
    if not (bodies and n > 26):
        assert_same(outputs(create(device, tb, state, E, SPLIT=0), (2, 1)), outputs(create(device, tb, state, E, SPLIT=1), (1, 2), True))
