"""Sizes at the edges of what the path accepts: one env, the largest articulation (32 links; 64 coordinates would need
more links than fit, so 31 scalar joints under a floating base: 37 coordinates, two per lane), a world without
collidables, and templates just past the limits."""
import numpy as np
import pytest

import nuka
from nuka import Field as F, templates as T

pytestmark = pytest.mark.gpu


def chain(links, floating=True):
    """A serial chain of revolute joints with alternating axes under a floating (or fixed) root."""
    tb = T.TemplateBuilder(dt=1.0 / 500.0, vel_iters=4, max_contacts=0)
    tb.add_link(None, T.FLOATING if floating else T.FIXED, mass=2.0, inertia_diag=(0.02, 0.02, 0.02))
    for i in range(links - 1):
        tb.add_link(i, T.REVOLUTE, axis=(0, 0, 1) if i % 2 == 0 else (0, 1, 0), offset=(0.0 if i == 0 else 0.1, 0, 0), mass=0.3,
                    inertia_diag=T.box_inertia(0.3, (0.1, 0.02, 0.02)), com=(0.05, 0, 0), kp=5.0, kd=0.2)
    return tb


def rel(a, b):
    return float(np.abs(np.asarray(a, np.float64) - np.asarray(b, np.float64)).max() / max(np.abs(b).max(), 1e-12))


def test_largest_articulation_matches_the_oracle(device, oracle):
    E, L = 6, 32
    tb = chain(L)
    rng = np.random.Generator(np.random.PCG64(3))
    q = np.zeros((E, L), np.float32)
    q[:, 1:] = rng.uniform(-0.3, 0.3, size=(E, L - 1))
    blob = tb.blob()
    w = nuka.World.create_from_template(device, blob, E)
    o = oracle.World(blob, E)
    w.upload(F.JOINT_POSITION, q); o.set("q", q)
    w.forward_kinematics(); o.refresh()
    assert w.info.links_per_env == 32 and w.info.dofs_per_env == 37
    assert rel(w.download(F.ARTICULATION_LINK_POSE), o.get("link_pose", 7 * L)) < 1e-6
    w.run_stage(1); o.dynamics(False)
    assert rel(w.download(F.MASS_MATRIX), o.get("mass_matrix", 37 * 37)) < 1e-5
    w.step_n(20); o.step(20)
    assert rel(w.download(F.JOINT_POSITION), o.get("q", L)) < 1e-4
    assert not w.download(F.ENV_STATUS).any() and np.isfinite(w.download(F.JOINT_VELOCITY)).all()
    w.destroy()


def test_one_env_and_a_world_without_collidables(device):
    w = nuka.World.create_from_template(device, T.arm7(0).blob(), 1)
    assert w.info.env_count == 1 and w.info.contact_slots_per_env == 0
    w.step_n(10)
    assert np.isfinite(w.download(F.JOINT_POSITION)).all() and w.download(F.JOINT_POSITION).shape == (1, 8)
    w.reset_envs(np.array([0], np.uint32))
    assert np.array_equal(w.download(F.JOINT_POSITION), np.zeros((1, 8), np.float32))
    w.destroy()


def test_templates_past_the_limits_are_rejected(device):
    lib = nuka._abi.lib()
    too_long = chain(33).blob()                              # 33 links
    assert lib.nuka_b200_template_check(too_long, len(too_long)) == nuka._abi.NOT_SUPPORTED
    with pytest.raises(nuka.NukaError) as e:
        nuka.World.create_from_template(device, too_long, 4)
    assert e.value.code == nuka._abi.NOT_SUPPORTED and "32 links" in str(e.value)
    crowded = T.TemplateBuilder(dt=1.0 / 240.0, vel_iters=4, max_contacts=64)
    for k in range(257):                                      # 257 collidable rows
        crowded.add_free_body((T.SPHERE, 0.05), 1.0, (0.001, 0.001, 0.001), (0.2 * k, 0.0, 1.0, 1.0, 0.0, 0.0, 0.0))
    blob = crowded.blob()
    assert lib.nuka_b200_template_check(blob, len(blob)) == nuka._abi.NOT_SUPPORTED
    slots = T.box_pile(0, count=4)
    slots.cfg["max_contacts"] = 1025                          # more contact slots than the path holds
    blob = slots.blob()
    assert lib.nuka_b200_template_check(blob, len(blob)) == nuka._abi.NOT_SUPPORTED
    with pytest.raises(nuka.NukaError):
        nuka.World.create_from_template(device, T.arm7(0).blob(), 0)       # an empty batch


def test_a_world_that_does_not_fit_leaves_no_error_behind(device):
    """A batch of two hundred million arms (6 GB for each array of joints) is refused for want of memory; the next world, a small
    one, steps, and so does one that stood by."""
    blob = T.arm7(0).blob()
    by = nuka.World.create_from_template(device, blob, 2)
    for _ in range(2):
        with pytest.raises(nuka.NukaError) as err:
            nuka.World.create_from_template(device, blob, 200_000_000)
        assert err.value.code == nuka._abi.OUT_OF_MEMORY
        by.step()
        w = nuka.World.create_from_template(device, blob, 2)
        w.step()
        w.synchronize()
        w.destroy()
    by.synchronize()
    by.destroy()


def standing(kind):
    """A world without a coordinate whose shapes touch the ground: a fixed link, a chain of two, a body of infinite mass."""
    tb = T.TemplateBuilder(1.0 / 200.0, 6, max_contacts=8)
    if kind == "body":
        tb.add_free_body((T.SPHERE, 0.05), np.inf, (np.inf,) * 3, (0.0, 0.0, 0.0495, 1.0, 0.0, 0.0, 0.0))
    else:
        root = tb.add_link(None, T.FIXED, mass=1.0, inertia_diag=(0.01, 0.01, 0.01), offset=(0.0, 0.0, 0.0495), shape=(T.SPHERE, 0.05))
        if kind == "chain":
            tb.add_link(root, T.FIXED, mass=1.0, inertia_diag=(0.01, 0.01, 0.01), offset=(0.3, 0.0, 0.0), shape=(T.BOX, 0.05, 0.05, 0.05))
    tb.add_plane()
    return tb


# the position phase descends the same blocks again; no sweep at all goes straight to it
@pytest.mark.parametrize("vel_iters,pos_iters", [(6, 32), (6, 0), (0, 4)])
@pytest.mark.parametrize("kind,points", [("link", 1), ("chain", 5), ("body", 1)])
def test_worlds_without_a_coordinate_stand_still(device, oracle, kind, points, vel_iters, pos_iters):
    """Contacts that act on no block: the world has heads and nothing that moves."""
    tb = standing(kind)
    tb.cfg.update(vel_iters=vel_iters, pos_iters=pos_iters)
    blob = tb.blob()
    for E in (1, 37):
        w, o = nuka.World.create_from_template(device, blob, E), oracle.World(blob, E)
        assert w.info.dofs_per_env == 0
        w.forward_kinematics()
        o.refresh()
        fields = [F.RIGID_BODY_TRANSFORM] + ([F.ARTICULATION_LINK_POSE, F.LINK_VELOCITY] if kind != "body" else [])
        before = [w.download(f) for f in fields]
        for n in (1, 3):
            w.step_n(n)
        o.step(4)
        assert not w.download(F.ENV_STATUS).any() and (w.download(F.CONTACT_COUNT).sum(axis=1) == points).all()
        assert np.array_equal(w.download(F.CONTACT_COUNT), o.get("contact_count", tb.cfg["max_contacts"]))
        assert np.array_equal(w.download(F.SOLVER_SWEEPS).ravel(), o.get("solver_sweeps", 1).ravel())
        for f, a in zip(fields, before):
            assert np.array_equal(w.download(f), a), f
        w.destroy()


# slices of exactly the 220 KB that a template may take
@pytest.mark.parametrize("count,contacts,points", [(40, 325, 564), (41, 331, 560)])
def test_piles_that_just_fit_are_accepted(device, count, contacts, points):
    tb = T.box_pile(0, count=count)
    tb.cfg["max_contacts"], tb.max_points = contacts, points
    w = nuka.World.create_from_template(device, tb.blob(), 3)
    w.step_n(40)                                             # they have landed
    assert not w.download(F.ENV_STATUS).any() and w.download(F.CONTACT_COUNT).sum() > 0
    w.destroy()


# a revolute limb beside one that is fixed to the hub, two and three revolute limbs: spheres at the tips, which can touch across
# branches, and free ones to fill the slice
@pytest.mark.parametrize("joints,stub,floating,contacts", [(1, True, True, 433), (2, False, True, 433), (3, True, False, 469)])
def test_a_slice_that_joined_branches_would_overfill_does_without(device, monkeypatch, joints, stub, floating, contacts):
    """Near the limit the branches stay apart and the envs where they touch take dense systems, as with joining switched off."""
    tb = T.TemplateBuilder(1.0 / 200.0, 8, max_contacts=contacts, max_points=contacts)
    hub = tb.add_link(None, T.FLOATING if floating else T.FIXED, mass=2.0, inertia_diag=(0.02,) * 3, offset=(0.0, 0.0, 1.0))
    limb = dict(mass=0.3, inertia_diag=(0.001,) * 3, com=(0.0, 0.0, 0.05), shape=(T.SPHERE, 0.05), shape_pos=(0.0, 0.0, 0.1), conaffinity=1)
    if stub:
        tb.add_link(hub, T.FIXED, offset=(0.09, 0.0, 0.0), **limb)
    for k in range(joints):
        tb.add_link(hub, T.REVOLUTE, axis=(0, 1, 0), offset=(-0.09 * k, 0.0, 0.0), **limb)
    for k in range(41):
        tb.add_free_body((T.SPHERE, 0.05), 1.0, (0.001,) * 3, (0.2 * k, 0.0, 3.0, 1.0, 0.0, 0.0, 0.0))
    tb.add_plane()
    states = []
    for dense in (False, True):
        if dense:
            monkeypatch.setenv("NUKA_B200_DENSE", "1")
        w = nuka.World.create_from_template(device, tb.blob(), 3)
        states.append([w.step_n(4)] + [w.download(f) for f in (F.JOINT_VELOCITY, F.BASE_POSE, F.RIGID_BODY_TRANSFORM, F.CONTACT_COUNT, F.ENV_STATUS)])
        w.destroy()
    assert states[0][4].sum() > 0 and not states[0][5].any()
    for a, b in zip(*states):
        assert np.array_equal(a, b)
