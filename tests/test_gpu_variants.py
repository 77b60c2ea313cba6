"""One env's step in the shapes a launch can take: one kernel or split around the solve, persistent blocks whose warps take the
next env, contact points in the slice or in their read-out arrays.  Who runs a step and where its data waits changes no result,
so the comparisons are bit-exact.  Each test reads from the printed layout that the shape it is about was taken."""
import contextlib
import ctypes
import os
import re

import numpy as np
import pytest

import nuka
from nuka import Field as F, templates as T

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def layout(**forced):
    """Layout choices forced through the environment; read while a world is created."""
    before = {k: os.environ.get("NUKA_B200_" + k) for k in forced}
    os.environ.update({"NUKA_B200_" + k: str(v) for k, v in forced.items()})
    try:
        yield
    finally:
        for k, v in before.items():
            os.environ.pop("NUKA_B200_" + k) if v is None else os.environ.update({"NUKA_B200_" + k: v})


def create(device, tb, state, E, mode=0, **forced):
    with layout(DEBUG_LAYOUT=1, **forced):
        w = nuka.World.create_from_template(device, tb.blob(), E, control_mode=mode)
    names = {"q": F.JOINT_POSITION, "qdot": F.JOINT_VELOCITY, "base_pose": F.BASE_POSE, "body_pose": F.RIGID_BODY_TRANSFORM}
    for k, v in state.items():
        w.upload(names[k], v[:E])
    w.forward_kinematics()
    return w


def outputs(w, steps, graph=False):
    w.set_execution_mode(graph)
    for n in steps:
        w.step_n(n)
    fields = [F.RIGID_BODY_TRANSFORM, F.BODY_LINEAR_VELOCITY, F.ENV_STATUS, F.SOLVER_SWEEPS, F.SOLVER_RESIDUAL]
    if w.info.contact_slots_per_env:
        fields += [F.CONTACT_COUNT, F.CONTACT_POINT, F.CONTACT_NORMAL]
    if w.info.links_per_env:
        fields += [F.JOINT_POSITION, F.JOINT_VELOCITY, F.BASE_POSE, F.LINK_VELOCITY, F.ACTUATOR_EFFORT]
    out = {f.name: w.download(f) for f in fields}
    w.destroy()
    return out


@pytest.fixture
def shapes(capfd):
    """The launch shapes of the worlds created since the last call, one dict each."""
    def read():
        text, out = capfd.readouterr().err, []
        split = False
        for line in text.splitlines():
            split |= "] split: " in line
            m = re.search(r"registers per thread(.*?); .* (\d+) warps per block, (\d+) per env, meetings of (\d+), (\d+) persistent blocks(.*)", line)
            if m:
                out.append({"slim": "slim" in m[1], "block": int(m[2]), "team": int(m[3]), "group": int(m[4]), "persistent": int(m[5]),
                            "far": "read-out" in m[6], "split": split})
                split = False
        return out
    return read


def assert_same(a, b, envs=slice(None)):
    for k in a:
        assert np.array_equal(a[k][envs], b[k][envs]), k


def scene(name, E, seed):
    if name == "boxes":
        return T.quadruped(0, boxes=4), T.quadruped_state(E, 4)
    return getattr(T, name)(0), getattr(T, name + "_state")(E, seed)


# fewer envs than one part of a split step, one more than an SM's worth, a part that is not full; one step to a call and several
@pytest.mark.parametrize("name,E,steps,graph", [("quadruped", 1, (1, 2), False), ("quadruped", 149, (30,), False), ("quadruped", 601, (25, 1), True),
                                                ("humanoid", 7, (20,), False), ("boxes", 5, (30,), False), ("boxes", 150, (30, 1), True)])
def test_split_steps_equal_whole_ones(device, shapes, name, E, steps, graph):
    tb, st = scene(name, E, 2)
    whole = outputs(create(device, tb, st, E, SPLIT=0), steps)
    split = outputs(create(device, tb, st, E, SPLIT=1), steps, graph)
    assert [x["split"] for x in shapes()] == [False, True]
    assert whole["CONTACT_COUNT"].sum() > 0 or sum(steps) < 10
    assert_same(whole, split)


# a buffer that holds the batch in even rounds, with a remainder, with a last round of fewer envs than parts, and one env at a time
@pytest.mark.parametrize("name,E,room", [("quadruped", 96, 32), ("quadruped", 101, 33), ("quadruped", 7, 1), ("boxes", 50, 16)])
def test_split_steps_in_rounds_over_the_image_buffer(device, shapes, name, E, room):
    tb, st = scene(name, E, 2)
    whole = outputs(create(device, tb, st, E, SPLIT=0), (12, 3))
    for graph in (False, True):
        w = create(device, tb, st, E, SPLIT=1, IMAGE_ENVS=room)
        before = w.launch_count()
        w.step_n(1)
        assert w.launch_count() - before == 9 * -(-E // room)            # three parts of two stages and a solve in each round
        assert_same(whole, outputs(w, (11, 3), graph))


def pick(values, envs):
    return {k: v[envs] for k, v in values.items()}


@pytest.mark.parametrize("name,E,split", [("quadruped", 149, False), ("quadruped", 1500, False), ("quadruped", 4100, True), ("boxes", 1024, False),
                                          ("boxes", 4096, True)])
def test_an_env_does_not_depend_on_its_batch(device, shapes, name, E, split):
    """Block shapes, meetings and split steps follow the batch size.  4096 quadrupeds with boxes run split, four shards of 1024
    run whole."""
    tb, st = scene(name, E, 3)
    some = [0, 1, 2, E - 3, E - 2, E - 1]
    a = outputs(create(device, tb, pick(st, some), 6), (20, 3))
    b = outputs(create(device, tb, st, E), (20, 3))
    assert shapes()[1]["split"] == split
    assert_same(a, pick(b, some))


# more envs than an SM keeps, in one kernel: warps take the next env from the launch's queue, which has to be empty again for the
# next launch.  Warps that meet (quadrupeds in blocks of several, also of 3 that do not fill them evenly), one to a block (humanoids),
# without meetings (arms, computed torque)
@pytest.mark.parametrize("name,E,forced,group", [("quadruped", 4100, {"SPLIT": 0}, 16), ("quadruped", 2500, {"SPLIT": 0, "WARPS_PER_BLOCK": 3}, 3),
                                                 ("boxes", 1700, {}, None), ("humanoid", 1000, {}, 1), ("arm7", 4500, {}, 0), ("arm7", 3001, {"mode": 3}, 0)])
def test_warps_of_a_persistent_launch_take_the_next_env(device, shapes, name, E, forced, group):
    tb, st = scene(name, E, 5)
    some = sorted(set(np.linspace(0, E - 1, 48).astype(int)) | {E - 2})
    mode = forced.get("mode", 0)
    few = outputs(create(device, tb, pick(st, some), len(some), mode=mode), (9, 1, 4))
    for graph in (False, True):
        many = outputs(create(device, tb, st, E, **forced), (9, 1, 4), graph)
        assert_same(few, pick(many, some))
    small, *large = shapes()
    assert small["persistent"] == 0
    for x in large:
        assert 0 < x["persistent"] * x["block"] < E and not x["split"] and (group is None or x["group"] == group), x


def test_a_world_is_created_where_its_images_find_no_room(device):
    """The buffer of split steps (about 25 KB per env here) is taken after the state: with room for the buffer and half of the state the
    world is created, steps in one kernel, and gives the same states."""
    torch = pytest.importorskip("torch")
    E = 8192
    tb, st = scene("boxes", E, 0)
    free = lambda: torch.cuda.mem_get_info(0)[0]
    torch.cuda.empty_cache()
    needs, worlds = [], []
    for split in (0, 1, 0, 1):                    # the first two load their kernels
        before = free()
        w = create(device, tb, st, E, SPLIT=split)
        w.step_n(2)
        w.synchronize()
        needs.append(before - free())
        worlds.append((w.launch_count(), {f.name: w.download(f) for f in (F.RIGID_BODY_TRANSFORM, F.JOINT_POSITION)}))
        w.destroy()
    state, images = needs[2], needs[3] - needs[2]
    assert images > state > 32 << 20
    fill = torch.empty(free() - images - state // 2, dtype=torch.uint8, device="cuda:0")
    w = create(device, tb, st, E, SPLIT=1)
    w.step_n(2)
    assert w.launch_count() == worlds[2][0] != worlds[3][0]
    for k, v in worlds[3][1].items():
        assert np.array_equal(v, w.download(F[k])), k
    w.destroy()
    del fill
    torch.cuda.empty_cache()


def test_split_steps_keep_the_callers_stream_priority(device):
    """Every kernel of a step, those on the world's side streams too: read from the nodes of a captured one."""
    torch = pytest.importorskip("torch")
    runtime = pytest.importorskip("cuda.bindings.runtime")
    stream = torch.cuda.Stream(priority=-1)
    borrowed = nuka.Device.create(0, cuda_stream=stream.cuda_stream)
    w = create(borrowed, T.quadruped(0), T.quadruped_state(32, 0), 32, SPLIT=1)
    w.step_n(1)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        w.step_n(2)
    raw = runtime.cudaGraph_t(graph.raw_cuda_graph())
    count = runtime.cudaGraphGetNodes(raw)[2]
    kernels = [n for n in runtime.cudaGraphGetNodes(raw, count)[1] if runtime.cudaGraphNodeGetType(n)[1] == runtime.cudaGraphNodeType.cudaGraphNodeTypeKernel]
    priorities = [runtime.cudaGraphKernelNodeGetAttribute(n, runtime.cudaLaunchAttributeID.cudaLaunchAttributePriority)[1].priority for n in kernels]
    assert len(priorities) == 15 and set(priorities) == {-1}           # three parts of three stages and two solves
    w.destroy()
    borrowed.destroy()


@pytest.mark.parametrize("count,team", [(48, 8), (48, 1), (40, 3)])
def test_contact_points_in_their_read_out_arrays(device, shapes, count, team):
    """A pile's contact points and normals stay in global memory where that makes room for another env."""
    E = 3
    tb, st = T.box_pile(0, count=count), T.box_pile_state(E, 0, count=count)
    near = outputs(create(device, tb, st, E, NEAR=1, TEAM=team), (25,))
    far = outputs(create(device, tb, st, E, TEAM=team), (25,))
    assert [(x["far"], x["team"]) for x in shapes()] == [(False, team), (True, team)]
    assert near["CONTACT_COUNT"].sum() > count
    assert_same(near, far)


def test_read_out_keeps_its_last_values_while_off(device, shapes):
    """The steps then keep their contact points elsewhere: the arrays stay as they were, and the states do not change."""
    E = 2
    tb, st = T.box_pile(0, count=48), T.box_pile_state(E, 0, count=48)
    on = outputs(create(device, tb, st, E), (20, 5))
    w = create(device, tb, st, E)
    assert shapes()[-1]["far"]
    w.step_n(20)
    before = w.download(F.CONTACT_POINT)
    w.set_contact_readout(False)
    w.step_n(5)
    assert np.array_equal(w.download(F.CONTACT_POINT), before)
    assert np.array_equal(w.download(F.RIGID_BODY_TRANSFORM), on["RIGID_BODY_TRANSFORM"])
    w.set_contact_readout(True)
    w.step_n(1)
    assert not np.array_equal(w.download(F.CONTACT_POINT), before)
    w.destroy()


@pytest.mark.parametrize("room", [0.5, 1.5])
def test_read_out_stays_on_where_the_contacts_find_no_other_place(device, shapes, room):
    """The points and the normals need an array each while the read-out is off; with room for neither or for one of them the call
    fails and changes nothing, and succeeds later."""
    torch = pytest.importorskip("torch")
    E = 4096
    tb, st = T.box_pile(0, count=48), T.box_pile_state(E, 0, count=48)
    on = outputs(create(device, tb, st, E), (3, 2, 2))
    w = create(device, tb, st, E)
    assert all(x["far"] for x in shapes())
    w.step_n(3)
    w.synchronize()
    size = on["CONTACT_POINT"].nbytes
    assert size > 16 << 20
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info(0)[0] - int(room * size), dtype=torch.uint8, device="cuda:0")
    before = w.download(F.CONTACT_POINT)
    with pytest.raises(nuka.NukaError):
        w.set_contact_readout(False)
    w.step_n(2)
    assert not np.array_equal(w.download(F.CONTACT_POINT), before)                # still written
    del fill
    torch.cuda.empty_cache()
    w.set_contact_readout(False)
    w.step_n(1)
    w.set_contact_readout(True)
    w.step_n(1)
    for k, v in on.items():
        assert np.array_equal(v, w.download(F[k])), k
    w.destroy()


def test_downloads_outlive_the_world_and_one_another(device):
    E = 64
    w = create(device, T.quadruped(0), T.quadruped_state(E, 1), E)
    first = w.download(F.JOINT_POSITION)
    kept = first.copy()
    w.step_n(3)
    second = w.download(F.JOINT_POSITION)
    assert np.array_equal(first, kept) and not np.array_equal(first, second)
    kept2 = second.copy()
    w.destroy()
    v = create(device, T.quadruped(0), T.quadruped_state(E, 5), E)
    again = [v.download(F.JOINT_POSITION) for _ in range(4)]
    assert np.array_equal(first, kept) and np.array_equal(second, kept2)
    assert all(np.array_equal(again[0], a) for a in again)
    v.destroy()


def test_a_download_released_twice_is_handed_out_once(device):
    w = create(device, T.quadruped(0), T.quadruped_state(16, 1), 16)
    lib = nuka._abi.lib()

    def block():
        ptr, size = ctypes.c_void_p(), ctypes.c_size_t()
        assert lib.nuka_b200_world_download_host(w._h, int(F.JOINT_POSITION), ctypes.byref(ptr), ctypes.byref(size)) == 0
        return ptr.value

    first = block()
    lib.nuka_b200_host_release(first)
    lib.nuka_b200_host_release(first)
    a, b = block(), block()
    assert a != b
    lib.nuka_b200_host_release(a)
    lib.nuka_b200_host_release(b)
    w.destroy()
