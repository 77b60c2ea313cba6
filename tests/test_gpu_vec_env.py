"""The RL step loop over a world: action write, decimated stepping, GPU observations, autoreset."""
import numpy as np
import pytest

import nuka
from nuka import Field as F, shard, templates as T
from nuka.vec_env import NukaVecEnv

pytestmark = pytest.mark.gpu


def test_step_loop_shapes_reset_and_autoreset(device):
    torch = pytest.importorskip("torch")
    E = 64
    env = NukaVecEnv(device, T.quadruped(0).blob(), E, decimation=4, episode_length_s=0.4)      # 20 control steps per episode
    obs0 = env.reset()
    assert obs0.shape == (E, shard.OBS_FLOATS) and env.num_joints == 12
    gen = torch.Generator(device="cuda").manual_seed(0)
    resets = 0
    for k in range(45):
        actions = 0.2 * torch.randn((E, 12), generator=gen, device="cuda")
        obs, reward, terminated, truncated, info = env.step(actions)
        assert obs.shape == (E, shard.OBS_FLOATS) and reward.shape == (E,)
        assert torch.isfinite(obs).all() and torch.isfinite(reward).all()
        resets += int(info["done"].sum())
        if k == 19:                                  # every env hits the episode limit together
            assert bool(truncated.all()) and not bool(terminated.any())
            assert torch.equal(obs[:, 12:24], obs0[:, 12:24])      # fresh-episode joint positions (q - default)
            assert bool((obs[:, 36:48] == 0).all())                # and a cleared last action
    assert resets >= 2 * E
    # the last targets written are default + scale * action (the last step reset no env: 45 is not a multiple of 20)
    env.world.synchronize()
    targets = env.world.download(F.DRIVE_TARGET)
    want = env.default_targets.cpu().numpy()[:, 1:] + env.action_scale * actions.cpu().numpy()
    assert np.allclose(targets[:, 1:], want, atol=1e-6)
    assert torch.equal(obs[:, 36:48], actions)                      # the record carries the action just applied
    env.close()


def test_joint_order_permutes_observations_and_actions(device):
    """Caller joint i is library slot joint_order[i] on the way out, and actions go back through the inverse map
    (python/nuka/tasks/go2_obs.py:252-262, 307-325)."""
    torch = pytest.importorskip("torch")
    E = 8
    order = [3, 4, 5, 0, 1, 2, 9, 10, 11, 6, 7, 8]
    env = NukaVecEnv(device, T.quadruped(0).blob(), E, joint_order=order)
    plain = NukaVecEnv(device, T.quadruped(0).blob(), E)
    o1, o0 = env.reset(), plain.reset()
    assert torch.equal(o1[:, :12], o0[:, :12])
    a = 0.3 * torch.randn((E, 12), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    inverse = torch.empty(12, dtype=torch.long); inverse[torch.tensor(order)] = torch.arange(12)
    o1 = env.step(a)[0]
    o0 = plain.step(a[:, inverse.cuda()])[0]                # the same physical targets in the library's own order
    env.world.synchronize(); plain.world.synchronize()
    assert torch.equal(o1[:, 12:24], o0[:, 12:24][:, order]) and torch.equal(o1[:, 24:36], o0[:, 24:36][:, order])
    env.close(); plain.close()


def test_fallen_envs_terminate_and_restart(device):
    torch = pytest.importorskip("torch")
    E = 16
    env = NukaVecEnv(device, T.quadruped(0).blob(), E, termination_height=0.5)       # standing height is below 0.5: all fall
    env.reset()
    obs, reward, terminated, truncated, info = env.step(torch.zeros((E, 12), device="cuda"))
    assert bool(terminated.all()) and int(info["done"].sum()) == E
    assert int(env.episode_steps.max()) == 0
    env.close()


class OwnReward(NukaVecEnv):
    """A task with a reward of its own: its loop runs as tensor operations."""

    def compute_reward(self):
        return super().compute_reward()


# one env, an odd batch, more than one block of every kernel; actions beyond the clip and not a number, ends by fall and by length
@pytest.mark.parametrize("E,order", [(1, None), (37, [3, 4, 5, 0, 1, 2, 9, 10, 11, 6, 7, 8]), (1031, None)])
def test_episode_pass_equals_the_tensor_operations(device, E, order):
    torch = pytest.importorskip("torch")
    make = lambda kind: kind(device, T.quadruped(0).blob(), E, decimation=3, episode_length_s=0.12, joint_order=order)
    envs = make(NukaVecEnv), make(OwnReward)
    launches = []
    for env in envs:
        env.reset()
        env.episode_steps.copy_(torch.arange(E, device="cuda") % 5)
    gen = torch.Generator(device="cuda").manual_seed(E)
    for k in range(12):
        actions = 0.5 * torch.randn((E, 12), generator=gen, device="cuda")
        actions[::5, 3] = 150.0
        actions[k % E, 7] = float("nan")
        before = [env.world.launch_count() for env in envs]
        (obs, reward, *flags, info), (obs1, reward1, *flags1, info1) = (env.step(actions) for env in envs)
        launches.append([env.world.launch_count() - n for env, n in zip(envs, before)])
        assert torch.equal(torch.nan_to_num(obs, 7.0), torch.nan_to_num(obs1, 7.0)) and obs is not envs[0].obs
        assert torch.allclose(reward, reward1, rtol=1e-6, atol=1e-6, equal_nan=True)         # an ulp of exp
        for a, b in zip(flags + [info["done"]], flags1 + [info1["done"]]):
            assert a.dtype == torch.bool and torch.equal(a, b)
        for name in ("obs", "last_action", "episode_steps", "_targets", "_base"):
            assert torch.equal(torch.nan_to_num(getattr(envs[0], name), 7.0), torch.nan_to_num(getattr(envs[1], name), 7.0)), (k, name)
    assert all(a == b + 2 for a, b in launches)               # both forms count the world's launches: actions and verdicts are two more
    for env in envs:
        env.close()


@pytest.mark.parametrize("where", ["class", "object", "subclass"])
def test_a_replaced_reward_is_the_one_that_is_paid(device, monkeypatch, where):
    torch = pytest.importorskip("torch")
    mine = lambda self: self._base[:, 2] + 7.0
    kind = type("Task", (NukaVecEnv,), {"compute_reward": mine}) if where == "subclass" else NukaVecEnv
    env = kind(device, T.quadruped(0).blob(), 5, decimation=2)
    env.reset()
    if where == "class":
        monkeypatch.setattr(NukaVecEnv, "compute_reward", mine)
    elif where == "object":
        env.compute_reward = mine.__get__(env)
    reward = env.step(torch.zeros((5, 12), device="cuda"))[1]
    assert torch.equal(reward, mine(env))                            # no env ended: the base is where the reward saw it
    env.close()


@pytest.mark.parametrize("where", ["class", "object"])
def test_replaced_methods_of_the_world_are_called(device, monkeypatch, where):
    torch = pytest.importorskip("torch")
    env, calls = NukaVecEnv(device, T.quadruped(0).blob(), 3), []
    env.reset()
    for name in ("step_n", "reset_envs_masked", "pack_observations"):
        stock = getattr(type(env.world), name)
        watched = lambda world, *args, stock=stock, name=name: (calls.append(name), stock(world, *args))[1]
        if where == "class":
            monkeypatch.setattr(type(env.world), name, watched)
        else:
            setattr(env.world, name, watched.__get__(env.world))
    env.step(torch.zeros((3, 12), device="cuda"))
    assert calls == ["step_n", "reset_envs_masked", "pack_observations"]
    env.close()


# a value per joint or per env, a device scalar, a float where a count is usual, numpy numbers, a length past 32 bits
@pytest.mark.parametrize("name,make", [("action_scale", lambda t: t.linspace(0.1, 0.4, 12, device="cuda")), ("action_scale", lambda t: t.tensor(0.3, device="cuda")),
                                       ("action_scale", lambda t: np.float32(0.25)), ("termination_height", lambda t: t.linspace(0.1, 0.4, 6, device="cuda")),
                                       ("min_up", lambda t: t.full((6,), 0.9999, device="cuda")), ("max_episode_length", lambda t: 2.0),
                                       ("max_episode_length", lambda t: np.int64(2)), ("max_episode_length", lambda t: 1 << 40),
                                       ("max_episode_length", lambda t: t.arange(6, device="cuda"))])
def test_settings_that_are_no_plain_numbers(device, name, make):
    torch = pytest.importorskip("torch")
    envs = [kind(device, T.quadruped(0).blob(), 6, decimation=2) for kind in (NukaVecEnv, OwnReward)]
    for env in envs:
        env.reset()
        setattr(env, name, make(torch))
    gen = torch.Generator(device="cuda").manual_seed(5)
    for _ in range(3):
        actions = 0.5 * torch.randn((6, 12), generator=gen, device="cuda")
        (obs, reward, *flags, info), (obs1, reward1, *flags1, info1) = (env.step(actions) for env in envs)
        assert torch.equal(obs, obs1) and torch.equal(reward, reward1)
        assert all(torch.equal(a, b) for a, b in zip(flags + [info["done"]], flags1 + [info1["done"]]))
    for env in envs:
        env.close()


def test_episode_steps_refuse_what_does_not_fit(device):
    """Each refusal of the library's episode pass, with nothing launched and nothing written."""
    torch = pytest.importorskip("torch")
    env = NukaVecEnv(device, T.quadruped(0).blob(), 4)
    env.reset()
    world, width = env.world, env.obs_width
    actions = torch.zeros((4, 12), device="cuda")                    # the desc holds addresses only
    desc = env._episode_desc(actions)
    out, copy, flags = torch.full((4, width), 3.0, device="cuda"), torch.full((4, width), 3.0, device="cuda"), torch.zeros((4, 4), device="cuda")
    desc.reward, desc.terminated, desc.truncated, desc.done = (row.data_ptr() for row in flags)
    before, observed = world.launch_count(), {name: getattr(env._obs_desc, name) for name in ("command", "command_stride", "reward", "row_stride", "clip")}
    refused = lambda code=nuka._abi.INVALID_ARG: pytest.raises(nuka.NukaError, check=lambda e: e.code == code)
    for name in ("actions", "last_action", "default_position", "joint_order", "default_targets", "command", "episode_steps", "reward", "terminated", "truncated",
                 "done", "done_mask"):
        kept = getattr(desc, name)
        setattr(desc, name, None)
        with refused():
            world.episode_step(desc, env._obs_desc, 1, out, copy)
        setattr(desc, name, kept)
    for name, value in (("command", None), ("command_stride", 2), ("reward", flags.data_ptr()), ("row_stride", width + 1), ("clip", -1.0)):
        setattr(env._obs_desc, name, value)
        with refused():
            world.episode_step(desc, env._obs_desc, 1, out, copy)
        setattr(env._obs_desc, name, observed[name])
    for pair in ((out[:3], copy), (out, copy[:3]), (out.view(-1)[:-1], copy)):
        with refused():
            world.episode_step(desc, env._obs_desc, 1, *pair)
    for wrong in (copy.double(), copy.int(), copy.cpu(), torch.zeros((4, 2 * width), device="cuda")[:, ::2]):
        for pair in ((wrong, copy), (out, wrong)):
            with pytest.raises(ValueError):
                world.episode_step(desc, env._obs_desc, 1, *pair)
    arm = nuka.World.create_from_template(device, T.arm7(0).blob(), 4)
    with refused(nuka._abi.NOT_SUPPORTED):
        arm.episode_step(desc, env._obs_desc, 1, out, copy)
    env.world.synchronize()
    torch.cuda.synchronize()
    assert world.launch_count() == before and bool((out == 3.0).all()) and bool((copy == 3.0).all())
    world.episode_step(desc, env._obs_desc, 1, out, copy)
    env.world.synchronize()
    assert world.launch_count() > before and torch.equal(out, copy) and not bool((out == 3.0).any())
    arm.destroy()
    env.close()
