"""What a program that uses this framework has it do, as a list of measurable cases.

    listed()              the cases: the smallest calls, the ordinary ones and the largest of each part of the path
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   what the program holds before the call: networks, runner states, datasets, captured graphs
    run(state)            one pass through the public entry points
    work(case)            bytes and floating-point operations that the pass cannot do without
    tolerance(case)       how far two correct fp32 implementations may be apart

The kinds: `evaluate` (inference), `train` (forward, loss gradient, backward, optimizer step), `rollout` (actor inference fused with the
environment step; on the device or, with host = True, into the caller's host buffers), `ppo_loop` (collect, advantages, epochs of
minibatch updates), `ppo_update` (the update alone on a given dataset), `sac_loop` (runner step, replay sampling, critic and actor updates).
"""
import importlib
import math

import torch

pkg = importlib.import_module("rl-tools_b200")
loops = importlib.import_module("rl-tools_b200.loops")
parallel = importlib.import_module("rl-tools_b200.parallel")
ppo = importlib.import_module("rl-tools_b200.ppo")

ENVS = {"pendulum": (pkg.ENV_PENDULUM, 3, 2, 2), "acrobot_swingup": (pkg.ENV_ACROBOT_SWINGUP, 6, 4, 2), "acrobot": (pkg.ENV_ACROBOT, 6, 4, 4),
        "l2f": (None, 18, 23, 0)}                                    # id, observation, state and reset dimensions
ACTIONS = {"pendulum": 1, "acrobot_swingup": 1, "acrobot": 1, "l2f": 4}

# a 31 g quadrotor (the parameter set of the framework's quadrotor tests): dynamics in the order of L2fParameters, reward and termination
# constants, distribution of the initial states
_ARM, _THRUST, _UP = 0.028, [0.00352526, 0.01437313, 0.09223048], [0.0, 0.0, 1.0]
L2F_DYNAMICS = ([_ARM, -_ARM, 0.0, -_ARM, -_ARM, 0.0, -_ARM, _ARM, 0.0, _ARM, _ARM, 0.0] + _UP * 4 + [0.0, 0.0, -1.0, 0.0, 0.0, 1.0] * 2 + _THRUST * 4 + [0.004665] * 4 +
                [0.05545454] * 4 + [0.24939394] * 4 + [0.0306, 0.0, 0.0, -9.81] + [9.416557e-06, 0.0, 0.0, 0.0, 9.644052e-06, 0.0, 0.0, 0.0, 1.7459517e-05] +
                [106195.93, 0.0, 0.0, 0.0, 103690.86, 0.0, 0.0, 0.0, 57275.352] + [0.72613895, 0.0, 1.0])
L2F_MDP = [0.0, 1.0, 0.5, -100.0, 1.0, 0.0, 0.1, 0.0, 0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0, 1.0, 2.0, 35.0]
L2F_INIT = [0.1, 0.5, 1.5707964, 1.0, 1.0, 1.0, -1.0, 0.0, 0.0, 0.0, 0.0, 0.0]


def listed():
    return [
        # a policy asked for the actions of one batch of observations: the smallest call, all launch and host time
        dict(name="evaluate_actor_256", kind="evaluate", input=3, hidden=64, depth=2, output=2, act="relu", out_act="identity", batch=256),
        # bulk inference of the wide network: the largest forward pass
        dict(name="evaluate_wide_1048576", kind="evaluate", input=64, hidden=256, depth=3, output=16, act="relu", out_act="identity", batch=1048576),
        # one critic regression step at the batch size of the off-policy algorithms
        dict(name="train_critic_256", kind="train", input=4, hidden=256, depth=2, output=1, act="relu", out_act="identity", batch=256, chunks=1),
        # an ordinary supervised step with sizes that fit no tile: odd batch and input, a width that is no power of two, tanh
        dict(name="train_ragged_5003", kind="train", input=33, hidden=200, depth=2, output=7, act="tanh", out_act="identity", batch=5003, chunks=1),
        # the data-parallel training step of the wide network on one GPU's chunk of rows: the largest step
        dict(name="train_wide_1048576", kind="train", input=64, hidden=256, depth=3, output=16, act="relu", out_act="identity", batch=1048576, chunks=1),
        # whole episodes of many environments under a fixed policy: the headline rollout
        dict(name="rollout_pendulum_65536", kind="rollout", env="pendulum", hidden=64, envs=65536, steps=200, limit=200, resets="table", host=False),
        # the same for a caller whose data lives on the host; an odd number of environments
        dict(name="rollout_host_10007", kind="rollout", env="pendulum", hidden=64, envs=10007, steps=200, limit=200, resets="table", host=True),
        # a small evaluation run of another environment with another actor width, odd sizes
        dict(name="rollout_acrobot_1003", kind="rollout", env="acrobot", hidden=32, envs=1003, steps=50, limit=200, resets="table", host=False),
        # the quadrotor's rollout with initial states drawn in the kernel
        dict(name="rollout_l2f_16384", kind="rollout", env="l2f", hidden=64, envs=16384, steps=50, limit=500, resets="device", host=False),
        # the on-policy training loop with its default configuration: everything small, many dependent launches
        dict(name="ppo_loop_64x64", kind="ppo_loop", envs=64, steps=64, batch=512, epochs=10),
        # the update of a locomotion-sized policy: 64 environments x 1024 steps, minibatches of 2048, ten shuffled epochs
        dict(name="ppo_update_27_8", kind="ppo_update", obs=27, actions=8, hidden=64, batch=2048, minibatches=32, envs=64, epochs=10),
        # one step of the off-policy training loop with 256-wide networks at batch 256
        dict(name="sac_loop_256", kind="sac_loop", env="pendulum", hidden=256, batch=256, envs=1),
    ]


def _log(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "train", "train", "train", "rollout", "rollout", "rollout", "ppo_loop", "ppo_update", "sac_loop"])
    if kind in ("evaluate", "train"):
        c = dict(kind=kind, input=_log(rng, 3, 64), hidden=rng.choice([32, 64, 64, 100, 128, 200, 256, 256]), depth=rng.choice([2, 2, 3]), output=_log(rng, 1, 16),
                 act=rng.choice(["relu", "relu", "tanh", "fast_tanh"]), out_act=rng.choice(["identity", "identity", "tanh"]), batch=_log(rng, 32, 1 << 19))
        if kind == "train":
            c["chunks"] = rng.choice([1, 1, 2]) if c["batch"] <= 1 << 17 else 1
        return c
    if kind == "rollout":
        env = rng.choice(["pendulum", "pendulum", "pendulum", "acrobot_swingup", "acrobot", "l2f"])
        hidden = rng.choice([64, 64, 64, 32, 16] if env == "l2f" else [64, 64, 64, 32, 128])
        host = env == "pendulum" and hidden == 64 and rng.random() < 0.25
        resets = "device" if env == "l2f" or (env == "pendulum" and hidden == 64 and not host and rng.random() < 0.5) else "table"
        return dict(kind=kind, env=env, hidden=hidden, envs=_log(rng, 64, 32768 if env == "pendulum" else 16384), steps=_log(rng, 8, 200 if env == "pendulum" else 50),
                    limit=200 if env != "l2f" else 500, resets=resets, host=host)
    if kind == "ppo_loop":
        return dict(kind=kind, envs=8 * _log(rng, 2, 32), steps=0, batch=8 * _log(rng, 16, 256), epochs=rng.choice([2, 4, 10]))
    if kind == "ppo_update":
        return dict(kind=kind, obs=_log(rng, 3, 32), actions=_log(rng, 1, 8), hidden=rng.choice([32, 64, 64]), batch=32 * _log(rng, 8, 128), minibatches=_log(rng, 4, 16),
                    envs=32, epochs=rng.choice([1, 2, 4]))
    return dict(kind=kind, env=rng.choice(["pendulum", "pendulum", "l2f"]), hidden=rng.choice([32, 64, 64, 128, 256]), batch=_log(rng, 64, 512), envs=_log(rng, 1, 32))


# ---- the networks ---------------------------------------------------------------------------------------------------------------------------
def _dims(case):
    return [case["hidden"]] * case["depth"] + [case["output"]]


def _products(inp, dims):
    """sum over the layers of input x output"""
    total = 0
    for d in dims:
        total += inp * d
        inp = d
    return total


def _init(params, inp, dims, gen):
    """weights and biases uniform in +- 1 / sqrt(fan in), the framework's default initialisation"""
    off = 0
    for d in dims:
        n = d * inp + d
        params[off:off + n] = (torch.rand(n, device="cuda", generator=gen) * 2 - 1) / math.sqrt(inp)
        off += n
        inp = d


def _in_training(net, gen, second_moment):
    """optimizer state of a run that is under way: first moments around zero, second moments that have seen larger gradients, age 1000"""
    net.m.copy_(torch.randn(net.m.shape, device="cuda", generator=gen) * (0.1 * math.sqrt(second_moment)))
    net.v.copy_((torch.rand(net.v.shape, device="cuda", generator=gen) + 0.5) * second_moment)
    net.adam_state[0] = 1000


# ---- prepare ----------------------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    torch.manual_seed(seed)
    return _PREPARE[case["kind"]](case, seed, gen)


def _prepare_network(case, seed, gen):
    dims = _dims(case)
    net = pkg.Mlp(case["input"], dims, [case["act"]] * case["depth"] + [case["out_act"]], case["batch"])
    _init(net.params, case["input"], dims, gen)
    rows = case["batch"] * case.get("chunks", 1)
    s = dict(kind=case["kind"], net=net, rows=rows, x=torch.randn((rows, case["input"]), device="cuda", generator=gen))
    if case["kind"] == "train":
        _in_training(net, gen, 1e-7)
        s["y"] = torch.randn((rows, case["output"]), device="cuda", generator=gen)
    return s


def _prepare_rollout(case, seed, gen):
    env, obs, state, reset = ENVS[case["env"]]
    N, T, A, H = case["envs"], case["steps"], ACTIONS[case["env"]], case["hidden"]
    shape = pkg.MlpShape.make(obs, [H, H, A], ["relu", "relu", "tanh"])
    params = torch.zeros(shape.num_params(), device="cuda")
    _init(params, obs, [H, H, A], gen)
    rounds = T // case["limit"] + 1
    table = None
    if case["resets"] == "table":
        table = torch.rand((rounds, N, reset), device="cuda", generator=gen) * 2 - 1
        if case["env"] == "pendulum":
            table[..., 0] *= math.pi
        else:
            table *= 0.1
    host = case["host"]
    new = lambda shape, dtype=torch.float32: torch.zeros(shape, dtype=dtype, pin_memory=True) if host else torch.zeros(shape, dtype=dtype, device="cuda")
    s = dict(kind="rollout", case=case, env=env, shape=shape, params=params, table=table, seed=seed, calls=0, states=new((N, state)), episode_step=new(N, torch.int32),
             truncated=new(N, torch.uint8), episode_return=new(N), obs=new((T * N, obs)), act=new((T * N, A)), rew=new(T * N) if case["env"] == "l2f" else new((T * N, 1)))
    s["truncated"].fill_(1)                                           # every environment starts with a reset
    if host:
        s["params"], s["table"] = params.cpu().pin_memory(), table.cpu().pin_memory()
    else:
        s["error_flag"] = new(1, torch.int32)
    if case["env"] in ("acrobot", "l2f"):
        s["terminated"] = new(T * N, torch.uint8)
    if case["env"] == "l2f":
        s["parameters"] = pkg.L2fParameters.make(L2F_DYNAMICS, 0.01)
    return s


def _prepare_ppo_loop(case, seed, gen):
    loop = loops.PendulumPpoLoop(n_envs=case["envs"], steps_per_env=case["steps"] or case["batch"] // 8, batch_size=case["batch"], n_epochs=case["epochs"], seed=seed,
                                 adam=dict(alpha=3e-4))
    _in_training(loop.actor, gen, 1e-3)
    _in_training(loop.critic, gen, 10.0)                              # returns of minus several hundred: gradients of several units
    return dict(kind="ppo_loop", loop=loop)


def _prepare_ppo_update(case, seed, gen):
    O, A, H, B, N = case["obs"], case["actions"], case["hidden"], case["batch"], case["envs"]
    T = B * case["minibatches"] // N
    layout = ppo.DatasetLayout(O, A)
    acts = ["tanh", "tanh", "identity"]
    actor, critic = pkg.Mlp(O, [H, H, A], acts, B, extra_params=A), pkg.Mlp(O, [H, H, 1], acts, B)
    actor.hyper, critic.hyper = pkg.AdamHyper(alpha=3e-4), pkg.AdamHyper(alpha=3e-4)
    for net, out in ((actor, A), (critic, 1)):
        _init(net.params, O, [H, H, out], gen)
        _in_training(net, gen, 1e-3)
    actor.extra("params").fill_(math.log(0.5))
    rows = (T + 1) * N
    randn = lambda *shape: torch.randn(shape, device="cuda", generator=gen)
    dataset = torch.zeros((rows, layout.data_dim), device="cuda")
    dataset[:, layout.observations] = randn(rows, O)
    mean = torch.cat([actor.evaluate(dataset[b:b + B, layout.observations]) for b in range(0, rows, B)])
    noise = randn(rows, A)
    dataset[:, layout.actions_mean] = mean
    dataset[:, layout.actions] = mean + 0.5 * noise
    dataset[:, layout.action_log_probs] = (-0.5 * noise ** 2 - math.log(0.5) - 0.5 * math.log(2 * math.pi)).sum(1)
    dataset[:, layout.rewards] = randn(rows)
    dataset[:, layout.truncated] = (torch.rand(rows, device="cuda", generator=gen) < 1e-3).float()
    graphs = ppo.MinibatchGraphs(actor, critic, dataset, layout, N * T, B)
    return dict(kind="ppo_update", actor=actor, critic=critic, dataset=dataset, layout=layout, envs=N, steps=T, batch=B, epochs=case["epochs"], graphs=graphs,
                rng=pkg.rng_init_host(seed))


def _prepare_sac_loop(case, seed, gen):
    warm = max(50, -(-case["batch"] // case["envs"]))
    common = dict(n_envs=case["envs"], batch_size=case["batch"], hidden_dim=case["hidden"], step_limit=1 << 30, n_warmup_steps=warm, replay_capacity=10000, seed=seed)
    if case["env"] == "l2f":
        loop = loops.L2fSacLoop(pkg.L2fParameters.make(L2F_DYNAMICS, 0.01), L2F_MDP, L2F_INIT, **common)
    else:
        loop = loops.PendulumSacLoop(**common)
    a = loop.agent
    for net in [a.actor] + a.critics:
        _in_training(net, gen, 1e-5)
    for _ in range(warm + 1):                                         # fills the replay buffers; the step after the warm-up captures the loop's graph
        loop.step()
    return dict(kind="sac_loop", loop=loop)


_PREPARE = dict(evaluate=_prepare_network, train=_prepare_network, rollout=_prepare_rollout, ppo_loop=_prepare_ppo_loop, ppo_update=_prepare_ppo_update, sac_loop=_prepare_sac_loop)


# ---- run --------------------------------------------------------------------------------------------------------------------------------------
def run(s):
    return _RUN[s["kind"]](s)


def _run_evaluate(s):
    return s["net"].evaluate(s["x"])


def _nets(*nets):
    return [t for n in nets for t in (n.params, n.grads, n.m, n.v)]


def _run_train(s):
    net = s["net"]
    parallel.sharded_train_step(pkg, net, s["x"], s["y"], s["rows"])
    return _nets(net) + [net.pre, net.out]


def _run_rollout(s):
    c, T, limit = s["case"], s["case"]["steps"], s["case"]["limit"]
    runner = (s["states"], s["episode_step"], s["truncated"], s["episode_return"])
    out = dict(obs=s["obs"], act=s["act"], rew=s["rew"])
    if c["host"]:
        pkg.pendulum_rollout_host(s["shape"], s["params"], *runner, s["table"], T, **out, step_limit=limit)
    elif c["env"] == "l2f":
        pkg.l2f_rollout_device_rng(s["parameters"], L2F_MDP, L2F_INIT, s["shape"], s["params"], *runner, s["seed"], s["calls"] * T, T, limit, **out, terminated=s["terminated"])
    elif c["env"] == "pendulum" and c["resets"] == "device":
        pkg.pendulum_rollout_device_rng(s["shape"], s["params"], *runner, s["seed"], s["calls"] * T, T, limit, **out, error_flag=s["error_flag"])
    elif c["env"] == "pendulum":
        pkg.pendulum_rollout(s["shape"], s["params"], *runner, s["table"], T, limit, **out, error_flag=s["error_flag"])
    else:
        pkg.env_rollout(s["env"], s["shape"], s["params"], *runner, s["table"], T, limit, **out, error_flag=s["error_flag"], terminated=s.get("terminated"))
    s["calls"] += 1
    return [*runner, s["obs"], s["act"], s["rew"]] + [s[k] for k in ("terminated", "error_flag") if k in s]


def _run_ppo_loop(s):                                                 # gradients and first moments are those of the last minibatch, scratch of the loop
    loop = s["loop"]
    mean_reward = loop.step()
    nets = [t for n in (loop.actor, loop.critic) for t in (n.params, n.v)]
    return nets + [loop.dataset, loop.states, loop.episode_step, loop.truncated, loop.episode_return, mean_reward]


def _run_ppo_update(s):
    actor, critic, dataset, layout, rows = s["actor"], s["critic"], s["dataset"], s["layout"], s["envs"] * s["steps"]
    ppo.evaluate_values(critic, dataset, layout)
    ppo.estimate_generalized_advantages(dataset, layout, s["envs"], s["steps"])
    ppo.train(actor, critic, dataset, layout, rows, s["batch"], n_epochs=s["epochs"], shuffle_rng_state=s["rng"], graphs=s["graphs"])
    return [t for n in (actor, critic) for t in (n.params, n.m, n.v)] + [dataset]


def _run_sac_loop(s):
    loop = s["loop"]
    loop.step()
    a, b = loop.agent, loop.batch
    return (_nets(a.actor, *a.critics) + [t.params for t in a.critics_target] +
            [a.log_alpha, loop.states, loop.actions, loop.episode_step, loop.truncated, b["oa_base"], b["rewards"], b["terminated"]])


_RUN = dict(evaluate=_run_evaluate, train=_run_train, rollout=_run_rollout, ppo_loop=_run_ppo_loop, ppo_update=_run_ppo_update, sac_loop=_run_sac_loop)


# ---- work -------------------------------------------------------------------------------------------------------------------------------------
def _train_work(inp, dims, rows, once=1):
    """One training step of a network on `rows` rows: forward, both backward contractions (no input gradient of the first layer), optimizer.
    forward and backward are separate calls, so pre-activations and outputs are written by one and read by the other."""
    p, acts = _products(inp, dims), sum(dims)
    n = p + acts
    bytes_ = 4 * (rows * (inp + dims[-1]) + rows * (2 * acts + 2 * acts - dims[-1]) + once * 8 * n)
    return bytes_, 2 * rows * (3 * p - inp * dims[0])


def work(case):
    k = case["kind"]
    if k == "evaluate":
        p, dims, B = _products(case["input"], _dims(case)), _dims(case), case["batch"]
        return dict(bytes=4 * (B * (case["input"] + case["output"]) + p + sum(dims)), flops=2 * B * p)
    if k == "train":
        b, f = _train_work(case["input"], _dims(case), case["batch"] * case["chunks"])
        return dict(bytes=b, flops=f)
    if k == "rollout":
        _, obs, state, reset = ENVS[case["env"]]
        A, H, n = ACTIONS[case["env"]], case["hidden"], case["envs"] * case["steps"]
        row = 4 * (obs + A + 1) + (1 if case["env"] in ("acrobot", "l2f") else 0)
        return dict(bytes=n * row + case["envs"] * (8 * state + 17 + 4 * reset), flops=2 * n * _products(obs, [H, H, A]))
    if k == "ppo_loop":
        T = case["steps"] or case["batch"] // 8
        n = case["envs"] * T
        updates = case["epochs"] * (n // case["batch"])
        b, f = _train_work(3, [64, 64, 1], case["batch"])
        p = _products(3, [64, 64, 1])
        return dict(bytes=2 * updates * b + n * 4 * 13 + case["epochs"] * n * 4 * 7 * 2, flops=2 * updates * f + 2 * 2 * n * p)
    if k == "ppo_update":
        O, A, H, n = case["obs"], case["actions"], case["hidden"], case["batch"] * case["minibatches"]
        updates = case["epochs"] * case["minibatches"]
        ba, fa = _train_work(O, [H, H, A], case["batch"])
        bc, fc = _train_work(O, [H, H, 1], case["batch"])
        return dict(bytes=updates * (ba + bc) + case["epochs"] * n * 4 * (O + A + 3) * 2 + n * 4 * (O + 6), flops=updates * (fa + fc) + 2 * n * _products(O, [H, H, 1]))
    O, A = (18, 4) if case["env"] == "l2f" else (3, 1)
    H, B, N = case["hidden"], case["batch"], case["envs"]
    pa, pc = _products(O, [H, H, 2 * A]), _products(O + A, [H, H, 1])
    na, nc = pa + 2 * H + 2 * A, pc + 2 * H + 1
    # runner step, next action, two targets x two critics, two critic steps, actor step through both critics
    flops = 2 * N * pa + 2 * B * pa + 8 * B * pc + 2 * 2 * B * (3 * pc - (O + A) * H) + 2 * B * (3 * pa - O * H) + 2 * 2 * B * 2 * pc
    return dict(bytes=4 * (8 * na + 2 * 8 * nc + 2 * 3 * nc) + 4 * B * (2 * O + A + 3), flops=flops)


def tolerance(case):
    return TOLERANCE[case["kind"]] if case["kind"] != "rollout" else TOLERANCE[case["kind"]][case["env"]]


# evaluate: fp32 sums of up to 256 products. train: gradients are sums over the rows, and the optimizer's update is theirs over a root; the
# largest difference is that of an entry whose terms cancel. rollout: the dynamics carry a step's rounding into the next ones (and
# a step's termination may fall on the other side of its bound). The loops chain
# many optimizer steps (an epoch's minibatches, one after the other), each of which carries the rounding of those before it, and the clipped
# policy gradient jumps where a sample's ratio crosses the clipping bound.
TOLERANCE = dict(evaluate={"rel": 1e-5, "max": 1e-4}, train={"rel": 5e-5, "max": 2e-3},
                 rollout={env: {"rel": 3e-4, "max": 0.1, "differ": 1e-3} for env in ENVS},
                 ppo_loop={"rel": 1e-2, "max": 0.5}, ppo_update={"rel": 1e-2, "max": 0.5}, sac_loop={"rel": 1e-3, "max": 0.1})
