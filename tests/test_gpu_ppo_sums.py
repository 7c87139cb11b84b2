"""The order of the sums in the one-call PPO epoch. The clipped surrogate jumps where a sample's ratio crosses the clipping bound, so that after some hundred minibatches another order of a sum
ends with the actor's first moments percents apart: the kernel keeps one, restated here in numpy, operation by operation, and an epoch is as many minibatches as separate calls, bit for bit."""
import numpy as np
import pytest

import make_golden as mg
from test_gpu_train_step import _net

pytestmark = pytest.mark.gpu
F, D = np.float32, np.float64


def _fma(a, b, c):
    """a * b + c of floats, rounded once: the exact product, the sum rounded to odd, then to float."""
    p, c = a.astype(D) * b.astype(D), np.asarray(c).astype(D)
    s = p + c
    t = s - p
    err = (p - (s - t)) + (c - t)
    odd = np.where((err != 0) & ((s.view(np.int64) & 1) == 0), np.nextafter(s, np.where(err > 0, np.inf, -np.inf)), s)
    return odd.astype(F)


def test_fma_of_the_restatement():
    """Against exact rational arithmetic, with sums that lie at and beside the middle between two floats."""
    from fractions import Fraction
    a = np.array([1 + 2.0 ** -23, 1 + 2.0 ** -12, 3.0, 1.5, -0.3], F)
    b = np.array([1 - 2.0 ** -23, 1 + 2.0 ** -12, 2.0 ** -24, 2.0 ** -24, 7.7], F)
    c = np.array([2.0 ** -60, 2.0 ** -70, 1.0, 1.0, 2.31], F)
    for x, y, z, got in zip(a, b, c, _fma(a, b, c)):
        exact = Fraction(float(x)) * Fraction(float(y)) + Fraction(float(z))
        near = [np.nextafter(got, F(-np.inf)), got, np.nextafter(got, F(np.inf))]
        assert abs(Fraction(float(got)) - exact) == min(abs(Fraction(float(v)) - exact) for v in near)


def _up4(n):
    return (n + 3) // 4 * 4


def _parts(tiles, pieces):
    s = 1
    while s < 32 and 2 * s * tiles <= 256 and 2 * s <= pieces:
        s *= 2
    return s


def _added(parts):
    total = parts[0]
    for p in parts[1:]:
        total = total + p
    return total


def _forward(W, b, x, R):
    O, I = W.shape
    pieces, n = I // 4 + 1, _parts(R // 4 * (_up4(O) // 4), (I // 4 + 1) // 2)
    a, w = np.zeros((x.shape[0], 4 * pieces), F), np.zeros((O, 4 * pieces), F)
    a[:, :I], a[:, I], w[:, :I], w[:, I] = x, 1, W, b                    # the bias is a weight of the input 1
    sums = []
    for g in range(n):
        chain = [np.zeros((x.shape[0], O), F) for _ in range(2)]          # even and odd inputs
        for k in range(4 * g, 4 * pieces, 4 * n):
            for i in range(k, k + 4):
                chain[i & 1] = _fma(a[:, i, None], w[None, :, i], chain[i & 1])
        sums.append(chain[0] + chain[1])
    return _added(sums)


def _backward(W, d, R):
    O, I = W.shape
    n = _parts(R // 4 * ((I + 3) // 4), _up4(O) // 4)
    sums = []
    for g in range(n):
        s = np.zeros((d.shape[0], I), F)
        for k in range(4 * g, O, 4 * n):
            for o in range(k, min(k + 4, O)):
                s = _fma(d[:, o, None], W[None, o, :], s)
        sums.append(s)
    return _added(sums)


def _over_teams(tiles, lanes):
    """Sums of the teams ([teams, ...]): thread y of `lanes` those of the teams y, y + lanes, ..., then the threads pairwise, halves first."""
    at = []
    for y in range(lanes):
        s = np.zeros(tiles.shape[1:], F)
        for t in range(y, tiles.shape[0], lanes):
            s = s + tiles[t]
        at.append(s)
    while len(at) > 1:
        at = [p + q for p, q in zip(at[:len(at) // 2], at[len(at) // 2:])]
    return at[0]


def _tiled(v, R, teams):
    """[rows, ...] -> [teams, tiles of a team, R, ...], zeros beyond the rows"""
    n = -(-v.shape[0] // (R * teams))
    out = np.zeros((n * teams * R,) + v.shape[1:], F)
    out[:v.shape[0]] = v
    return out.reshape(n, teams, R, *v.shape[1:]).swapaxes(0, 1)


def _gradients(layers, x, loss, R, teams, lanes):
    """The parameter arena's gradients (layer by layer, weights before biases) for relu hidden layers and a linear last one"""
    inputs, pres = [x], []
    for l, (W, b) in enumerate(layers):
        pres.append(_forward(W, b, inputs[-1], R))
        inputs.append(np.maximum(pres[-1], 0) if l + 1 < len(layers) else pres[-1])
    d, out = loss(inputs[-1]), []
    for l in reversed(range(len(layers))):
        W, b = layers[l]
        ones = np.concatenate([inputs[l], np.ones((x.shape[0], 1), F)], 1)
        dt, at = _tiled(d, R, teams), _tiled(ones, R, teams)
        s = np.zeros((teams, W.shape[0], W.shape[1] + 1), F)
        for k in range(dt.shape[1]):
            for r in range(R):
                s = _fma(dt[:, k, r, :, None], at[:, k, r, None, :], s)
        g = _over_teams(s, lanes)
        out = [g[:, :-1].reshape(-1), g[:, -1]] + out
        if l > 0:
            d = np.where(pres[l - 1] > 0, _backward(W, d, R), F(0))
    return np.concatenate(out)


def _log_density(p):
    """log of the normal density at standard deviation 1, rounded once: p * p and the difference as pairs of floats"""
    c = F(-0.5 * D(F(np.log(D(F(2) * F(3.14159265358979323846))))))
    h = p * p
    lo, hh = _fma(p, p, -h), F(0.5) * h
    d = c - hh
    db = d - c
    de = (c - (d - db)) - (hh + db)
    return d + _fma(np.full_like(lo, -0.5), lo, de)


def _split(net, I, dims):
    p, layers, off = net.params.cpu().numpy(), [], 0
    for O in dims:
        layers.append((p[off:off + O * I].reshape(O, I), p[off + O * I:off + O * I + O]))
        off += O * I + O
        I = O
    return layers


# one tile per team and three; sums in 1 to 16 parts; inputs with the bias in their last piece and in one of its own; patches of each size
@pytest.mark.parametrize("batch,obs,actions,hidden", [(2048, 27, 8, [64, 64]), (150, 27, 3, [64, 64]), (3001, 8, 1, [32, 33]), (40, 5, 6, [16, 12]), (700, 30, 2, [100, 96]), (260, 3, 4, [64, 64]), (150, 3000, 3, [4])])
def test_order_of_the_sums_of_a_minibatch(lib, batch, obs, actions, hidden):
    import torch
    from rl_tools_b200 import ppo
    assert torch.cuda.get_device_properties(0).multi_processor_count == 148
    layout = ppo.DatasetLayout(obs, actions)
    data = mg.det_normal(3, batch * layout.data_dim).reshape(batch, layout.data_dim).astype(F)
    acts = ["relu"] * len(hidden) + ["identity"]
    actor, critic = _net(lib, torch, batch, obs, hidden + [actions], acts, 20, extra=actions), _net(lib, torch, batch, obs, hidden + [1], acts, 30)
    actor.extra("params").fill_(0.0)                                     # standard deviation 1
    ctas = 74
    R = min(32, _up4(-(-batch // ctas)))
    teams = min(ctas, -(-batch // R))

    def lanes(dims):
        n, quads, I = 4, 0, obs
        for O in dims:
            quads += _up4(O) * (I // 4 + 1)
            I = O
        while n < 32 and 2 * n <= teams and 2 * n * quads <= ctas * 256:
            n *= 2
        return n

    x = data[:, layout.observations]
    layers = {net: _split(net, obs, hidden + [last]) for net, last in ((actor, actions), (critic, 1))}
    # the log-probabilities of the dataset are those of the policy: every ratio is exp(0)
    mean = x
    for l, (W, b) in enumerate(layers[actor]):
        mean = _forward(W, b, mean, R)
        if l < len(hidden):
            mean = np.maximum(mean, 0)
    ps = data[:, layout.actions] - mean
    terms, log_prob = _log_density(ps), np.zeros(batch, F)
    for k in range(actions):
        log_prob = log_prob + terms[:, k]
    data[:, layout.action_log_probs] = log_prob
    dl = F(-1) / F(batch) * data[:, layout.advantages]
    value_constant = F(2) / F(batch) * F(0.5)
    want_critic = _gradients(layers[critic], x, lambda v: (v - data[:, layout.target_values, None]) * value_constant, R, teams, lanes(hidden + [1]))
    want_actor = _gradients(layers[actor], x, lambda _: ps * dl[:, None], R, teams, lanes(hidden + [actions]))
    per_row = _tiled(dl[:, None] * (F(-1) + ps * ps), R, teams)
    s = np.zeros((teams, actions), F)
    for k in range(per_row.shape[1]):
        for r in range(R):
            s = s + per_row[:, k, r]
    # the entropy bonus of every sample: a product and a sum, each rounded (at batches that are no power of two the product is not exact)
    entropy = F(0.01)
    want_std = _over_teams(s, 32) + F(batch) * (F(-1) / F(batch) * entropy)

    dataset = torch.from_numpy(data).cuda()
    assert ppo._train_epoch(actor, critic, dataset, layout, 1, batch, epsilon_clip=0.2, entropy_coefficient=float(entropy), advantage_epsilon=1e-8, normalize_advantage=False, learn_action_std=True)
    assert np.array_equal(critic.grads.cpu().numpy(), want_critic)
    got = actor.grads.cpu().numpy()
    assert np.array_equal(got[:-actions], want_actor)
    assert np.array_equal(got[-actions:], want_std)


@pytest.mark.parametrize("batch,minibatches,obs,actions,hidden", [(2048, 64, 27, 8, 64), (97, 130, 5, 3, 32), (3001, 5, 18, 4, 64)])
def test_an_epoch_is_its_minibatches(lib, batch, minibatches, obs, actions, hidden):
    """An epoch hands the parameters on inside the kernel and keeps the moments in registers; a call per minibatch reads and writes the arenas. The same bits, with ratios on both sides of the
    clipping bound."""
    import torch
    from rl_tools_b200 import ppo
    layout = ppo.DatasetLayout(obs, actions)
    rows = batch * minibatches
    data = mg.det_normal(7, rows * layout.data_dim).reshape(rows, layout.data_dim).astype(F)
    data[:, layout.action_log_probs] = data[:, layout.action_log_probs] * F(0.5) - actions
    dataset = torch.from_numpy(data).cuda()
    acts = ["tanh", "tanh", "identity"]
    nets = [[_net(lib, torch, batch, obs, [hidden, hidden, actions], acts, 20, extra=actions), _net(lib, torch, batch, obs, [hidden, hidden, 1], acts, 30)] for _ in range(2)]
    options = dict(epsilon_clip=0.2, entropy_coefficient=0.01, advantage_epsilon=1e-8, normalize_advantage=True, learn_action_std=True)
    assert ppo._train_epoch(*nets[0], dataset, layout, minibatches, batch, **options)
    for k in range(minibatches):
        assert ppo._train_epoch(*nets[1], dataset[k * batch:(k + 1) * batch], layout, 1, batch, **options)
    for got, want in zip(*nets):
        for name in ("params", "m", "v", "grads", "adam_state"):
            assert torch.equal(getattr(got, name), getattr(want, name)), name
