"""raf.op.lans without a tensor list (rafb200_lans_many): one block per tensor up to 16384 elements, three
launches above, 512 tensors a launch.  Against the oracle, at the 1e-5 that sums of squares in fp32
allow for LANS, and against the persistent kernel, whose arithmetic is the same but for the order
of the sums."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from raf_b200 import _lib, op
from tests.util import rel_err, to_numpy

gpu = pytest.mark.gpu

LISTS = {
    "one": [1],
    "block": [1, 3, 4, 127, 128, 4095, 4096, 4097, 16383, 16384],
    "phases": [16385, 1, 2047, 2048, 2049, 4096],
    "many": [5 + i % 300 for i in range(513)],
    "many_large": [17000] + [1 + i % 40 for i in range(600)],
    "empty_among": [0, 10, 0, 20000, 0],
}


def _lists(sizes, shift, seed):
    rng = np.random.default_rng(seed)
    host = [[(rng.standard_normal(n) * s).astype(np.float32) for n in sizes] for s in (1e-2, 0.1, 1e-3)]
    host.append([(1e-6 * (0.5 + rng.random(n))).astype(np.float32) for n in sizes])

    def place(x):  # `shift` elements past an allocation's start
        buf = torch.zeros(x.size + shift, device="cuda")
        buf[shift:] = torch.from_numpy(x).cuda()
        return buf[shift:]

    return host, [[place(x) for x in xs] for xs in host]


@gpu
@pytest.mark.parametrize("mode,normalize", [(1, True), (0, True), (1, False)])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("name", list(LISTS))
def test_lans_rows_match_oracle_and_list_kernel(name, shift, mode, normalize):
    sizes = LISTS[name]
    host, dev = _lists(sizes, shift, 3)
    other = [[t.clone() for t in ts] for ts in dev]
    args = (7, 1e-3, 0.9, 0.999, 1e-6, 1, 0.01, 1, mode, normalize)
    assert _lib.ops().lans(sum(dev, []), *args) is True
    full = [i for i, n in enumerate(sizes) if n]
    O.lans(*[[xs[i] for i in full] for xs in host], 7, 1e-3, 0.9, 0.999, 1e-6, 1, 0.01, 1, mode, int(normalize), 1.0)
    tl = op.TensorList(sizes, torch.float32, torch.float32)
    tl.bind(*other)
    op.lans_list_(tl, *args)
    op.lans_status(tl)
    for what in (1, 2, 3):
        for i in full:
            assert rel_err(to_numpy(dev[what][i]), host[what][i]) < 1e-5, (what, sizes[i])
            assert rel_err(to_numpy(dev[what][i]), to_numpy(other[what][i])) < 1e-5, (what, sizes[i])


@gpu
def test_lans_rows_edge_values():
    # a zero gradient (no normalisation, trust ratio 1) and a zero parameter, in both forms
    for n in (100, 20000):
        g, p, m, v = ([torch.zeros(n, device="cuda"), torch.full((n,), 0.5, device="cuda")] for _ in range(4))
        hg, hp, hm, hv = ([to_numpy(x).copy() for x in xs] for xs in (g, p, m, v))
        op.lans(g + p + m + v, 1, 1e-3, 0.9, 0.999, 1e-6, 1, 0.01, 1, 1, True)
        O.lans(hg, hp, hm, hv, 1, 1e-3, 0.9, 0.999, 1e-6, 1, 0.01, 1, 1, 1, 1.0)
        for a, b in zip(p + m + v, hp + hm + hv):
            assert rel_err(to_numpy(a), b) < 1e-5


@gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", ["block", "phases"])
def test_lans_rows_without_eps(name, mode):
    """eps = 0: lanes past the end of a tensor hold zeros, whose directions 0 / 0 belong to no sum."""
    sizes = LISTS[name] + [17408, 24577]
    host, dev = _lists(sizes, 0, 5)
    args = (7, 1e-3, 0.9, 0.999, 0.0, 1, 0.01, 1, mode, True)
    other = [[t.clone() for t in ts] for ts in dev]
    assert _lib.ops().lans(sum(dev, []), *args) is True
    tl = op.TensorList(sizes, torch.float32, torch.float32)
    tl.bind(*other)
    op.lans_list_(tl, *args)
    op.lans_status(tl)
    O.lans(*host, *args[:-1], 1, 1.0)
    for what in (1, 2, 3):
        for a, c, b in zip(dev[what], other[what], host[what]):
            assert rel_err(to_numpy(a), b) < 1e-5 and rel_err(to_numpy(c), b) < 1e-5, (what, b.size)


# A learning rate, a decay and an eps of the size at which every term of the update moves p by far more than 1e-5.
BOLD = dict(step=7, lr=1.0, beta1=0.9, beta2=0.999, eps=1e-3, bias_correction=1, weight_decay=0.3, grad_averaging=1,
            mode=1, normalize_grad=1)
BOLD_SIZES = [3, 1000, 16384, 20000]


def _bold_host():
    rng = np.random.default_rng(11)
    host = [[(rng.standard_normal(n) * s).astype(np.float32) for n in BOLD_SIZES] for s in (1e-2, 0.1, 1e-3)]
    return host + [[(1e-6 * (0.5 + rng.random(n))).astype(np.float32) for n in BOLD_SIZES]]


@gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("bias_correction", [0, 1])
@pytest.mark.parametrize("grad_averaging", [0, 1])
@pytest.mark.parametrize("count", [3, 4])  # without the 20000 elements: one block per tensor
def test_lans_rows_every_term(mode, bias_correction, grad_averaging, count):
    kw = dict(BOLD, mode=mode, bias_correction=bias_correction, grad_averaging=grad_averaging)
    host = [xs[:count] for xs in _bold_host()]
    dev = [[torch.from_numpy(x.copy()).cuda() for x in xs] for xs in host]
    assert _lib.ops().lans(sum(dev, []), *kw.values()) is True
    O.lans(*host, **kw)
    for what in (1, 2, 3):
        for a, b in zip(dev[what], host[what]):
            assert rel_err(to_numpy(a), b) < 1e-5, (what, b.size)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("other", [dict(weight_decay=0.0), dict(bias_correction=0), dict(grad_averaging=0), dict(lr=1.005),
                                   dict(eps=0.0), dict(beta1=0.899), dict(beta2=0.998), dict(normalize_grad=0),
                                   dict(step=8)])
def test_every_term_shows_in_the_parameters(mode, other):
    """What test_lans_rows_every_term would let pass: the oracle with a term changed, on the same inputs."""
    host, changed = _bold_host(), _bold_host()
    O.lans(*host, **dict(BOLD, mode=mode))
    O.lans(*changed, **dict(BOLD, mode=mode, **other))
    worst = [max(rel_err(a, b) for a, b in zip(changed[what], host[what])) for what in (1, 2, 3)]
    assert worst[0] > 1e-3


@gpu
def test_tied_parameters_and_device_steps_take_the_list_kernel():
    x = [torch.ones(64, device="cuda") for _ in range(4)]
    tied = [x[0], x[0], x[1], x[1], x[2], x[2], x[3], x[3]]
    args = (1e-3, 0.9, 0.999, 1e-6, 1, 0.01, 1, 1, True)
    assert _lib.ops().lans(tied, 1, *args) is None
    assert _lib.ops().lans(x, torch.ones((), device="cuda"), *args) is None
    op.lans(x, torch.ones((), device="cuda"), *args)
