"""LANS where an overflowed gradient (or a state that is no number any more) makes the norms infinite or NaN:
the step has to end with the oracle's values, infinities and NaN in the same places."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from raf_b200 import _lib, op
from tests.util import rel_err, to_numpy, to_torch

pytestmark = pytest.mark.gpu

HYPER = (7, 1e-3, 0.9, 0.999, 1e-6, 1, 0.01, 1)


def inputs(sizes, what, value, g_dtype="float32"):
    rng = np.random.default_rng(len(sizes) + sizes[0])
    host = [[(rng.standard_normal(n) * s).astype(np.float32) for n in sizes] for s in (1e-2, 0.1, 1e-3)]
    host.append([(1e-6 * (0.5 + rng.random(n))).astype(np.float32) for n in sizes])
    for i, x in enumerate(host[what]):  # one element of every other tensor
        if i % 2 == 0:
            x[x.size // 3] = value
    host[0] = [x.astype(np.float16) if g_dtype == "float16" else x for x in host[0]]
    return host, [[to_torch(x, g_dtype if j == 0 else "float32") for x in xs] for j, xs in enumerate(host)]


def assert_same(got, want):
    got, odd = to_numpy(got), ~np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[odd & ~np.isnan(want)], want[odd & ~np.isnan(want)])  # the infinities
    assert odd.all() or rel_err(got[~odd], want[~odd]) < 1e-5


def oracle_step(host, mode, normalize):
    with np.errstate(all="ignore"):
        O.lans(*host, *HYPER, mode, int(normalize), 1.0)


# every tensor parked; odd sizes; one beyond the parking room (148 x 29 x 5/8 chunks of 1024 elements)
@pytest.mark.parametrize("sizes", [[1000], [4096, 4095, 20001], [3_000_001]])
@pytest.mark.parametrize("what,value", [(0, np.inf), (0, np.nan), (1, np.inf), (2, -np.inf), (2, np.nan), (3, np.inf), (3, np.nan)])
@pytest.mark.parametrize("mode,normalize,g_dtype", [(1, True, "float32"), (0, False, "float32"), (1, True, "float16")])
def test_list_kernel(sizes, what, value, mode, normalize, g_dtype):
    host, dev = inputs(sizes, what, value, g_dtype)
    tl = op.TensorList(sizes, g_dtype, torch.float32)
    tl.set_wait_limit(500)
    tl.bind(*dev)
    op.lans_list_(tl, *HYPER, mode, normalize)
    op.lans_status(tl)
    oracle_step(host, mode, normalize)
    for j in (1, 2, 3):
        for a, b in zip(dev[j], host[j]):
            assert_same(a, b)
    tl.close()


@pytest.mark.parametrize("sizes", [[1000], [4096, 4095, 16384], [4096, 4095, 20001]])  # one block a tensor; three launches
@pytest.mark.parametrize("what,value", [(0, np.inf), (0, np.nan), (1, np.inf), (2, -np.inf), (2, np.nan), (3, np.inf), (3, np.nan)])
@pytest.mark.parametrize("mode,normalize", [(1, True), (0, False)])
def test_without_a_list(sizes, what, value, mode, normalize):
    host, dev = inputs(sizes, what, value)
    assert _lib.ops().lans(sum(dev, []), *HYPER, mode, normalize) is True
    oracle_step(host, mode, normalize)
    for j in (1, 2, 3):
        for a, b in zip(dev[j], host[j]):
            assert_same(a, b)
