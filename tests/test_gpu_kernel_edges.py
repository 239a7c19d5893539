"""Kernels whose work split depends on sizes or alignment, at the edges of those splits, against the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

import om_binding as omb
from backends import scaled_diff
from om_binding import f32, i32, i64

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K(oracle_built):
    return oracle_built


def normal(seed, *shape, scale=1.0):
    return (np.random.default_rng(seed).standard_normal(shape) * scale).astype(np.float32)


def table(pointers):
    return (C.c_void_p * len(pointers))(*pointers)


class SgdHyper(C.Structure):
    _fields_ = [(n, C.c_float) for n in ("lr", "weight_decay", "momentum", "dampening", "grad_scale")] + [("nesterov", C.c_int32), ("has_momentum", C.c_int32)]


@pytest.mark.parametrize("sizes", [[1, 3, 1023, 1024, 1025, 4099], [8 * 148 * 4096 - 5, 4, 9], [8 * 148 * 4096 + 3, 4097, 2]])
@pytest.mark.parametrize("momentum,nesterov,wd", [(0.0, 0, 0.0), (0.9, 1, 0.1)])
def test_sgd_visits_are_bit_exact(ctx, K, sizes, momentum, nesterov, wd):
    """Edges of the visits (1024 or 4096 elements by the launch's total), their ragged ends, and tensors that start off a
    16-byte boundary (every second one): the bits of the reference's update."""
    shift = [i % 2 for i in range(len(sizes))]
    ps, bufs = ([normal(7 * i + j, n) for i, n in enumerate(sizes)] for j in (0, 1))
    P, B = ([ctx.to_device(np.concatenate([np.zeros(s, np.float32), a])) for a, s in zip(arrs, shift)] for arrs in (ps, bufs))
    at = lambda arrs: table([a.ptr.value + 4 * s for a, s in zip(arrs, shift)])  # noqa: E731
    hyper = SgdHyper(0.05, wd, momentum, 0.1, 1.0, nesterov, int(momentum != 0.0))
    for step in range(2):
        gs = [normal(100 + 7 * i + step, n) for i, n in enumerate(sizes)]
        G = [ctx.to_device(np.concatenate([np.zeros(s, np.float32), a])) for a, s in zip(gs, shift)]
        ctx.call("om_optim_sgd_step", ctx.handle, i32(len(sizes)), at(P), at(G), at(B), omb.int_array([int(step == 0)] * len(sizes)),
                 omb.int_array(sizes, C.c_int64), C.byref(hyper), None)
        for p, g, b in zip(ps, gs, bufs):
            K.sgd_step(p, g, b, step == 0, 0.05, wd, momentum, 0.1, bool(nesterov))
    for i, s in enumerate(shift):
        assert np.array_equal(P[i].numpy()[s:], ps[i]), sizes[i]
        if momentum:
            assert np.array_equal(B[i].numpy()[s:], bufs[i]), sizes[i]
