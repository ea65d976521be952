"""Several training steps in one call.  Within a call a step's launches are let in while the step before still
runs, its samples are drawn before that step's update and its scratch is the one that step used; a call of one
step has none of that.  So the steps of one call are compared, bit for bit, with the same steps made by a call
each: the sums of a step do not depend on the order of the blocks, and a call of one step takes the rate it is
given as it is.  Batches: one part of the weight gradient, several, more than there are parts."""
import ctypes as C
import ctypes.util

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f = np.float32


def rate(lr, k, steps):
    """The learning rate of step k of a call: lr (0.1 + 0.45 (1 + cos(pi k / steps))) in FP32."""
    libm = C.CDLL(ctypes.util.find_library("m") or "libm.so.6")
    libm.cosf.restype, libm.cosf.argtypes = C.c_float, [C.c_float]
    c = f(libm.cosf(float(f(3.14159265) * f(k) / f(steps))))
    return f(lr) * (f(0.1) + f(0.45) * (f(1.0) + c))


def network(ctx, pool, weight=1.0):
    from tressfx_gb300.api import NeuralSDF
    lo, hi = np.array([-0.2, 1.3, -0.25]), np.array([0.25, 1.8, 0.2])
    rng = np.random.default_rng(pool)
    samples = np.zeros((pool, 8), f)
    samples[:, :3] = rng.uniform(lo, hi, (pool, 3))
    samples[:, 3] = rng.uniform(-3.0, 3.0, pool)
    samples[:, 4:7] = rng.uniform(-0.6, 0.6, (pool, 3))
    samples[:, 7] = weight
    nsdf = NeuralSDF(ctx, lo, hi, cell_size=0.004, pose_scale=1.0 / 0.7, seed=29, max_samples=pool, max_eval_samples=0)
    nsdf.set_samples(0, samples)
    return nsdf


@pytest.mark.parametrize("batch,steps", [(512, 40), (1536, 23), (8192, 40), (33280, 12)])
def test_steps_of_one_call_equal_single_steps(ctx, batch, steps):
    assert rate(1.0, 0, 1) == f(1.0)
    got = []
    for single in (False, False, True):
        nsdf = network(ctx, 5003)
        if single:
            for k in range(steps):
                nsdf.train(1, batch=batch, lr=float(rate(1e-3, k, steps)))
        else:
            nsdf.train(steps, batch=batch, lr=1e-3)
        got.append((nsdf.params().view(np.uint32), nsdf.gradients().view(np.uint32)))
        nsdf.close()
    for w, g in got[1:]:
        assert np.array_equal(got[0][0], w)
        assert np.array_equal(got[0][1], g)


def test_gradient_is_the_rounded_sum_of_its_parts(ctx):
    """A step's gradient is the sum of one part per 512 samples.  A part by itself is the gradient of the same step
    with the weight of every other part's samples zero (their terms are exact zeros; samples that two parts draw
    are left out of both).  The whole gradient is the 64-bit sum of the parts, rounded: parameter by parameter, but
    for sums within the carried error's own rounding (2^-44 or so) of a rounding boundary, of which 20,000
    parameters hold none to speak of."""
    import nsdf_ref as R
    batch, pool, seed = 4608, 1 << 20, 29
    drawn = R.drawn_samples(seed, 1, batch, pool).reshape(-1, 512)
    count = np.zeros(pool, np.int64)
    for d in drawn:
        count[np.unique(d)] += 1
    shared = count > 1

    def gradient(parts):
        nsdf = network(ctx, pool, weight=np.isin(np.arange(pool), drawn[parts]) & ~shared)
        nsdf.train(1, batch=batch, lr=1e-3)
        g = nsdf.gradients()
        nsdf.close()
        return g

    exact = sum(gradient([k]).astype(np.float64) for k in range(len(drawn)))
    whole = gradient(list(range(len(drawn))))
    assert np.count_nonzero(whole) > 15000
    assert np.count_nonzero(whole != exact.astype(f)) <= 2
    ulp = np.spacing(np.abs(whole)).astype(np.float64)
    assert (np.abs(whole - exact) <= 0.5001 * ulp).all()


@pytest.mark.parametrize("batch,digest", [
    (512, "fd0d026164a943451bef625650d19f591780f039e1bb7506a8ab8f77d0880f3b"),
    (1024, "5c67298a3a14a3aefa36fdb376ba654a83e692f453d61b351a9fd33e3ee4c3dc")])
def test_training_of_up_to_two_parts_is_as_ever(ctx, batch, digest):
    """One part, and two (whose sum has no order), gave the same bits in every run when the parts were added by
    atomics too: the digest is of that version's weights and gradients after 40 steps."""
    import hashlib
    nsdf = network(ctx, 5003)
    nsdf.train(40, batch=batch, lr=1e-3)
    h = hashlib.sha256(nsdf.params().tobytes() + nsdf.gradients().tobytes()).hexdigest()
    nsdf.close()
    assert h == digest
