"""The PLAIN matched filter with several lanes per output: its results do not depend on
how many lanes share one, to the bit.  A call of many outputs takes one lane each; its
first rows or columns alone take 4, 8 or 32."""
import numpy as np
import pytest
import torch

from benchkit import scenes
from gpu_helpers import mf_backward, mf_forward

pytestmark = pytest.mark.gpu


# outputs that take 32, 8, 4 lanes and one (148 SMs), with remainders of the blocks
@pytest.mark.parametrize("S", [5, 16, 33, 70])
def test_forward_bits_do_not_depend_on_the_lanes(cuda, S):
    rng = np.random.default_rng(S)
    tx, rx = scenes.virtual_array(1)
    ch = scenes.chirp(S)
    re, im = rng.standard_normal((2, tx.shape[0], S)).astype(np.float32)
    vox = rng.uniform((-0.1, -0.1, 0.3), (0.1, 0.1, 0.5), (160001, 3)).T.astype(np.float32)
    run = lambda n: mf_forward(re, im, tx, rx, np.ascontiguousarray(vox[:, :n]), ch.adc_sample_rate, ch.As_sci, "plain")
    full = run(vox.shape[1])
    for n in (1, 257, 9001, 20003, 40001):
        for got, ref in zip(run(n), full):
            np.testing.assert_array_equal(got, ref[:n])


@pytest.mark.parametrize("N", [1, 15, 16, 33, 300])
def test_backward_bits_do_not_depend_on_the_lanes(cuda, N):
    rng = np.random.default_rng(N)
    tx, rx = scenes.virtual_array(15)
    S = 70
    ch = scenes.chirp(S)
    vox = rng.uniform((-0.1, -0.1, 0.3), (0.1, 0.1, 0.5), (N, 3)).T.astype(np.float32).copy()
    gr, gi = rng.standard_normal((2, N)).astype(np.float32)
    run = lambda a: mf_backward(gr, gi, tx[:a], rx[:a], vox, a, S, ch.adc_sample_rate, ch.As_sci, "plain")
    full = run(2700)  # 189000 outputs
    for a in (1, 64, 128, 512):  # a power of two antennas: dividing by them is exact
        for got, ref in zip(run(a), full):
            np.testing.assert_allclose(got * a, ref[:a] * 2700, rtol=2e-7, atol=0)


# rows of several steps of terms, and rows that leave no room in shared memory to exchange terms
@pytest.mark.parametrize("S", [128, 300, 11500])
def test_forward_bits_on_long_rows(cuda, S):
    rng = np.random.default_rng(S)
    tx, rx = scenes.virtual_array(1)
    tx, rx = tx[:3], rx[:3]
    ch = scenes.chirp(S)
    re, im = rng.standard_normal((2, 3, S)).astype(np.float32)
    vox = rng.uniform((-0.1, -0.1, 0.3), (0.1, 0.1, 0.5), (160001, 3)).T.astype(np.float32)
    run = lambda n: mf_forward(re, im, tx, rx, np.ascontiguousarray(vox[:, :n]), ch.adc_sample_rate, ch.As_sci, "plain")
    full = run(vox.shape[1])
    for n in (257, 9001, 20003, 40001):
        for got, ref in zip(run(n), full):
            np.testing.assert_array_equal(got, ref[:n])


# outputs in the middle of the range that takes 8 lanes (64 to 192 per SM), voxels in whole steps and not
@pytest.mark.parametrize("N", [16, 33, 64, 300])
def test_backward_bits_with_eight_lanes(cuda, N):
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    A, S = 256, sms // 2
    rng = np.random.default_rng(N)
    tx, rx = scenes.virtual_array(18)
    ch = scenes.chirp(S)
    vox = rng.uniform((-0.1, -0.1, 0.3), (0.1, 0.1, 0.5), (N, 3)).T.astype(np.float32).copy()
    gr, gi = rng.standard_normal((2, N)).astype(np.float32)
    run = lambda a: mf_backward(gr, gi, tx[:a], rx[:a], vox, a, S, ch.adc_sample_rate, ch.As_sci, "plain")
    full = run(2048 + A)  # one lane each
    for got, ref in zip(run(A), full):
        np.testing.assert_allclose(got * A, ref[:A] * (2048 + A), rtol=2e-7, atol=0)
