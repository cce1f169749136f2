"""The MIXED matched filter through range cells, at sizes large enough to take it,
against the FP64 oracle.

Tolerance: the interpolation of the sample sums errs by at most 1.6e-7 per
sample, the hardware sine and cosine by 4e-7, the phase by ~1e-7 cycles
(6e-7 rad), the FP32 sums by a few 1e-7; 2e-6 covers their sum."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from benchkit import scenes
from gpu_helpers import cu, mf_backward, mf_forward
from oracle import rf_oracle as orc

pytestmark = pytest.mark.gpu

TOL = 2e-6


def box_points(rng, n, lo=(-0.1, -0.1, 0.3), hi=(0.1, 0.1, 0.5)):
    return np.ascontiguousarray(rng.uniform(lo, hi, (n, 3)).T.astype(np.float32))


def signal(rng, tx, rx, ch, extent=1.0, snr=20.0):
    pos = rng.uniform((-0.1, -0.1, 0.3), (0.1, 0.1, 0.5), (6, 3)) * extent
    amp = rng.standard_normal(6) + 1j * rng.standard_normal(6)
    return scenes.synthesize_if_numpy(tx, rx, pos.astype(np.float32), amp, ch, snr_db=snr, rng=rng)


def case(seed, A, S, N, shuffle=False, box=None, bandwidth=4e9):
    rng = np.random.default_rng(seed)
    tx, rx = scenes.virtual_array(int(np.ceil(np.sqrt(A / 12))))
    pick = rng.permutation(tx.shape[0])[:A] if shuffle else np.arange(A)
    tx, rx = np.ascontiguousarray(tx[pick]), np.ascontiguousarray(rx[pick])
    ch = scenes.chirp(S, bandwidth=bandwidth)
    re, im = signal(rng, tx, rx, ch)
    return dict(re=re, im=im, tx=tx, rx=rx, ch=ch, vox=box_points(rng, N, *(box or ())), rng=rng)


def oracle(c):
    ch = c["ch"]
    r = orc.mf_forward(c["re"], c["im"], c["tx"], c["rx"], c["vox"], ch.adc_sample_rate, ch.As_sci)
    return r[0] + 1j * r[1]


def forward(c, **kw):
    ch = c["ch"]
    y = mf_forward(c["re"], c["im"], c["tx"], c["rx"], c["vox"], ch.adc_sample_rate, ch.As_sci, "mixed", **kw)
    return y[0] + 1j * y[1]


# (antennas, samples, voxels): remainders of the 8-antenna stages, of the 256-sample
# table tiles, of the 512-voxel blocks; the smallest voxel count; long rows
SHAPES = [(1000, 200, 512), (1001, 199, 513), (131, 33, 24000), (197, 256, 4097), (148, 257, 3000), (132, 1025, 800),
          (130, 4096, 515), (129, 256, 40000)]


@pytest.mark.parametrize("shuffle", [False, True], ids=["mimo_order", "shuffled"])
@pytest.mark.parametrize("A,S,N", SHAPES)
def test_forward_vs_fp64(cuda, A, S, N, shuffle):
    c = case(A + S, A, S, N, shuffle)
    assert rel_l2(forward(c), oracle(c)) < TOL


def backward(c, **kw):
    ch, A, S = c["ch"], c["tx"].shape[0], c["re"].shape[1]
    N = c["vox"].shape[1]
    gr, gi = c["rng"].standard_normal((2, N)).astype(np.float32)
    h = mf_backward(gr, gi, c["tx"], c["rx"], c["vox"], A, S, ch.adc_sample_rate, ch.As_sci, "mixed", **kw)
    r = orc.mf_backward(gr, gi, c["tx"], c["rx"], c["vox"], A, S, ch.adc_sample_rate, ch.As_sci)
    return h[0] + 1j * h[1], r[0] + 1j * r[1]


# remainders of the 32-antenna warps, of the 128-voxel tiles and their pairs, of the samples' blocks
@pytest.mark.parametrize("A,S,N", [(24, 256, 16385), (33, 128, 24001), (64, 200, 8192), (130, 33, 24000), (1000, 200, 512),
                                   (257, 129, 3100), (40, 4096, 700)])
@pytest.mark.parametrize("order", ["grid", "random"])
def test_backward_vs_fp64(cuda, A, S, N, order):
    c = case(A + S, A, S, N)
    if order == "grid":  # neighbouring voxels share cells
        c["vox"] = np.ascontiguousarray(c["vox"][:, np.lexsort(c["vox"].round(2))])
    got, ref = backward(c)
    assert rel_l2(got, ref) < TOL


@pytest.mark.parametrize("box,bandwidth", [(((-0.6, -0.6, 0.2), (0.6, 0.6, 1.9)), 4e9),
                                           (((-0.1, -0.1, 8.2), (0.1, 0.1, 8.4)), 1e9),
                                           (((-0.1, -0.1, 3.9), (0.1, 0.1, 4.1)), 4e9)],
                         ids=["wide_band", "long_legs", "far_scene"])
def test_backward_bands_that_leave_the_cells(cuda, box, bandwidth):
    got, ref = backward(case(8, 140, 256, 4000, box=box, bandwidth=bandwidth))
    assert rel_l2(got, ref) < 1e-5


@pytest.mark.parametrize("box", [None, ((-0.6, -0.6, 0.2), (0.6, 0.6, 1.9))], ids=["cells", "wide_band"])
@pytest.mark.parametrize("A,S,N", [(24, 256, 16385), (130, 33, 24001)])
def test_nufft_form_vs_fp64(cuda, A, S, N, box):
    """The NUFFT form takes the cells too (its own kernels where the band does not fit)."""
    c = case(A + S, A, S, N, box=box)
    ch = c["ch"]
    args = (c["tx"], c["rx"], c["vox"])
    y = mf_forward(c["re"], c["im"], *args, ch.adc_sample_rate, ch.As_sci, "nufft")
    ref = oracle(c)
    scale = np.linalg.norm(c["re"] + 1j * c["im"]) / np.sqrt(A)  # the wide scene's voxels see noise only
    assert np.linalg.norm(y[0] + 1j * y[1] - ref) / np.sqrt(N) < 5e-6 * max(scale, np.linalg.norm(ref) / np.sqrt(N))
    gr, gi = c["rng"].standard_normal((2, N)).astype(np.float32)
    h = mf_backward(gr, gi, *args, A, S, ch.adc_sample_rate, ch.As_sci, "nufft")
    r = orc.mf_backward(gr, gi, *args, A, S, ch.adc_sample_rate, ch.As_sci)
    assert rel_l2(h[0] + 1j * h[1], r[0] + 1j * r[1]) < 5e-6


def test_backward_nan_voxel_poisons_every_sample(cuda):
    c = case(9, 140, 128, 6001)
    c["vox"][0, 5] = np.nan
    got, _ = backward(c)
    assert np.isnan(got.real).all() and np.isnan(got.imag).all()


@pytest.mark.parametrize("splits", [1, 5])
def test_forward_takes_any_tuning(cuda, splits):
    c = case(3, 144, 128, 9001)
    assert rel_l2(forward(c, tuning={"threads": 256, "items_per_thread": 2, "splits": splits}), oracle(c)) < TOL


@pytest.mark.parametrize("box,bandwidth", [(((-0.6, -0.6, 0.2), (0.6, 0.6, 1.9)), 4e9),   # more cells than fit
                                           (((-0.1, -0.1, 8.2), (0.1, 0.1, 8.4)), 1e9),   # legs beyond 8 m
                                           (((-0.1, -0.1, 3.9), (0.1, 0.1, 4.1)), 4e9)],  # long legs, narrow band
                         ids=["wide_band", "long_legs", "far_scene"])
def test_forward_bands_that_leave_the_cells(cuda, box, bandwidth):
    """The band is known on the device only: scenes whose cells do not fit run the direct kernel."""
    c = case(8, 140, 256, 4000, box=box, bandwidth=bandwidth)
    pos = c["rng"].uniform(box[0], box[1], (6, 3)).astype(np.float32)
    c["re"], c["im"] = scenes.synthesize_if_numpy(c["tx"], c["rx"], pos, np.ones(6) + 0.5j, c["ch"], snr_db=20.0,
                                                  rng=c["rng"])
    # the direct kernel's own error grows with the phase step: its bound is the MIXED form's
    assert rel_l2(forward(c), oracle(c)) < 1e-5


def test_forward_without_a_sweep_and_with_a_falling_one(cuda):
    c = case(5, 140, 128, 6000)
    for As in (0.0, -c["ch"].As_sci):
        args = (c["re"], c["im"], c["tx"], c["rx"], c["vox"], c["ch"].adc_sample_rate, As)
        y, r = mf_forward(*args, "mixed"), orc.mf_forward(*args)
        assert rel_l2(y[0] + 1j * y[1], r[0] + 1j * r[1]) < 1e-5


def test_forward_half_inputs(cuda):
    c = case(6, 140, 128, 6001)
    r = {k: c[k].astype(np.float16).astype(np.float32) for k in ("re", "im", "tx", "rx", "vox")}
    ref = oracle({**c, **r})
    assert rel_l2(forward(c, dtype=torch.float16), ref) < 2e-3  # half-precision outputs


def test_forward_non_finite_inputs(cuda):
    """A NaN voxel gives NaN there and leaves the others alone; a voxel or antenna at infinity
    runs the direct kernel; a voxel on an antenna stays finite."""
    c = case(7, 140, 128, 6002)
    ref = oracle(c)
    c["vox"][1, 77] = np.nan
    c["vox"][:, 600] = c["tx"][5]
    ref600 = oracle({**c, "vox": np.ascontiguousarray(c["vox"][:, 600:601] + np.float32(1e-7))})
    y = forward(c)
    assert np.isnan(y[77].real) and np.isnan(y[77].imag)
    keep = np.setdiff1d(np.arange(y.size), [77, 600])
    assert rel_l2(y[keep], ref[keep]) < TOL
    assert np.isfinite(y[600]) and abs(y[600] - ref600[0]) < 1e-2 * np.abs(ref).max()
    c["vox"][1, 77] = np.inf
    y = forward(c)
    keep = np.setdiff1d(np.arange(y.size), [77, 600])
    assert rel_l2(y[keep], ref[keep]) < 1e-5 and not np.isfinite(y[77])


# The result does not depend on where the scene lies: only differences of positions enter it.  The
# oracle takes the same FP32 positions, whose grid at the largest offset is 6 cm.
@pytest.mark.parametrize("offset", [(0.0, 0.0, 100.0), (-1e3, 300.0, 0.0), (3e3, 3e3, -3e3), (1e4, 0.0, 0.0), (0.0, 1e6, 0.0)])
@pytest.mark.parametrize("precision", ["mixed", "nufft"])
def test_scenes_far_from_the_origin(cuda, offset, precision):
    A, S, N = 140, 128, 6001
    c = case(11, A, S, N)
    for k in ("tx", "rx"):
        c[k] = np.ascontiguousarray((c[k] + np.array(offset)).astype(np.float32))
    c["vox"] = np.ascontiguousarray((c["vox"] + np.array(offset)[:, None]).astype(np.float32))
    ch = c["ch"]
    args = c["tx"], c["rx"], c["vox"]
    pos = c["vox"][:, c["rng"].integers(0, N, 6)].T
    c["re"], c["im"] = scenes.synthesize_if_numpy(*args[:2], pos, np.ones(6) + 0.5j, ch, snr_db=20.0, rng=c["rng"])
    y = mf_forward(c["re"], c["im"], *args, ch.adc_sample_rate, ch.As_sci, precision)
    assert rel_l2(y[0] + 1j * y[1], oracle(c)) < TOL
    gr, gi = c["rng"].standard_normal((2, N)).astype(np.float32)
    h = mf_backward(gr, gi, *args, A, S, ch.adc_sample_rate, ch.As_sci, precision)
    r = orc.mf_backward(gr, gi, *args, A, S, ch.adc_sample_rate, ch.As_sci)
    assert rel_l2(h[0] + 1j * h[1], r[0] + 1j * r[1]) < TOL


def test_backward_many_voxels_of_one_cell(cuda):
    """200000 voxels within 0.2 mm, gradients of one sign: every antenna adds them all up in
    one cell, in a call of so many antennas that no thread shares its voxels.  Two levels of
    sums, 128 terms and then 1563, err by 2^-24 sqrt(n) / 3 rms each, 8e-7 together; three times that
    beside TOL.  (One chain of 200000 would err by 9e-6.)"""
    A, S, N = 38016, 32, 200000
    rng = np.random.default_rng(12)
    tx, rx = (np.ascontiguousarray(x[:A]) for x in scenes.virtual_array(57))
    ch = scenes.chirp(S)
    vox = box_points(rng, N, (-1e-4, -1e-4, 0.4), (1e-4, 1e-4, 0.4002))
    gr, gi = rng.uniform(0, 1, (2, N)).astype(np.float32)
    h = mf_backward(gr, gi, tx, rx, vox, A, S, ch.adc_sample_rate, ch.As_sci, "mixed")
    some = np.arange(0, A, A // 12)
    r = orc.mf_backward(gr, gi, np.ascontiguousarray(tx[some]), np.ascontiguousarray(rx[some]), vox, some.size, S,
                        ch.adc_sample_rate, ch.As_sci)
    assert rel_l2((h[0] + 1j * h[1])[some] * A, (r[0] + 1j * r[1]) * some.size) < TOL + 3 * 8e-7


@pytest.mark.parametrize("value,part", [(np.inf, 0), (-np.inf, 1)])
def test_infinite_gradient(cuda, value, part):
    """One infinite gradient leaves no finite sample, and the first one of every antenna (no
    recurrence yet) infinite with the sign of the phase."""
    c = case(41, 200, 64, 10000)
    g = c["rng"].standard_normal((2, 10000)).astype(np.float32)
    g[part, 100] = value
    ch = c["ch"]
    got = mf_backward(*g, c["tx"], c["rx"], c["vox"], 200, 64, ch.adc_sample_rate, ch.As_sci, "mixed")
    assert not np.isfinite(got).any()
    one = np.zeros((2, 1))
    one[part] = np.sign(value)
    ref = orc.mf_backward(*one, c["tx"], c["rx"], np.ascontiguousarray(c["vox"][:, 100:101]), 200, 64,
                          ch.adc_sample_rate, ch.As_sci)
    for x, r in zip(got, ref):
        clear = np.abs(r[:, 0]) > 1e-3 / 200
        assert clear.sum() > 150
        np.testing.assert_array_equal(x[clear, 0], np.copysign(np.inf, r[clear, 0]))
