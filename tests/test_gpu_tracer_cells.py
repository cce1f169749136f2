"""The MIXED and NUFFT tracers through range cells against the FP64 oracle, where
their special paths are: scenes whose cells share slots (deferred points), bands
that leave the adjoint's tables, runs of points longer than a pass, remainders.

Tolerance: FP32 geometry (~5e-7), phases good to 1e-7 cycles, hardware sine and
cosine (4e-7) and FP32 sums, with the positions' gradient a difference of terms ten
times its size: 2e-5."""
import numpy as np
import pytest
import torch

from conftest import rel_l2
from benchkit import scenes
from gpu_helpers import cu, tracer_backward, tracer_forward
from oracle import rf_oracle as orc

pytestmark = pytest.mark.gpu

TOL = 2e-5


def case(seed, A, P, S, depth=(0.3, 0.5), bandwidth=4e9):
    """Points of a slab facing the array, most of the pairs live."""
    rng = np.random.default_rng(seed)
    tx, rx = scenes.virtual_array(4)
    tx, rx = tx[:A], rx[:A]
    pts = np.stack([rng.uniform(-0.2, 0.2, P), rng.uniform(-0.2, 0.2, P), rng.uniform(*depth, P)], 1)
    nrm = -pts / np.linalg.norm(pts, axis=1, keepdims=True) + rng.normal(0, 0.15, (P, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    ch = scenes.chirp(S, bandwidth=bandwidth)
    f = np.float32
    return dict(normals=nrm.astype(f), sigmas=rng.uniform(0, 1, (A, P)).astype(f), points=pts.astype(f),
                tx=tx.astype(f), rx=rx.astype(f), inbounds=rng.uniform(0, 1, P) < 0.9, fs=f(ch.adc_sample_rate),
                f0=f(770.0), As=f(ch.As_sci), S=S, rng=rng)


def check(c, precision, tuning=None):
    scal = float(c["fs"]), float(c["f0"]), float(c["As"])
    geo = (c["normals"], c["sigmas"], c["points"], c["tx"], c["rx"], c["inbounds"])
    x = tracer_forward(c, c["S"], precision, tuning=tuning)
    r = orc.tracer_forward(*geo, c["S"], *scal, "f64")
    assert rel_l2(x[0] + 1j * x[1], r[0] + 1j * r[1]) < TOL
    A = c["tx"].shape[0]
    gr, gi = c["rng"].standard_normal((2, A, c["S"])).astype(np.float32)
    got = tracer_backward(c, gr, gi, precision, tuning=tuning)
    ref = orc.tracer_backward(gr, gi, *geo, *scal)
    for g, w in zip(got, ref):
        assert rel_l2(g, w) < TOL


@pytest.mark.parametrize("precision", ["mixed", "nufft"])
@pytest.mark.parametrize("A,P,S", [(1, 129, 32), (33, 1024, 33), (12, 5003, 101), (70, 700, 256), (3, 40001, 64)])
def test_shapes(cuda, A, P, S, precision):
    check(case(A + S, A, P, S), precision)


@pytest.mark.parametrize("depth,bandwidth", [((0.3, 3.3), 4e9),   # cells up to 160 apart: several passes over a run
                                             ((0.3, 6.0), 4e9),   # and a band outside the adjoint's tables
                                             ((0.3, 0.5), 60e9)], # the same by a wide sweep
                         ids=["deep", "deeper", "wide_sweep"])
@pytest.mark.parametrize("splits", [0, 1])
def test_cells_that_share_slots(cuda, depth, bandwidth, splits):
    check(case(4, 7, 3000, 128, depth, bandwidth), "mixed", {"splits": splits})


def test_runs_longer_than_a_pass(cuda):
    check(case(5, 2, 40001, 48), "mixed", {"splits": 1})


@pytest.mark.parametrize("depth", [(0.3, 0.5), (0.3, 3.3)], ids=["near", "deep"])
def test_ragged_runs(cuda, depth):
    """Long work items (several passes each), antennas of 1 to 33000 points, against the tracer
    over each antenna's points alone."""
    from geraf_b200.ops.RFSignalTracer.ragged import signal_tracer_ragged

    c = case(6, 4, 36000, 64, depth)
    counts = [1, 33000, 511, 2488]
    off = np.concatenate([[0], np.cumsum(counts)])
    sig = c["sigmas"][0]
    t = {k: cu(v).requires_grad_(True) for k, v in (("normals", c["normals"]), ("points", c["points"]), ("sigmas", sig))}
    xr, xi = signal_tracer_ragged(t["normals"], t["sigmas"], t["points"], torch.tensor(off, device="cuda"), cu(c["tx"]),
                                  cu(c["rx"]), c["S"], float(c["fs"]), float(c["f0"]), float(c["As"]),
                                  inbounds=torch.tensor(c["inbounds"], device="cuda"), tuning={"items_per_thread": 512})
    gr, gi = c["rng"].standard_normal((2, 4, c["S"])).astype(np.float32)
    gn, gs, gp = torch.autograd.grad((xr, xi), (t["normals"], t["sigmas"], t["points"]), (cu(gr), cu(gi)))
    x = xr.detach().cpu().numpy() + 1j * xi.detach().cpu().numpy()
    pairs = [], [], []  # every pair's gradients, without its antenna's 1 / points: (got, reference)
    for a in range(4):
        e = slice(off[a], off[a + 1])
        args = (c["normals"][e], sig[None, e], c["points"][e], c["tx"][a:a + 1], c["rx"][a:a + 1], c["inbounds"][e])
        scal = float(c["fs"]), float(c["f0"]), float(c["As"])
        r = orc.tracer_forward(*args, c["S"], *scal, "f64")
        assert rel_l2(x[a], (r[0] + 1j * r[1])[0]) < TOL
        rn, rs, rp = orc.tracer_backward(gr[a:a + 1], gi[a:a + 1], *args, *scal)
        for k, (got, ref) in enumerate(((gn, rn), (gs, rs[0]), (gp, rp))):
            pairs[k].append((counts[a] * got[e].double().cpu().numpy(), counts[a] * ref))
    for p in pairs:
        assert rel_l2(np.concatenate([g for g, _ in p]), np.concatenate([r for _, r in p])) < TOL


@pytest.mark.parametrize("depth", [(0.3, 0.5), (0.3, 3.3)], ids=["near", "deep"])
def test_forward_bits_repeat(cuda, depth):
    """Which cell takes a slot does not depend on the order of the threads."""
    c = case(7, 7, 20000, 128, depth)
    first = tracer_forward(c, c["S"], "mixed", tuning={"splits": 2})
    for _ in range(5):
        for got, ref in zip(tracer_forward(c, c["S"], "mixed", tuning={"splits": 2}), first):
            np.testing.assert_array_equal(got, ref)


@pytest.mark.parametrize("splits", [0, 1])
def test_many_points_of_one_cell(cuda, splits):
    """400000 live points within 0.1 mm, one contribution as large as the next: they are summed
    by batches of 128, then by batch (3125 terms: 2^-24 sqrt(n) / 3 = 1.1e-6 rms; three times that), in one block or
    in many.  FP32 geometry, phase, sine and cosine: 2e-6.  (One chain would err by 1.3e-5.)"""
    P, S = 400000, 64
    c = case(13, 2, P, S)
    c["points"] = (np.array([0.01, 0.02, 0.4]) + c["rng"].uniform(-5e-5, 5e-5, (P, 3))).astype(np.float32)
    c["normals"] = (-c["points"] / np.linalg.norm(c["points"], axis=1, keepdims=True)).astype(np.float32)
    x = tracer_forward(c, S, "mixed", tuning={"splits": splits})
    r = orc.tracer_forward(c["normals"], c["sigmas"], c["points"], c["tx"], c["rx"], c["inbounds"], S, float(c["fs"]),
                           float(c["f0"]), float(c["As"]), "f64")
    assert rel_l2(x[0] + 1j * x[1], r[0] + 1j * r[1]) < 2e-6 + 3 * 1.1e-6


@pytest.mark.parametrize("S", [33, 300])
@pytest.mark.parametrize("splits", [1, 3])
def test_scene_that_leaves_its_slots_midway(cuda, S, splits):
    """Points sorted by their distance, 150 cells of them: a share's first batches go through the
    cells, the rest does not (300 samples: two sweeps over it)."""
    c = case(14, 5, 3000, S, (0.3, 3.3))
    order = np.argsort(np.linalg.norm(c["points"], axis=1))
    for k in ("normals", "points", "inbounds"):
        c[k] = np.ascontiguousarray(c[k][order])
    c["sigmas"] = np.ascontiguousarray(c["sigmas"][:, order])
    check(c, "mixed", {"splits": splits})


# many antennas of few points (their moments become samples by warps): one share each and several,
# remainders of the 32 samples, the longest rows that go this way and longer ones, a falling sweep
@pytest.mark.parametrize("A,P,S,splits", [(300, 700, 33, 0), (300, 1500, 64, 3), (301, 130, 384, 1), (301, 130, 512, 1),
                                          (1200, 60, 100, 0)])
@pytest.mark.parametrize("fall", [1.0, -1.0])
def test_many_antennas_of_few_points(cuda, A, P, S, splits, fall):
    c = case(15, A, P, S)
    tx, rx = scenes.virtual_array(10)
    c["tx"], c["rx"] = tx[:A].astype(np.float32), rx[:A].astype(np.float32)
    c["As"] = np.float32(fall * c["As"])
    check(c, "mixed", {"splits": splits})


@pytest.mark.parametrize("depth", [(0.3, 0.5), (0.3, 3.3)], ids=["near", "deep"])
def test_ragged_many_antennas(cuda, depth):
    """Antennas of 0 to 40 points and one of 30000 in one call, against FP64."""
    from geraf_b200.ops.RFSignalTracer.ragged import signal_tracer_ragged

    A, S = 310, 96
    rng = np.random.default_rng(16)
    counts = rng.integers(0, 41, A)
    counts[[0, A - 1]] = 0
    counts[200] = 30000
    off = np.concatenate([[0], np.cumsum(counts)])
    c = case(16, 1, int(off[-1]), S, depth)
    tx, rx = (x[:A].astype(np.float32) for x in scenes.virtual_array(6))
    scal = float(c["fs"]), float(c["f0"]), float(c["As"])
    x = signal_tracer_ragged(cu(c["normals"]), cu(c["sigmas"][0]), cu(c["points"]), torch.tensor(off, device="cuda"), cu(tx),
                             cu(rx), S, *scal, inbounds=torch.tensor(c["inbounds"], device="cuda"),
                             tuning={"items_per_thread": 8})
    x = x[0].cpu().numpy() + 1j * x[1].cpu().numpy()
    got, ref = [], []
    for a in range(A):
        if counts[a] == 0:
            assert np.isnan(x[a]).all()
            continue
        e = slice(off[a], off[a + 1])
        r = orc.tracer_forward(c["normals"][e], c["sigmas"][:, e], c["points"][e], tx[a:a + 1], rx[a:a + 1],
                               c["inbounds"][e], S, *scal, "f64")
        got.append(counts[a] * x[a])
        ref.append(counts[a] * (r[0] + 1j * r[1])[0])
    assert rel_l2(np.array(got), np.array(ref)) < TOL


# fewer than 48 points per antenna on average (rows read from device memory, 16 bytes at a time where
# the samples allow it), and the most that is not
@pytest.mark.parametrize("most,S", [(1, 64), (40, 33), (40, 36), (94, 64), (97, 64)])
@pytest.mark.parametrize("dtype,with_points", [(torch.float32, True), (torch.float32, False), (torch.float64, True)])
def test_ragged_adjoint_of_short_antennas(cuda, most, S, dtype, with_points):
    from geraf_b200.ops.RFSignalTracer.ragged import signal_tracer_ragged

    A = 210
    rng = np.random.default_rng(most)
    counts = np.full(A, 1) if most == 1 else rng.permutation(np.arange(A) * (most + 1) // A)  # 0 .. most
    off = np.concatenate([[0], np.cumsum(counts)])
    c = case(most, 1, int(off[-1]), S)
    tx, rx = (x[:A].astype(np.float32) for x in scenes.virtual_array(5))
    scal = float(c["fs"]), float(c["f0"]), float(c["As"])
    t = [cu(c["normals"], dtype).requires_grad_(True), cu(c["sigmas"][0], dtype).requires_grad_(True),
         cu(c["points"], dtype).requires_grad_(with_points)]
    x = signal_tracer_ragged(*t, torch.tensor(off, device="cuda"), cu(tx, dtype), cu(rx, dtype), S, *scal,
                             inbounds=torch.tensor(c["inbounds"], device="cuda"))
    gr, gi = rng.standard_normal((2, A, S)).astype(np.float32)
    got = torch.autograd.grad(x, t[:2 + with_points], (cu(gr, dtype), cu(gi, dtype)))
    refs = [], [], []
    scale = np.repeat(counts, counts)  # without its antenna's 1 / points, as above
    for a in range(A):
        e = slice(off[a], off[a + 1])
        if counts[a]:
            r = orc.tracer_backward(gr[a:a + 1], gi[a:a + 1], c["normals"][e], c["sigmas"][:, e], c["points"][e],
                                    tx[a:a + 1], rx[a:a + 1], c["inbounds"][e], *scal)
            for k, w in enumerate((r[0], r[1][0], r[2])):
                refs[k].append(counts[a] * w)
    for g, w in zip(got, refs):
        g = g.double().cpu().numpy()
        assert rel_l2(g * scale.reshape(-1, *[1] * (g.ndim - 1)), np.concatenate(w)) < TOL


@pytest.mark.parametrize("precision", ["mixed", "nufft"])
def test_adjoint_tables_of_more_cells(cuda, precision):
    """640 cells with points enough for their tables (the general kernel takes them otherwise)."""
    check(case(17, 5, 9000, 128, (0.3, 6.0)), precision)


@pytest.mark.parametrize("value", [np.inf, -np.inf])
@pytest.mark.parametrize("splits", [0, 1])
def test_infinite_values(cuda, value, splits):
    """An infinite sigma leaves no finite sample, and the first of every antenna (no recurrence yet)
    infinite with the sign of the phase; so does an infinite residual at sample 0 with the gradients."""
    A, P, S, q = 5, 3000, 64, 77
    c = case(19, A, P, S)
    c["inbounds"][q] = True
    c["normals"][q] = -c["points"][q] / np.linalg.norm(c["points"][q])
    geo = lambda e, sig: (c["normals"][e], sig, c["points"][e], c["tx"], c["rx"], c["inbounds"][e])
    scal = float(c["fs"]), float(c["f0"]), float(c["As"])
    d = dict(c, sigmas=c["sigmas"].copy())
    d["sigmas"][:, q] = value
    got = tracer_forward(d, S, "mixed", tuning={"splits": splits})
    assert not np.isfinite(got).any()
    e = slice(q, q + 1)
    ref = orc.tracer_forward(*geo(e, np.full((A, 1), np.sign(value), np.float32)), S, *scal, "f64")
    for x, r in zip(got, ref):
        np.testing.assert_array_equal(x[:, 0], np.copysign(np.inf, r[:, 0]))
    g = np.zeros((2, A, S), np.float32)
    g[0, 2, 0] = value
    got = tracer_backward(c, *g, "mixed", tuning={"splits": splits})[1]
    unit = np.where(np.isinf(g), np.sign(g), 0).astype(np.float32)
    ref = orc.tracer_backward(*unit, *geo(slice(None), c["sigmas"]), *scal)[1]
    clear = np.abs(ref[2]) > 1e-3 * np.abs(ref[2]).max()
    np.testing.assert_array_equal(got[2][clear], np.copysign(np.inf, ref[2][clear]))
    np.testing.assert_array_equal(np.delete(got, 2, 0), 0)


@pytest.mark.parametrize("S", [700, 1024, 1025])
def test_many_antennas_of_long_rows(cuda, S):
    """The longest rows whose moments become samples by warps, and one longer."""
    c = case(20, 300, 90, S)
    tx, rx = scenes.virtual_array(6)
    c["tx"], c["rx"] = tx[:300].astype(np.float32), rx[:300].astype(np.float32)
    check(c, "mixed")


@pytest.mark.parametrize("depth,splits", [((0.3, 0.5), 16), ((0.3, 0.5), 17), ((0.3, 0.5), 0), ((0.3, 1.9), 5), ((0.3, 3.3), 5)],
                         ids=["most", "more", "default", "cells_of_two_rounds", "deep"])
def test_shares_of_many_antennas(cuda, depth, splits):
    """The shares of an antenna are added up before they become samples, where their cells agree (up to 16
    shares); in the deeper scenes they hold other cells in a slot, or rows beside cells."""
    c = case(21, 300, 3000, 70, depth)
    tx, rx = scenes.virtual_array(6)
    c["tx"], c["rx"] = tx[:300].astype(np.float32), rx[:300].astype(np.float32)
    order = np.argsort(np.linalg.norm(c["points"], axis=1))
    for k in ("normals", "points", "inbounds"):
        c[k] = np.ascontiguousarray(c[k][order])
    check(c, "mixed", {"splits": splits})


# many antennas of so few points that the cells are left out: no point in bounds, one point, the most
# (384) and one more; samples that leave several lanes to a sum (16, 32, 64), remainders, two sweeps
@pytest.mark.parametrize("P,S", [(1, 16), (7, 1), (384, 33), (385, 33), (200, 70), (130, 300), (384, 1030)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_many_antennas_of_so_few_points(cuda, P, S, dtype):
    c = case(22, 300, P, S)
    tx, rx = scenes.virtual_array(6)
    c["tx"], c["rx"] = tx[:300].astype(np.float32), rx[:300].astype(np.float32)
    c["inbounds"][0] = True
    geo = (c["normals"], c["sigmas"], c["points"], c["tx"], c["rx"], c["inbounds"])
    x = tracer_forward(c, S, "mixed", dtype=dtype)
    r = orc.tracer_forward(*geo, S, float(c["fs"]), float(c["f0"]), float(c["As"]), "f64")
    assert rel_l2(x[0] + 1j * x[1], r[0] + 1j * r[1]) < TOL
    c["inbounds"][:] = False
    for got in tracer_forward(c, S, "mixed", dtype=dtype):
        np.testing.assert_array_equal(got, 0)


# the adjoint's tables by 4 cells a block (fewer than 64 antennas) and by 16: samples that leave slices
# without one, and remainders of the basis's blocks of 64
@pytest.mark.parametrize("A,S", [(1, 32), (1, 1000), (2, 65), (63, 129), (64, 129)])
def test_adjoint_tables_of_few_antennas(cuda, A, S):
    check(case(23, A, 2000, S), "mixed")


# more work items than the GPU holds blocks: rows of items past their cells from a kernel of their own
@pytest.mark.parametrize("depth", [(0.3, 0.5), (0.3, 3.3)], ids=["near", "deep"])
def test_ragged_items_past_the_resident_blocks(cuda, depth):
    from geraf_b200.ops.RFSignalTracer.ragged import signal_tracer_ragged

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    P = 256 * 6 * sms + 129  # items of 256 points
    c = case(24, 2, P, 33, depth)
    off = [0, P - 700, P]
    scal = float(c["fs"]), float(c["f0"]), float(c["As"])
    x = signal_tracer_ragged(cu(c["normals"]), cu(c["sigmas"][0]), cu(c["points"]), torch.tensor(off, device="cuda"),
                             cu(c["tx"]), cu(c["rx"]), c["S"], *scal, inbounds=torch.tensor(c["inbounds"], device="cuda"),
                             tuning={"items_per_thread": 2})
    x = x[0].cpu().numpy() + 1j * x[1].cpu().numpy()
    for a in range(2):
        e = slice(off[a], off[a + 1])
        r = orc.tracer_forward(c["normals"][e], c["sigmas"][:1, e], c["points"][e], c["tx"][a:a + 1], c["rx"][a:a + 1],
                               c["inbounds"][e], c["S"], *scal, "f64")
        assert rel_l2(x[a], (r[0] + 1j * r[1])[0]) < TOL
