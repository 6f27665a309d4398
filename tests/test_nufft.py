"""GPU parity of the NUFFT (types 1 and 2) and the SENSE forward/adjoint against the FP64
direct NUDFT of the oracle.

Tolerance: the gridding error of the requested tolerance plus FP32 rounding; with
tol = 1e-6 (kernel width 7) the relative L2 error must be <= 1e-5, with tol = 1e-3
(width 4) <= 5e-3 (10x and 5x the requested tolerance)."""
import numpy as np
import pytest
import torch

from hastycompute_b200 import capi, synth
from hastycompute_b200.nufft import CUDANufft, NufftOptions, NufftPlan
from hastycompute_b200.toeplitz import ToeplitzPlan
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _c64(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a).astype(np.complex64)).to(dev)


def _np(t):
    return t.detach().cpu().numpy().astype(np.complex128)


def _coords(K, seed, lo=-np.pi, hi=np.pi):
    rng = np.random.default_rng(seed)
    return rng.uniform(lo, hi, (3, K)).astype(np.float32)


def _rand(shape, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("shape", [(16, 16, 16), (8, 16, 32), (32, 8, 8)])
@pytest.mark.parametrize("tol,bound", [(1e-6, 1e-5), (1e-3, 5e-3)])
def test_type1_type2_against_direct_nudft(cuda, shape, tol, bound):
    K = 2500
    coords = _coords(K, 1)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=tol, maxbatch=2)
    assert plan.width == int(np.ceil(np.log10(1 / tol))) + 1
    c = _rand((3, K), 2)
    f = plan.type1(_c64(c, cuda))
    ref = O.nudft_type1(coords, c, shape, +1)
    assert O.rel_l2(_np(f), ref) < bound
    fm = _rand((3,) + shape, 3)
    cc = plan.type2(_c64(fm, cuda))
    ref2 = O.nudft_type2(coords, fm, -1)
    assert O.rel_l2(_np(cc), ref2) < bound


@pytest.mark.parametrize("shape", [(32, 16), (8, 64), (64,), (16,)])
def test_lower_dimensional_plans_against_direct_nudft(cuda, shape):
    """The reference's 2-D and 1-D plans (nufft.ixx:72-160): coords [d, K], modes [ntransf, *shape]."""
    d, K = len(shape), 1500
    rng = np.random.default_rng(7)
    coords = rng.uniform(-np.pi, np.pi, (d, K)).astype(np.float32)
    ct = torch.from_numpy(coords).to(cuda)
    plan = NufftPlan(ct, shape, tol=1e-6, maxbatch=2)
    c = _rand((3, K), 8)
    assert O.rel_l2(_np(plan.type1(_c64(c, cuda))), O.nudft_type1(coords, c, shape, +1)) < 1e-5
    fm = _rand((3,) + shape, 9)
    assert O.rel_l2(_np(plan.type2(_c64(fm, cuda))), O.nudft_type2(coords, fm, -1)) < 1e-5
    # the reference-named mirror with nmodes [ntransf, *shape] (default tol 1e-5: bound 10x)
    op = CUDANufft(ct, [2, *shape], NufftOptions.type2())
    out = torch.empty((2, K), dtype=torch.complex64, device=cuda)
    op.apply(_c64(fm[:2], cuda), out)
    assert op.ndim() == d and O.rel_l2(_np(out), O.nudft_type2(coords, fm[:2], -1)) < 1e-4
    with pytest.raises(RuntimeError):
        NufftPlan(ct[:1] if d == 2 else torch.cat([ct, ct]), shape)  # rows must match the dimension


def test_signs_batching_and_periodicity(cuda):
    shape, K = (16, 16, 16), 1800
    coords = _coords(K, 4)
    c = _rand((5, K), 5)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6, maxbatch=2)
    # the other sign of each type
    f = plan.type1(_c64(c, cuda), isign=-1)
    assert O.rel_l2(_np(f), O.nudft_type1(coords, c, shape, -1)) < 1e-5
    fm = _rand((2,) + shape, 6)
    assert O.rel_l2(_np(plan.type2(_c64(fm, cuda), isign=+1)), O.nudft_type2(coords, fm, +1)) < 1e-5
    # 5 transforms in batches of 2 equal the transforms one by one
    f5 = _np(plan.type1(_c64(c, cuda)))
    for t in range(5):
        assert O.rel_l2(f5[t], _np(plan.type1(_c64(c[t:t + 1], cuda)))[0]) < 1e-6
    # coordinates are 2*pi periodic
    shifted = coords + np.float32(2 * np.pi) * np.sign(coords).astype(np.float32)
    plan2 = NufftPlan(torch.from_numpy(shifted).to(cuda), shape, tol=1e-6)
    assert O.rel_l2(_np(plan2.type1(_c64(c, cuda))), f5) < 1e-5


def test_type2_is_the_adjoint_of_type1(cuda):
    shape, K = (16, 8, 16), 2000
    coords = _coords(K, 7)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6)
    f = _rand(shape, 8)
    c = _rand((1, K), 9)
    lhs = np.vdot(_np(plan.type2(_c64(f, cuda), isign=-1)).ravel(), c.ravel())
    rhs = np.vdot(f.ravel(), _np(plan.type1(_c64(c, cuda), isign=+1)).ravel())
    assert abs(lhs - rhs) / abs(rhs) < 1e-5


def test_samples_on_the_grid_and_edges(cuda):
    # samples exactly on fine-grid points, on +-pi and at the origin
    shape = (16, 16, 16)
    g = np.linspace(-np.pi, np.pi, 9, dtype=np.float32)
    zz, yy, xx = np.meshgrid(g, g[::2], np.float32([0.0, np.pi / 16, -np.pi]), indexing="ij")
    coords = np.stack([zz.ravel(), yy.ravel(), xx.ravel()]).astype(np.float32)
    K = coords.shape[1]
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6)
    c = _rand((1, K), 10)
    assert O.rel_l2(_np(plan.type1(_c64(c, cuda))), O.nudft_type1(coords, c, shape, +1)) < 1e-5


def test_sense_adjoint_and_forward(cuda):
    shape, K, ncoil = (16, 16, 16), 2200, 5
    coords = _coords(K, 11)
    sm = synth.coil_maps(6, shape, seed=12)
    coils = [0, 2, 3, 5, 1]
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6, maxbatch=2)
    kd = _rand((ncoil, K), 13)
    out = plan.sense_adjoint(_c64(kd, cuda), _c64(sm, cuda), coils)
    assert O.rel_l2(_np(out), O.sense_adjoint(coords, kd, sm, coils)) < 1e-5
    # accumulate adds to the previous content
    plan.sense_adjoint(_c64(kd, cuda), _c64(sm, cuda), coils, out=out, accumulate=True)
    assert O.rel_l2(_np(out), 2 * O.sense_adjoint(coords, kd, sm, coils)) < 1e-5
    x = synth.gaussian_image(shape, seed=14)
    y = plan.sense_forward(_c64(x, cuda), _c64(sm, cuda), coils)
    assert O.rel_l2(_np(y), O.sense_forward(coords, x, sm, coils)) < 1e-5


@pytest.mark.parametrize("shape,ncoil,maxbatch", [((16, 16, 16), 4, 8), ((16, 16, 16), 5, 8), ((16, 16, 16), 12, 16),
                                                  ((32, 16), 20, 32), ((16, 16, 16), 11, 4)])
def test_sense_normal_in_place(cuda, shape, ncoil, maxbatch):
    """The image of sense_normal as its own output, in one group of coils and in several: every group reads
    the image as it was.  Against the oracle (1e-5 per transform) and the call with an output of its own
    (order of the sums of crowded tiles: 1e-6)."""
    d, K = len(shape), 1200
    coords = np.random.default_rng(87).uniform(-np.pi, np.pi, (d, K)).astype(np.float32)
    sm = synth.coil_maps(ncoil, (1,) * (3 - d) + shape, seed=88).reshape((ncoil,) + shape)
    x, y = _rand(shape, 89), _rand((ncoil, K), 90)
    w = np.random.default_rng(91).uniform(0.5, 1.0, K).astype(np.float32)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6, maxbatch=maxbatch)
    smt, kd, wt = _c64(sm, cuda), _c64(y, cuda), torch.from_numpy(w).to(cuda)
    ref = O.sense_normal_nufft(coords, x, sm, kdata=y, weights=w)
    apart = _np(plan.sense_normal(_c64(x, cuda), smt, kdata=kd, weights=wt))
    xt = _c64(x, cuda)
    assert plan.sense_normal(xt, smt, kdata=kd, weights=wt, out=xt) is xt
    assert O.rel_l2(_np(xt), ref) < 2e-5 and O.rel_l2(_np(xt), apart) < 1e-6
    xt = _c64(x, cuda)
    plan.sense_normal(xt, smt, kdata=kd, weights=wt, out=xt, accumulate=True)
    assert O.rel_l2(_np(xt), x + ref) < 2e-5
    # the result over a coil's map: maps are read by every group, too
    over = smt.clone()
    plan.sense_normal(_c64(x, cuda), over, kdata=kd, weights=wt, out=over[0])
    assert O.rel_l2(_np(over[0]), ref) < 2e-5
    over = smt.clone()
    plan.sense_adjoint(kd, over, out=over[0])
    assert O.rel_l2(_np(over[0]), O.sense_adjoint(coords, y, sm)) < 1e-5


def test_batched_sense_normal_in_place(cuda):
    """BatchedSenseNormal.apply(x, out=x) on more coils than one group transforms (10 x tol per transform)."""
    from hastycompute_b200.batched_sense import BatchedSenseNormal

    shape, ncoil, K = (16, 16, 16), 10, 900
    coords = [_coords(K, 92), _coords(K, 93)]
    sm, x = synth.coil_maps(ncoil, shape, seed=94), _rand((2, 1) + shape, 95)
    op = BatchedSenseNormal([torch.from_numpy(c) for c in coords], _c64(sm, cuda), maxbatch=16)
    xt = _c64(x, cuda)
    op.apply(xt, out=xt)
    for o in range(2):
        assert O.rel_l2(_np(xt[o, 0]), O.sense_normal_nufft(coords[o], x[o, 0], sm)) < 2e-4


def test_nufft_normal_equals_eight_times_toeplitz(cuda):
    """type1(type2(x)) / prod(N) (the reference's explicit normal operator) equals 8x the
    Toeplitz operator built from the same samples (the scaling of compare_normal_methods,
    lib/tests/tests1.cpp:351-549)."""
    shape, K = (16, 16, 16), 3000
    coords = _coords(K, 15)
    x = synth.gaussian_image(shape, seed=16)
    nplan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6)
    explicit = nplan.type1(nplan.type2(_c64(x, cuda)))[0] / float(np.prod(shape))
    tplan = ToeplitzPlan(shape, cuda)
    packed = tplan.build_diagonal(torch.from_numpy(coords).to(cuda))
    toep = torch.zeros(shape, dtype=torch.complex64, device=cuda)
    tplan.apply_add(_c64(x, cuda), toep, packed)
    assert O.rel_l2(_np(explicit), 8 * _np(toep)) < 1e-5


def test_cudanufft_mirror_and_errors(cuda):
    shape, K = (8, 8, 16), 900
    coords = torch.from_numpy(_coords(K, 17)).to(cuda)
    c = _rand((2, K), 18)
    op = CUDANufft(coords, [2] + list(shape), NufftOptions.type1(tol=1e-6))
    out = torch.empty((2,) + shape, dtype=torch.complex64, device=cuda)
    op.apply(_c64(c, cuda), out)
    assert O.rel_l2(_np(out), O.nudft_type1(coords.cpu().numpy(), c, shape, +1)) < 1e-5
    op2 = CUDANufft(coords, [2] + list(shape), NufftOptions.type2(tol=1e-6))
    kd = torch.empty((2, K), dtype=torch.complex64, device=cuda)
    op2.apply(out, kd)
    assert O.rel_l2(_np(kd), O.nudft_type2(coords.cpu().numpy(), _np(out), -1)) < 1e-5
    with pytest.raises(RuntimeError, match="nmodes"):
        op.apply(_c64(c, cuda), torch.empty((3,) + shape, dtype=torch.complex64, device=cuda))
    # 2 * 5 = 10 is not a compiled fine-grid length
    with pytest.raises(capi.HastyError) as e:
        NufftPlan(coords, (5, 8, 8))
    assert e.value.code == capi.HB_ERR_UNSUPPORTED
    with pytest.raises(capi.HastyError) as e:
        NufftPlan(coords, shape, tol=2.0)
    assert e.value.code == capi.HB_ERR_INVALID
    plan = NufftPlan(coords, shape)
    with pytest.raises(capi.HastyError) as e:
        plan.type1(_c64(c, cuda), isign=0)
    assert e.value.code == capi.HB_ERR_INVALID


@pytest.mark.parametrize("shape", [(16, 16, 16), (8, 16, 32), (32, 32, 32)])
def test_diagonal_through_the_nufft_matches_the_exact_build(cuda, shape):
    """hb_diag_build_nufft (the reference's NUFFT construction, tol 1e-6) against the
    FP64-exact hb_diag_build: complex T and the packed diagonal within 1e-5."""
    coords = torch.from_numpy(_coords(4000, 19)).to(cuda)
    plan = ToeplitzPlan(shape, cuda)
    pe, Te = plan.build_diagonal(coords, want_complex=True)
    pn, Tn = plan.build_diagonal(coords, want_complex=True, method="nufft", tol=1e-6)
    assert O.rel_l2(_np(Tn), _np(Te)) < 1e-5
    assert float((pn - pe).norm() / pe.norm()) < 1e-5
    # against the oracle too
    T = O.toeplitz_diagonal(coords.cpu().numpy().astype(np.float64), shape)
    assert O.rel_l2(_np(Tn), T) < 1e-5
    with pytest.raises(RuntimeError, match="method"):
        plan.build_diagonal(coords, method="fast")


@pytest.mark.parametrize("shape", [(96, 96, 8), (160, 160, 8)])
def test_diagonal_through_the_nufft_rejects_unsupported_grids(cuda, shape):
    """4*96 and 4*160 are not fine-grid lengths of the NUFFT: the build says so."""
    coords = torch.from_numpy(_coords(500, 23)).to(cuda)
    plan = ToeplitzPlan(shape, cuda)
    with pytest.raises(capi.HastyError) as e:
        plan.build_diagonal(coords, method="nufft")
    assert e.value.code == capi.HB_ERR_UNSUPPORTED


@pytest.mark.parametrize("shape,nt", [((256, 8, 8), 1), ((8, 256, 8), 3), ((8, 8, 256), 5), ((160, 8, 16), 2),
                                      ((48, 80, 8), 7), ((96, 8, 48), 9), ((80, 96), 6), ((128, 32), 8), ((160,), 4)])
def test_every_pass_length_and_group_of_transforms(cuda, shape, nt):
    """Each compiled line length on each axis, and batches that fill, pad and split the interleaved
    groups (1, 2, 4, 8; 5 = 4 + 1).  Bound: 10 x tol plus the worst phase error of a float32 grid
    position, pi/2 * n * 1.5 * 2^-24 at the highest mode."""
    d, K = len(shape), 400
    bound = 1e-5 + 1.41e-7 * 2 * max(shape)
    rng = np.random.default_rng(29)
    coords = rng.uniform(-np.pi, np.pi, (d, K)).astype(np.float32)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6, maxbatch=min(nt, 8))
    c, fm = _rand((nt, K), 30), _rand((nt,) + shape, 31)
    for sign in (+1, -1):
        f, ref = _np(plan.type1(_c64(c, cuda), isign=sign)), O.nudft_type1(coords, c, shape, sign)
        y, ref2 = _np(plan.type2(_c64(fm, cuda), isign=sign)), O.nudft_type2(coords, fm, sign)
        for t in range(nt):
            assert O.rel_l2(f[t], ref[t]) < bound and O.rel_l2(y[t], ref2[t]) < bound


@pytest.mark.parametrize("shape", [(48, 16), (32,)])
def test_five_transforms_of_a_lower_dimensional_plan(cuda, shape):
    """One group of eight with three unused transforms, then a group of its own after it.  Bound as in
    test_every_pass_length_and_group_of_transforms."""
    d, K = len(shape), 300
    bound = 1e-5 + 1.41e-7 * 2 * max(shape)
    coords = np.random.default_rng(33).uniform(-np.pi, np.pi, (d, K)).astype(np.float32)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6, maxbatch=8)
    for nt in (5, 13):
        c, fm = _rand((nt, K), 34), _rand((nt,) + shape, 35)
        f, ref = _np(plan.type1(_c64(c, cuda), isign=1)), O.nudft_type1(coords, c, shape, 1)
        y, ref2 = _np(plan.type2(_c64(fm, cuda), isign=-1)), O.nudft_type2(coords, fm, -1)
        for t in range(nt):
            assert O.rel_l2(f[t], ref[t]) < bound and O.rel_l2(y[t], ref2[t]) < bound


@pytest.mark.parametrize("W", [2, 3, 4, 5, 6, 7, 8, 10, 16])
def test_type2_every_width_and_group_writes_every_sample(cuda, W):
    """Type 2 of a 3-D plan at each layout of its lanes (kernel widths with 4 and 8 cells a load, one and two
    loads a row; groups of 1, 2, 4 and 8 transforms and their remainders), samples at both ends of the
    periodic grid included, into an output that starts as NaN.  Bound: 5 x tol (10 x below 1e-3) plus the
    float32 floor of test_every_pass_length_and_group_of_transforms and three axes of kernel values whose
    exponent, up to 2.30 W, is rounded twice."""
    shape, tol = (16, 32, 16), 1.01 * 10.0 ** (1 - W)
    bound = (5 if W <= 4 else 10) * tol + 1e-5 + 1.41e-7 * 2 * max(shape) + 3 * 2.30 * W * 2.0 ** -23
    ends = np.float32([-np.pi, -np.pi + 1e-4, -1e-4, 0.0, 1e-4, np.pi - 1e-4, np.pi])
    ends = np.stack([g.ravel() for g in np.meshgrid(ends, ends, ends, indexing="ij")])
    coords = np.concatenate([ends, _coords(150, 81)], 1).astype(np.float32)
    K = coords.shape[1]
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=tol, maxbatch=8)
    assert plan.width == W
    fm = _rand((12,) + shape, 82)
    ref, f = O.nudft_type2(coords, fm, -1), _c64(fm, cuda)
    for nt in (1, 2, 3, 4, 5, 8, 12):
        y = _np(plan.type2(f[:nt], torch.full((nt, K), complex("nan+nanj"), dtype=torch.complex64, device=cuda)))
        for t in range(nt):
            assert O.rel_l2(y[t], ref[t]) < bound, (nt, t)


@pytest.mark.parametrize("ncoil", [3, 4, 5, 12])
@pytest.mark.parametrize("tol", [1e-2, 1e-3])
def test_sense_normal_at_coarse_tolerances(cuda, ncoil, tol):
    """Groups of three and four coils (the remainders of 5 = 4 + 1 and 12 = 8 + 4 among them) at kernel widths 3 and
    4, twice with other inputs between, so that a sample left out would meet stale values.  Bound: 5 x tol
    for each of the two transforms."""
    shape, K = (16, 16, 16), 1500
    coords, sm = _coords(K, 83), synth.coil_maps(ncoil, shape, seed=84)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=tol, maxbatch=8)
    smt = _c64(sm, cuda)
    for seed in (85, 86):
        x, y = _rand(shape, seed), _rand((ncoil, K), seed + 10)
        out = plan.sense_normal(_c64(x, cuda), smt, kdata=_c64(y, cuda))
        ref = O.sense_normal_nufft(coords, x, sm, kdata=y)
        assert O.rel_l2(_np(out), ref) < 10 * tol


@pytest.mark.parametrize("shape,nt,maxbatch,K", [((32, 16), 9, 16, 300), ((16, 16), 9, 16, 40000), ((16, 16), 13, 16, 40000),
                                                 ((32, 16), 24, 16, 300), ((48, 16), 40, 32, 200), ((64,), 19, 32, 300),
                                                 ((16,), 32, 32, 50000), ((8, 8, 8), 16, 16, 500), ((16, 16, 16), 11, 16, 300)])
def test_batches_above_eight_transforms(cuda, shape, nt, maxbatch, K):
    """Small plans run several grids of eight transforms at once, with the last one padded or on its own,
    and batches beyond maxbatch.  Outputs start as NaN.  Bound as in test_every_pass_length_and_group_of_transforms."""
    d = len(shape)
    bound = 1e-5 + 1.41e-7 * 2 * max(shape)
    coords = np.random.default_rng(61).uniform(-np.pi, np.pi, (d, K)).astype(np.float32)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=1e-6, maxbatch=maxbatch)
    c, fm = _rand((nt, K), 62), _rand((nt,) + shape, 63)
    nan = complex("nan+nanj")
    f = _np(plan.type1(_c64(c, cuda), torch.full((nt,) + shape, nan, dtype=torch.complex64, device=cuda), isign=-1))
    y = _np(plan.type2(_c64(fm, cuda), torch.full((nt, K), nan, dtype=torch.complex64, device=cuda), isign=+1))
    ref, ref2 = O.nudft_type1(coords, c, shape, -1), O.nudft_type2(coords, fm, +1)
    for t in range(nt):
        assert O.rel_l2(f[t], ref[t]) < bound and O.rel_l2(y[t], ref2[t]) < bound
    # the coils of a SENSE operator in the same groups
    sm, x = _rand((nt,) + shape, 64), _rand(shape, 65)
    smt = _c64(sm, cuda)
    k = _np(plan.sense_forward(_c64(x, cuda), smt))
    ref = O.sense_forward(coords, x, sm)
    for t in range(nt):
        assert O.rel_l2(k[t], ref[t]) < bound
    assert O.rel_l2(_np(plan.sense_adjoint(_c64(c, cuda), smt)), O.sense_adjoint(coords, c, sm)) < bound


@pytest.mark.parametrize("W", [2, 4, 5, 7, 10, 16])
def test_gridding_kernel_values_and_their_square_root(cuda, W):
    """The kernel's own square root against FP64, s dense in [0, 1], towards 1 and down to the clamp at 1e-30: within
    0.5 + 2^-18 ulp.  The kernel exp(beta (sqrt(1 - t^2) - 1)) against FP64: t rounded twice and s once leave s within
    ds = 1.5 2^-22, the root within ds / sqrt(s) (at the edge sqrt(2 ds)) and two roundings, exp within 2 ulp."""
    n = 200000
    plan = NufftPlan(torch.from_numpy(_coords(10, 97)).to(cuda), (16, 16, 16), tol=1.01 * 10.0 ** (1 - W))
    assert plan.width == W
    rng = np.random.default_rng(98)
    s = np.concatenate([rng.uniform(0, 1, n // 4), 10.0 ** rng.uniform(-30, 0, n // 4), 1 - 2.0 ** rng.uniform(-24, 0, n // 4),
                        [1.0, 1e-30, 2.0 ** -24, 0.25]])
    s = np.clip(np.concatenate([s, rng.uniform(0.25, 1, n - len(s))]).astype(np.float32), np.float32(1e-30), 1)
    z = rng.uniform(-0.5 * W, 0.5 * W, n).astype(np.float32)
    z[:4] = [0.0, 0.5 * W, -0.5 * W, 0.51 * W]
    zt, st = torch.from_numpy(z).to(cuda), torch.from_numpy(s).to(cuda)
    phi, root = torch.empty_like(zt), torch.empty_like(zt)
    capi.check(plan.lib.hb_nufft_kernel_values(plan._h, zt.data_ptr(), st.data_ptr(), phi.data_ptr(), root.data_ptr(), n,
                                               torch.cuda.current_stream(cuda).cuda_stream))
    exact = np.sqrt(s.astype(np.float64))
    off = np.abs(root.cpu().numpy().astype(np.float64) - exact) / np.spacing(exact.astype(np.float32))
    assert off.max() <= 0.5 + 2.0 ** -18
    beta = float(np.float32(2.30 * W))
    q = np.maximum(1 - (z.astype(np.float64) / (0.5 * W)) ** 2, 0)
    ref = np.where(q > 0, np.exp(beta * (np.sqrt(q) - 1)), 0)
    ds = 1.5 * 2.0 ** -22
    dr = np.where(q > ds, ds / np.sqrt(np.maximum(q, ds)), np.sqrt(2 * ds)) + 2.0 ** -23
    rel = np.expm1(beta * dr) + beta * 2.0 ** -24 + 2.0 ** -22
    got = phi.cpu().numpy().astype(np.float64)
    assert (np.abs(got - ref) <= np.where(q > ds, ref * rel, np.exp(beta * (np.sqrt(2 * ds) - 1)) * (1 + rel))).all()
    assert got[0] == 1.0 and got[3] == 0.0


@pytest.mark.parametrize("shape,tol,nt", [((16, 16, 16), 1e-6, 8), ((32, 8, 48), 1e-4, 3), ((4, 4, 4), 1e-3, 2),
                                          ((16, 32, 16), 1e-9, 1), ((64, 32), 1e-6, 8), ((4, 64), 1e-3, 4),
                                          ((80, 16), 1e-5, 1)])
def test_spreading_crowded_and_empty_tiles(cuda, shape, tol, nt):
    """Tiles with thousands of samples (cut into pieces), with a few, and with none; samples on tile
    and grid edges; kernels from narrower to wider than a tile.  Bound: 10 x tol, and not below the
    float32 floor of test_every_pass_length_and_group_of_transforms."""
    d = len(shape)
    rng = np.random.default_rng(41)
    crowd = rng.normal(0.0, 0.02, (d, 3000))                          # around the origin (a grid corner)
    same = np.full((d, 700), 0.6)                                     # one position many times
    cell = 2 * np.pi / (2 * np.array(shape, float))[:, None]
    edge = cell * rng.integers(0, 2 * min(shape), (d, 60))            # on grid cells
    coords = np.concatenate([crowd, same, edge, rng.uniform(-np.pi, np.pi, (d, 20))], 1).astype(np.float32)
    plan = NufftPlan(torch.from_numpy(coords).to(cuda), shape, tol=tol, maxbatch=nt)
    c = _rand((nt, coords.shape[1]), 42)
    f, ref = _np(plan.type1(_c64(c, cuda))), O.nudft_type1(coords, c, shape, +1)
    for t in range(nt):
        assert O.rel_l2(f[t], ref[t]) < max(10 * tol, 1e-5 + 1.41e-7 * 2 * max(shape))


def test_diagonal_in_a_caller_workspace(cuda):
    """hb_diag_build_nufft_ws against hb_diag_build_nufft (to reduction order), its workspace size, and
    what it refuses."""
    import ctypes

    shape = (16, 8, 32)
    plan = ToeplitzPlan(shape, cuda)
    lib, st = plan.lib, torch.cuda.current_stream(cuda).cuda_stream
    coords = torch.from_numpy(_coords(3000, 71)).to(cuda)
    w = torch.rand(3000, device=cuda)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    a = torch.empty(plan.packed_numel(), device=cuda)
    b = torch.empty_like(a)
    T = torch.empty(plan.grid, dtype=torch.complex64, device=cuda)
    capi.check(lib.hb_diag_build_nufft(plan._h, ptr(coords), 3000, 1e-6, ptr(w), ptr(a), None, st))
    nb = lib.hb_diag_build_nufft_workspace_bytes(plan._h, 3000, 1e-6)
    ws = torch.empty(nb, dtype=torch.uint8, device=cuda)
    capi.check(lib.hb_diag_build_nufft_ws(plan._h, ptr(coords), 3000, 1e-6, ptr(w), ptr(b), ptr(T), ptr(ws), nb, st))
    assert float((a - b).norm() / a.norm()) < 1e-6
    assert float((plan.pack_diagonal(T) - b).norm() / a.norm()) < 1e-6
    assert lib.hb_diag_build_nufft_ws(plan._h, ptr(coords), 3000, 1e-6, None, ptr(b), None, ptr(ws), 1000, st) == \
        capi.HB_ERR_WORKSPACE
    assert lib.hb_diag_build_nufft_ws(plan._h, ptr(coords), 3000, 1e-6, None, None, None, ptr(ws), nb, st) == \
        capi.HB_ERR_INVALID
    assert lib.hb_diag_build_nufft_workspace_bytes(plan._h, 3000, 2.0) == 0
