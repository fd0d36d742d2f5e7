"""ILMC (adzc_ilmc) against the sequential restatement (oracle/adz_oracle_impl.h:
orc_ilmc) on the same fields: bit-exact, FP32 and FP64, sparse and dense
violations (the dense case needs many rounds of the order-preserving parallel
schedule), sweeps 1 to 3, with and without the final clip."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fields(st, dt, frac, seed):
    rng = np.random.default_rng(seed)
    sh = st.ext_shape
    mn = rng.random(sh).astype(dt)
    mx = (mn + 0.5 + rng.random(sh)).astype(dt)
    f = (mn + (mx - mn) * rng.random(sh)).astype(dt)
    air = (1.0 + 0.3 * rng.random(sh)).astype(dt)
    viol = rng.random(sh) < frac
    f = np.where(viol, np.where(rng.random(sh) < 0.5, mx + 0.3 * rng.random(sh), mn - 0.3 * rng.random(sh)),
                 f).astype(dt)
    return f, mn, mx, air


@pytest.mark.parametrize("prec_name,frac,sweeps,min_max", [("mixed", 0.01, 2, True), ("fp64", 0.01, 2, False),
                                                            ("ref32", 0.2, 2, True), ("mixed", 0.05, 1, False),
                                                            ("fp64", 0.05, 3, True), ("mixed", 0.2, 4, True)])
def test_ilmc_bit_exact(prec_name, frac, sweeps, min_max):
    from gem_b200 import adz as A, synth
    from oracle import oracle as O
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    prec = A.PREC_NAMES[prec_name]
    cfg = synth.config_small(40, 36, 16)
    st = O.Step(cfg, "oracle", "f64" if prec == A.FP64 else "f32")
    dt = np.float64 if prec == A.FP64 else np.float32
    trs = [_fields(st, dt, frac, seed) for seed in (3, 4)]
    air = trs[0][3]
    ad = A.Adz.from_config(cfg)
    fs = [torch.from_numpy(t[0].copy()).cuda() for t in trs]
    mns = [torch.from_numpy(t[1]).cuda() for t in trs]
    mxs = [torch.from_numpy(t[2]).cuda() for t in trs]
    rounds = A.ilmc(ad, prec, fs, mns, mxs, torch.from_numpy(air).cuda(), sweep_max=sweeps, min_max=min_max)
    torch.cuda.synchronize()
    assert rounds >= 1
    for t, g in zip(trs, fs):
        ref = st.ilmc(t[0], t[1], t[2], air, sweep_max=sweeps, min_max=min_max)
        got = g.cpu().numpy()
        diff = int(np.sum(got != ref))
        assert diff == 0, (diff, rounds)
        assert not np.array_equal(ref, t[0])  # the filter did something


# wavefronts with more listed tiles than the grid has warps (a wide region of
# narrow tiles), and mostly empty wavefronts (violations at a few corners)
@pytest.mark.parametrize("prec_name,size,ntr,frac,sweeps", [("mixed", (1200, 24, 8), 6, 0.3, 1),
                                                            ("fp64", (200, 30, 9), 1, 0.0, 2),
                                                            ("ref32", (45, 33, 21), 2, 0.0, 4)])
def test_ilmc_wavefront_sizes(prec_name, size, ntr, frac, sweeps):
    from gem_b200 import adz as A, synth
    from oracle import oracle as O
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    prec = A.PREC_NAMES[prec_name]
    cfg = synth.config_small(*size)
    st = O.Step(cfg, "oracle", "f64" if prec == A.FP64 else "f32")
    dt = np.float64 if prec == A.FP64 else np.float32
    trs = [_fields(st, dt, frac, 11 + q) for q in range(ntr)]
    air = trs[0][3]
    if frac == 0.0:  # the region's corners and its middle
        ad0 = A.Adz.from_config(cfg)
        i0, i1, j0, j1, k0 = ad0.set_range(A.SET_T)
        H = ad0.info.halox
        for f, mn, mx, _ in trs:
            for k in (k0, (k0 + cfg.nk) // 2, cfg.nk):
                for j in (j0, (j0 + j1) // 2, j1):
                    for i in (i0, i0 + 1, (i0 + i1) // 2, i1):
                        f[k - 1, j - 1 + H, i - 1 + H] = mx[k - 1, j - 1 + H, i - 1 + H] + dt(0.75)
    ad = A.Adz.from_config(cfg)
    fs = [torch.from_numpy(t[0].copy()).cuda() for t in trs]
    A.ilmc(ad, prec, fs, [torch.from_numpy(t[1]).cuda() for t in trs], [torch.from_numpy(t[2]).cuda() for t in trs],
           torch.from_numpy(air).cuda(), sweep_max=sweeps, min_max=False)
    torch.cuda.synchronize()
    assert ad.status() == 0
    for t, g in zip(trs, fs):
        ref = st.ilmc(t[0], t[1], t[2], air, sweep_max=sweeps, min_max=False)
        assert np.array_equal(g.cpu().numpy(), ref)
        assert not np.array_equal(ref, t[0])


@pytest.mark.parametrize("prec_name,sweeps", [("ref32", 2), ("fp64", 3)])
def test_ilmc_on_part_of_the_sms(prec_name, sweeps):
    """A stream of a green context owns some of the SMs: the filter's blocks,
    which run at once, must fit there."""
    from gem_b200 import adz as A, synth
    from oracle import oracle as O
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    prec = A.PREC_NAMES[prec_name]
    cfg = synth.config_small(40, 36, 12)
    st = O.Step(cfg, "oracle", "f64" if prec == A.FP64 else "f32")
    dt = np.float64 if prec == A.FP64 else np.float32
    t = _fields(st, dt, 0.05, 21)
    ad = A.Adz.from_config(cfg)
    f, mn, mx, air = (torch.from_numpy(x.copy()).cuda() for x in t)
    torch.cuda.synchronize()
    part = torch.cuda.GreenContext.create(num_sms=16, device_id=0)
    part.set_context()
    try:
        A.ilmc(ad, prec, [f], [mn], [mx], air, sweep_max=sweeps, min_max=False)
        torch.cuda.current_stream().synchronize()
    finally:
        part.pop_context()
    torch.cuda.synchronize()
    assert ad.status() == 0
    ref = st.ilmc(t[0], t[1], t[2], air=t[3], sweep_max=sweeps, min_max=False)
    assert np.array_equal(f.cpu().numpy(), ref) and not np.array_equal(ref, t[0])
