"""The step's gather kernels on shared-memory boxes against the direct ones,
bit for bit (they form the same sums in the same order): trajectories against
the phased batch plan (REF32 against the oracle), the iteration to a tolerance
against fixed updates, the position sets and BICUBH_QV against the same call
with a zero perturbation pattern, which the direct kernels run.  Small tiles,
which the direct kernels take, and sizes at the edges of tiles and boxes, rows
that are not 16-byte multiples, sources off a 16-byte boundary, few levels,
flows sheared within a tile, and flows so scattered that stencils leave their
box or the boxes are placed more than once."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(33, 9, 5), (64, 40, 24), (97, 51, 13), (40, 41, 4), (31, 2, 8)]
# from two waves of blocks on (303104 points in MIXED) every launch is staged
SIZES += [(97, 51, 62), (33, 400, 24), (2100, 9, 17), (40, 41, 190), (64, 1250, 4)]


def _case(prec_name, size, wild, ntr, seed=3):
    from gem_b200 import adz as A, synth
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    prec = A.PREC_NAMES[prec_name]
    ft = A._field_dtype(prec)
    cfg = synth.config_small(*size)
    cfg.ntracers, cfg.tracer_kind = ntr, "lognormal"
    inp = synth.make_inputs(cfg, device="cuda", dtype=ft)
    if wild == "shear":  # gyres of 24 cells, about two cells per step: many rows per tile
        k, j, i = (torch.arange(n, device="cuda", dtype=torch.float64) for n in inp["uu_ext"].shape)
        i, j, c = 0.262 * i + 0.1 * k.view(-1, 1, 1), 0.262 * j.view(1, -1, 1), 1.9 * cfg.dx / cfg.dt
        for key, f in (("uu_ext", torch.sin(j) * torch.cos(i)), ("vv_ext", -torch.cos(j) * torch.sin(i))):
            inp[key] = (c * f).to(ft).contiguous()
            inp[key.replace("u_ext", "t0").replace("v_ext", "t0")] = inp[key].clone()
    elif wild:  # departure points anywhere within the halo, levels away
        g = torch.Generator(device="cuda").manual_seed(seed)
        for key, amp in (("uu_ext", 2.5 * cfg.dx), ("vv_ext", 2.5 * cfg.dx), ("ww_ext", 1500.0), ("ut0", 2.5 * cfg.dx),
                         ("vt0", 2.5 * cfg.dx), ("zdt0", 1500.0)):
            amp = amp * float(wild)
            r = torch.rand(inp[key].shape, generator=g, device="cuda", dtype=torch.float64)
            inp[key] = ((2.0 * r - 1.0) * amp / cfg.dt).to(ft)
    return A, cfg, prec, ft, inp


def _bits(t):
    return t.contiguous().view(torch.int32 if t.dtype == torch.float32 else torch.int64)


# niter 6 from the arrival points is the cold start
@pytest.mark.parametrize("cold", [False, True])
@pytest.mark.parametrize("wild", [False, True, "shear"])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("prec_name", ["mixed", "fp64"])
def test_staged_step_equals_direct(prec_name, size, wild, cold):
    A, cfg, prec, ft, inp = _case(prec_name, size, wild, 4)
    srcs = [inp["src_u"], inp["src_v"], inp["src_w"]] + inp["tracers"]
    mono = [0, 0, 0, 1, 0, 2, 1]
    nf = [0, 1, 1, len(srcs) - 2]
    new = lambda: [torch.full(s.shape, -7.0, dtype=ft, device="cuda") for s in srcs]  # noqa: E731
    # direct: one phased batch step, warm from the given departure points
    ad = A.Adz.from_config(cfg, lam=False)
    _, wp = ad.new_state(prec)
    ad.adz_inittraj(prec, None, wp)
    arrival = wp.clone()
    ad.adz_traject(prec, cfg.dt, inp, None, wp)
    start = arrival if cold else wp
    wp_d, out_d = start.clone(), new()
    b = A.Batch(prec, [dict(adz=ad, dt=cfg.dt, winds=inp, wpxyz=wp_d, nfields=nf, srcs=srcs, dsts=out_d, mono=mono,
                            niter=6 if cold else 2)])
    b.select(8, A.Batch.PHASED)
    b.step()
    torch.cuda.synchronize()
    # staged
    ad2 = A.Adz.from_config(cfg, lam=False)
    wp_s, out_s = start.clone(), new()
    if cold:
        ad2.adz_inittraj(prec, None, wp_s)
    ad2.adz_traject(prec, cfg.dt, inp, None, wp_s, niter=0 if cold else 2)
    ad2.adz_tricub_sets(prec, nf, srcs, out_s, mono)
    torch.cuda.synchronize()
    assert b.status() == ad2.status()
    assert torch.equal(_bits(wp_s), _bits(wp_d))
    for x, y in zip(out_s, out_d):
        assert torch.equal(_bits(x), _bits(y))


@pytest.mark.parametrize("offset", [0, 1])  # elements of the sources past a 16-byte boundary
@pytest.mark.parametrize("wild", [False, True])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("prec_name,qv,n", [("mixed", False, 3), ("mixed", False, 17), ("fp64", False, 4),
                                            ("mixed", True, 2), ("mixed", True, 3)])
def test_staged_sets_equal_direct(prec_name, qv, n, size, wild, offset):
    A, cfg, prec, ft, inp = _case(prec_name, size, wild, n)
    ad = A.Adz.from_config(cfg, lam=False)
    _, wp = ad.new_state(prec)
    ad.adz_inittraj(prec, None, wp)
    ad.adz_traject(prec, cfg.dt, inp, None, wp)
    shp = ad.ext_shape
    srcs = []
    for t in inp["tracers"]:
        v = torch.empty(t.numel() + offset, dtype=ft, device="cuda")[offset:].view(shp)
        srcs.append(v.copy_(t))
    srcs[0][0, 1, 2] = srcs[0][shp[0] // 2, 5, 6] = srcs[0][-1, -2, -1] = float("nan")
    mono = [(A.QV if qv else 0) | ((1, 0, 2)[q % 3] if not qv else 1 + q % 2) for q in range(n)]
    res = []
    for pert in (None, torch.zeros((cfg.nj, cfg.ni), dtype=ft, device="cuda")):
        new = lambda: [torch.full(shp, -7.0, dtype=ft, device="cuda") for _ in srcs]  # noqa: E731
        out, post = new(), (new(), new(), new())
        ad.set_rhs_perturbation(pert)
        ad.adz_tricub_hlt(prec, A.SET_T, srcs, out, mono=mono, post=post)
        torch.cuda.synchronize()
        res.append(out + [t for p in post for t in p])
    assert ad.status() == 0
    for x, y in zip(*res):  # by value: d + 0 * |d - lin| is d up to the sign of a zero
        assert np.array_equal(x.cpu().numpy(), y.cpu().numpy(), equal_nan=True)


def test_boundary_flux_shared_and_many():
    """More tracers than one launch takes; one of them in its own flux array,
    two more in the flux arrays of the tracers before them."""
    A, cfg, prec, ft, inp = _case("mixed", (56, 44, 12), False, 11)
    ad = A.Adz.from_config(cfg)
    _, wp = ad.new_state(prec)
    ad.adz_inittraj(prec, None, wp)
    ad.adz_traject(prec, cfg.dt, inp, None, wp)
    new = lambda: [torch.zeros(ad.ext_shape, dtype=ft, device="cuda") for _ in inp["tracers"]]  # noqa: E731
    fo, fi = new(), new()
    ad.bc_lam_flux(prec, inp["tracers"], fo, fi)
    # tracer 2 read from the array that receives its outflow
    go, gi = new(), new()
    own = inp["tracers"][2].clone()
    srcs = list(inp["tracers"])
    srcs[2] = go[2] = own
    srcs[9] = go[0] = inp["tracers"][9].clone()
    srcs[10] = gi[8] = inp["tracers"][10].clone()
    m = ad.range_mask(A.SET_B, device="cuda")
    ad.bc_lam_flux(prec, srcs, go, gi)
    torch.cuda.synchronize()
    assert ad.status() == 0 and float(fi[0].abs().max()) > 0 and float(fo[0].abs().max()) > 0
    for q in range(len(srcs)):
        assert torch.equal(fo[q][m], go[q][m]) and torch.equal(fi[q][m], gi[q][m])


# warm REF32 trajectories are staged from 56832 points on; scattered flows of
# less amplitude than above, so that no stencil leaves the oracle's arrays
@pytest.mark.parametrize("wild", [False, 0.5, "shear"])
@pytest.mark.parametrize("size", [(33, 9, 5), (64, 40, 24), (97, 51, 13), (45, 300, 5), (40, 41, 60)])
def test_staged_ref32_equals_oracle(size, wild):
    from oracle import oracle as O
    A, cfg, prec, ft, inp = _case("ref32", size, wild, 1)
    st = O.Step(cfg, kind="oracle", prec="f32", lam=False)
    np_in = {k: inp[k].cpu().numpy() for k in ("uu_ext", "vv_ext", "ww_ext", "ut0", "vt0", "zdt0")}
    ad = A.Adz.from_config(cfg, lam=False)
    px, wp = ad.new_state(prec)
    st.inittraj()
    ad.adz_inittraj(prec, px, wp)
    for niter in (0, 1, 3):  # the first from the arrival points
        st.traject(np_in, niter or None)
        ad.adz_traject(prec, cfg.dt, inp, px, wp, niter=niter)
        torch.cuda.synchronize()
        assert ad.status() == 0
        own = (slice(None), slice(None), slice(2, -2), slice(2, -2))
        assert np.array_equal(px.cpu().numpy().view(np.int32), st.pxyzm.view(np.int32))
        assert np.array_equal(wp.cpu().numpy()[own].view(np.int64), st.wpxyz[own].view(np.int64))


@pytest.mark.parametrize("wild", [False, 0.5, "shear"])
@pytest.mark.parametrize("size", [(33, 9, 5), (64, 40, 24), (97, 51, 13), (40, 41, 4), (31, 2, 8)])
def test_tolerance_equals_fixed_updates(size, wild):
    """The iteration to a tolerance (staged at every size) against fixed
    updates of the direct kernel (small tiles): from the arrival points, from
    stored points that converge at once, and with the fallback of a start that
    does not; updates and counts."""
    from gem_b200 import guess
    A, cfg, prec, ft, inp = _case("mixed", size, wild, 1)
    ad = A.Adz.from_config(cfg, lam=False)
    n = cfg.ni * cfg.nj * cfg.nk
    _, stored = ad.new_state(prec)
    ad.adz_inittraj(prec, None, stored)
    ad.adz_traject(prec, cfg.dt, inp, None, stored)

    def run(tol, maxit, start):
        wp = stored.clone()
        it = torch.zeros(n, dtype=torch.uint8, device="cuda")
        st = torch.zeros(3, dtype=torch.int64, device="cuda")
        guess.traject_tol(ad, prec, cfg.dt, inp, wp, tol=tol, maxit=maxit, start=start, iters=it, stats=st)
        torch.cuda.synchronize()
        return wp, it.cpu().numpy(), st.cpu().tolist()

    def fixed(niter, cold):
        wp = stored.clone()
        if cold:
            ad.adz_inittraj(prec, None, wp)
        ad.adz_traject(prec, cfg.dt, inp, None, wp, niter=niter)
        torch.cuda.synchronize()
        return wp

    own = (slice(None), slice(None), slice(2, -2), slice(2, -2))
    # tolerance 0: a point stops where an update does not move it (further
    # updates would not either), else it takes all of them
    for tol, maxit, start, counts in ((0.0, 4, 0, [4 * n, 0, n]), (1e9, 3, 1, [n, 0, 0]), (0.0, 2, 1, [4 * n, n, n])):
        wp, it, st = run(tol, maxit, start)
        assert ad.status() == 0
        back = torch.from_numpy(it >= 128).cuda().view(cfg.nk, cfg.nj, cfg.ni)
        cold = fixed(maxit, True) if start == 0 or bool(back.any()) else wp
        warm = fixed(1 if tol > 0.0 else maxit, False) if start == 1 else cold
        assert ad.status() == 0
        assert torch.equal(_bits(wp[own]), torch.where(back, _bits(cold[own]), _bits(warm[own])))
        assert st[0] == int((it & 127).sum()) and st[1] == int(back.sum())
        if wild == 0.5 or tol > 0.0:  # no point stops early
            assert st == counts


def test_more_rows_than_the_staged_grid():
    """Above 131070 rows the grid of the staged kernels does not fit and the
    direct ones run: the rows of a tile of 131100 against those of one of
    131000, away from the upper edge."""
    from gem_b200 import guess
    A, cfg, prec, ft, big = _case("mixed", (8, 131100, 4), 0.5, 4)
    rows = 130900
    got = []
    for nj in (131100, 131000):
        cfg.nj = nj
        njt = nj + 2 * cfg.halo
        inp = {k: v[:, :njt].contiguous() for k, v in big.items() if k not in ("tracers", "uslt", "vslt")}
        trs = [t[:, :njt].contiguous() for t in big["tracers"]]
        ad = A.Adz.from_config(cfg, lam=False)
        _, wp = ad.new_state(prec)
        ad.adz_inittraj(prec, None, wp)
        ad.adz_traject(prec, cfg.dt, inp, None, wp)
        ad.adz_traject(prec, cfg.dt, inp, None, wp, niter=2)
        out = [torch.zeros(ad.ext_shape, dtype=ft, device="cuda") for _ in range(8)]
        ad.adz_tricub_hlt(prec, A.SET_T, trs, out[:4], mono=[1, 0, 1, 0])
        ad.adz_tricub_hlt(prec, A.SET_T, trs, out[4:], mono=[A.QV | 1] * 4)
        tol = wp.clone()
        it = torch.zeros(cfg.ni * nj * cfg.nk, dtype=torch.uint8, device="cuda")
        guess.traject_tol(ad, prec, cfg.dt, inp, tol, start=0, iters=it)
        torch.cuda.synchronize()
        assert ad.status() == 0
        H = cfg.halo
        got.append([w[:, :, 2:2 + rows, 2:-2] for w in (wp, tol)] + [o[:, H:H + rows] for o in out] +
                   [it.view(cfg.nk, nj, cfg.ni)[:, :rows]])
    for a, b in zip(*got):
        assert torch.equal(a, b) and float(a.double().abs().max()) > 0


# REF32 starts from the stored FP32 positions as they are.  maxcfl 1 (halo 2):
# the stencil corner of a position beyond the range of int is its last int.
# Not a number counts as cell 0, and the winds found there as not finite
@pytest.mark.parametrize("bad,status", [(float("nan"), 5), (3e9, 4), (-3e9, 4), (float("inf"), 4), (-float("inf"), 4)])
def test_ref32_position_without_a_cell(bad, status):
    """A point whose stored position has no cell in the array is reported as
    such and left as it is; the others are untouched by it."""
    from gem_b200 import adz as A, synth
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    cfg = synth.config_small(70, 21, 9)
    cfg.maxcfl, cfg.dt = 1, 60.0
    inp = synth.make_inputs(cfg, device="cuda", dtype=torch.float32)
    ad = A.Adz.from_config(cfg, lam=False)
    px, wp = ad.new_state(A.REF32)
    ad.adz_inittraj(A.REF32, px, wp)
    ad.adz_traject(A.REF32, cfg.dt, inp, px, wp)
    start_px, start_wp = px.clone(), wp.clone()
    ad.adz_traject(A.REF32, cfg.dt, inp, px, wp)
    torch.cuda.synchronize()
    assert ad.status() == 0
    for k, j, i in ((0, 0, 0), (4, 10, 2), (8, 20, 69)):
        px2, wp2 = start_px.clone(), start_wp.clone()
        px2[k, j, i, 0] = bad
        before = px2[k, j, i].clone()
        ad.adz_traject(A.REF32, cfg.dt, inp, px2, wp2)
        torch.cuda.synchronize()
        assert ad.status() == status
        assert torch.equal(_bits(px2[k, j, i]), _bits(before))
        px2[k, j, i] = px[k, j, i]
        wp2[:, k, j + 2, i + 2] = wp[:, k, j + 2, i + 2]
        assert torch.equal(_bits(px2), _bits(px)) and torch.equal(_bits(wp2), _bits(wp))
