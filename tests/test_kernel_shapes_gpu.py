"""The kernels at the sizes where their tiling can go wrong -- remainders of
lanes, groups, positions and angles, the smallest and largest of each form --
against the FP64 oracle.

Tolerances: FP64 operators 1e-11 of the peak, FP64 lite steps 1e-10 (as in
test_parity_gpu.py).  Float state starts from float values, so an operator's
error is that of its float arithmetic: one rounding of the result for the
energy sweep (2^-24 = 6e-8, bar 1e-6), some thirty operations on differences of
neighbours for the transport (bar 2e-6), four passes of up to 32 products for
the angular step (4 * 32 * 2^-24 = 8e-6, bar 2e-5)."""
import numpy as np
import pytest

from conftest import rel_err, table_dir
from test_parity_gpu import OP_TOL, STEP_TOL, assert_states, build, seeded_states, set_both, small_cfg
from test_bundle_gpu import alone, check, pick
from test_out_of_core_gpu import cfg_of, compare
from bfpn_gpu_b200 import capi, read_tables

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

PRECISIONS = [capi.PREC_FP64, capi.PREC_MIXED]


def _states(ctx, seed, precision):
    s = seeded_states(ctx, seed)
    return [a.astype(np.float32).astype(np.float64) for a in s] if precision == capi.PREC_MIXED else s


# (ny, nz, nmu, nom, ng): one lane per thread with 1, 2, 4 and 3 mod 4 groups;
# vectors (75,776 float / 37,888 double lanes and more) with odd and even groups,
# whole and partial operand tiles of positions and angles
ENERGY_SHAPES = [(3, 2, 3, 3, 5), (4, 4, 5, 7, 2), (6, 5, 4, 5, 40), (2, 8, 9, 1, 43), (17, 17, 16, 16, 7),
                 (20, 21, 14, 14, 6)]


def _energy_cfg(shape, **flags):
    ny, nz, nmu, nom, ng = shape
    return small_cfg(ny=ny, nz=nz, nmu=nmu, nom=nom, ng=ng, lg=1.475 * ng, beam_energy=1.0 * ng, **flags)


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("flags", [{}, {"eq15_straggling": True, "trapezoidal_yz": True}, {"legacy_energy": True}])
@pytest.mark.parametrize("shape", ENERGY_SHAPES)
def test_energy_sweep_shapes(shape, flags, precision):
    cfg = _energy_cfg(shape, **flags)
    ctx, ora = build(cfg, precision=precision)
    set_both(ctx, ora, _states(ctx, 41, precision))
    ctx.energy(0, 0.5 * cfg.dt())
    ora.energy(0, 0.5 * cfg.dt())
    assert_states(ctx, ora, OP_TOL if precision == capi.PREC_FP64 else 1e-6, ((0, 0), (0, 1)))


# with a source (from 12 groups on these tables have one): 0 to 3 mod 4 groups;
# the last three take one lane per thread in FP64 and balance to blocks of 608,
# 640 and, over several rounds, 640 threads where the ring lets them
SOURCED_SHAPES = [(6, 5, 4, 5, 40), (2, 8, 9, 1, 43), (3, 2, 3, 3, 17), (4, 4, 5, 7, 18), (17, 17, 16, 16, 16),
                  (20, 21, 14, 14, 19), (26, 26, 11, 11, 16), (19, 19, 15, 15, 16), (100, 100, 9, 11, 12)]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("flags", [{}, {"eq15_straggling": True, "trapezoidal_yz": True}, {"legacy_energy": True}])
@pytest.mark.parametrize("shape", SOURCED_SHAPES)
def test_sourced_energy_sweep_shapes(shape, flags, precision):
    cfg = _energy_cfg(shape, **flags)
    ctx, ora = build(cfg, precision=precision)
    states = _states(ctx, 47, precision)
    set_both(ctx, ora, states)
    h = 0.5 * cfg.dt()
    ora.energy(1, h)
    plain = [ora.get_state(1, cf) for cf in (0, 1)]
    ora.set_state(1, 0, states[2])
    ora.set_state(1, 1, states[3])
    ctx.secondary_source()
    ora.source()
    ctx.energy(1, h, with_source=True)
    ora.energy(1, h, with_source=True)
    if precision == capi.PREC_FP64:
        assert_states(ctx, ora, OP_TOL, ((1, 0), (1, 1)))
    added = 0.0
    for cf in (0, 1):
        want = ora.get_state(1, cf)
        d = np.abs(want - plain[cf]).max()
        # the sweep's own rounding, and the bar of the float source on what it adds
        assert np.abs(ctx.get_state(1, cf) - want).max() <= 1e-6 * np.abs(want).max() + 2e-5 * d
        added = max(added, d)
    assert added > 0


# a whole step at the same blocks: its IDD, summed from the sweeps' partials, is
# that of the state it leaves.  Sums of double terms some 200 additions deep
# (24 groups, a block's tree, its 150 blocks) in two orders: 1e-12 of the sum of
# their magnitudes
@pytest.mark.parametrize("ny,ang", [(26, 11), (19, 15)])
def test_odd_angle_step_dose(ny, ang):
    cfg = small_cfg(ny=ny, nz=ny, nmu=ang, nom=ang, ng=24)
    ctx, _ = build(cfg)
    ctx.step(1)  # the first step has no secondary half
    for k, a in enumerate(_states(ctx, 48, capi.PREC_FP64)):
        ctx.set_state(k // 2, k % 2, a)
    got = ctx.step(1)[0][0]
    want = ctx.idd()[0]
    left = [ctx.get_state(k // 2, k % 2) for k in range(4)]
    terms = 0.0
    for keep in (0, 1):
        for k, a in enumerate(left):
            ctx.set_state(k // 2, k % 2, np.abs(a) if k % 2 == keep else np.zeros_like(a))
        terms += abs(ctx.idd()[0])
    assert np.abs(left[2]).max() > 0 and terms > 0
    assert abs(got - want) <= 1e-12 * terms


def test_out_of_core_odd_angle_chunks():
    """Lane chunks of 33 x 33 positions x 81 angles (608 threads), the last partial."""
    compare(cfg_of(ny=49, nz=49, nmu=9, nom=9, ng=24, ly=8.0, lz=8.0, t_final=0.5), capi.PREC_FP64, 4, (1089 * 81, 5))


@pytest.mark.parametrize("straggling", [False, True])
@pytest.mark.parametrize("shape", ENERGY_SHAPES)
def test_fused_pass_shapes(shape, straggling):
    """Steps with the fused primary pass against the separate passes, states
    as test_parity_gpu.py compares them (one rounding far below the peak)."""
    cfg = _energy_cfg(shape, eq15_straggling=straggling, trapezoidal_yz=straggling)
    got = []
    for fused in (0, 1):
        ctx, _ = build(cfg, precision=capi.PREC_MIXED)
        ctx.set_option(capi.OPT_STEP_OVERLAP, 2 * fused)
        ctx.set_option(capi.OPT_FUSED_ENERGY, fused)
        ctx.step(4)
        got.append([ctx.get_state(sp, cf) for sp in (0, 1) for cf in (0, 1)])
    for a, b in zip(*got):
        peak = np.abs(a).max()
        assert np.abs(a - b).max() <= 1e-12 * peak
        big = np.abs(a) >= 1e-6 * peak
        assert np.array_equal(a[big], b[big])


# widths: one position to 128 over every (lanes, positions per lane) form and
# both of its ends; angle grids whose pairs all share signs (4 x 4), partly do
# (5 x 6, lone angles and mixed warps) or lack a partner (5 x 3, odd rows)
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("ny,nz,ang", [(1, 3, (4, 4)), (2, 1, (5, 6)), (7, 9, (5, 3)), (8, 3, (4, 4)), (11, 2, (5, 6)),
                                       (23, 5, (5, 3)), (32, 4, (5, 6)), (37, 29, (4, 4)), (47, 2, (2, 2)),
                                       (48, 5, (5, 6)), (64, 3, (5, 3)), (80, 6, (5, 6)), (95, 2, (4, 4)),
                                       (96, 3, (5, 6)), (127, 2, (5, 3)),
                                       # beyond one line-walk tile: float's lone angles march too
                                       (7, 100, (5, 6)), (11, 70, (5, 3)), (27, 28, (3, 3)), (32, 24, (5, 6)),
                                       (47, 17, (5, 3)), (64, 12, (5, 6)), (96, 8, (5, 3)), (127, 6, (5, 6))])
def test_march_transport_shapes(ny, nz, ang, precision):
    cfg = small_cfg(ny=ny, nz=nz, nmu=ang[0], nom=ang[1], ng=3, ly=0.2 * ny, lz=0.25 * nz)
    ctx, ora = build(cfg, precision=precision)
    Ng, nyz, NA = ctx.shape
    states = [a.reshape(Ng, nyz, NA) for a in _states(ctx, 42, precision)]
    for a in states:
        a[1, : nyz // 2] = a[1, 0]                                   # flat
        a[2] = np.float32(3e-11) * np.arange(nyz)[:, None]            # differences around the limiter's epsilon
    if precision == capi.PREC_MIXED:
        states = [a.astype(np.float32).astype(np.float64) for a in states]
    set_both(ctx, ora, [a.ravel() for a in states])
    for sp, cf, dtf, keep in ((0, 0, 0.5, False), (0, 1, 0.5, True), (1, 0, 0.31, False), (1, 1, 0.5, True)):
        ctx.transport(sp, cf, dtf * cfg.dt(), keep)
        ora.transport(sp, cf, dtf * cfg.dt(), keep)
    assert_states(ctx, ora, OP_TOL if precision == capi.PREC_FP64 else 2e-6)


# rows and columns of different lengths, lengths without a square kernel, one
# line, odd counts of lines, tiles over the end of a group
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("nom,nmu", [(15, 12), (12, 15), (1, 7), (8, 1), (32, 3), (5, 32), (31, 31), (26, 30), (9, 17)])
def test_rectangular_angle_shapes(nom, nmu, precision):
    cfg = small_cfg(ny=4, nz=6, nmu=nmu, nom=nom, ng=5, lz=2.0)
    ctx, ora = build(cfg, precision=precision)
    set_both(ctx, ora, _states(ctx, 43, precision))
    for sp, cf in ((0, 0), (1, 1)):
        ctx.angle(sp, cf, 0.7 * cfg.dt())
        ora.angle(sp, cf, 0.7 * cfg.dt())
    assert_states(ctx, ora, OP_TOL if precision == capi.PREC_FP64 else 2e-5)


# odd and even angle counts, partial 32-output tiles and 8-row chunks, positions
# around one 64-position tile; the last grid's kernel has zero blocks
@pytest.mark.parametrize("ny,nz,nmu,nom,ng,tables", [(3, 4, 3, 3, 40, "synthetic500"), (7, 7, 5, 7, 40, "synthetic500"),
                                                     (8, 6, 8, 8, 40, "synthetic500"), (2, 2, 20, 20, 500, "water")])
def test_fp64_source_shapes(ny, nz, nmu, nom, ng, tables):
    cfg = small_cfg(ny=ny, nz=nz, nmu=nmu, nom=nom, ng=ng, lg=0.518 * ng if ng == 500 else 59.0,
                    beam_energy=230.0 if ng == 500 else 40.0)
    ctx, ora = build(cfg, tables=tables)
    set_both(ctx, ora, seeded_states(ctx, 44))
    ctx.secondary_source()
    s = ora.source()
    assert np.abs(s).max() > 0
    assert rel_err(ctx.source(), s) < OP_TOL


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("ny,nz,nmu,nom,ng", [(2, 3, 3, 3, 2), (6, 5, 4, 5, 43), (17, 17, 16, 16, 9)])
def test_lite_step_shapes(ny, nz, nmu, nom, ng, precision):
    cfg = small_cfg(ny=ny, nz=nz, nmu=nmu, nom=nom, ng=ng, lg=1.475 * ng, beam_energy=1.0 * ng, lite_memory=True,
                    trapezoidal_yz=True)
    ctx, ora = build(cfg, precision=precision)
    idd_g, prox = ctx.step(6)
    idd_o, _ = ora.step(6)
    # float: one rounding of the state per step and group above (6e-8 each)
    tol = STEP_TOL if precision == capi.PREC_FP64 else 2e-6
    assert np.abs(idd_o).max() > 0 and not np.any(prox)
    assert rel_err(idd_g, idd_o) < tol
    a, b = ctx.get_state(0, 0), ora.get_state(0, 0)
    # (two groups lose the beam within the steps: float values end below 2^-126, where a rounding is 2^-150)
    floor = 0.0 if precision == capi.PREC_FP64 else 6 * 2.0 ** -149
    assert np.abs(a - b).max() <= tol * np.abs(b).max() + floor


# 16-byte pieces and not (a caller's array may start at any value; odd lane
# counts), fewer groups than one share, with and without the secondary
@pytest.mark.parametrize("dtype,precision", [(torch.float64, capi.PREC_FP64), (torch.float32, capi.PREC_MIXED)])
@pytest.mark.parametrize("ny,nz,nmu,nom,ng,shift", [(2, 2, 3, 3, 3, 0), (6, 5, 4, 6, 41, 0), (6, 5, 4, 6, 41, 1),
                                                    (20, 21, 12, 12, 19, 0), (4, 4, 5, 5, 100, 2)])
def test_caller_owned_dose_shapes(ny, nz, nmu, nom, ng, shift, dtype, precision):
    cfg = small_cfg(ny=ny, nz=nz, nmu=nmu, nom=nom, ng=ng, trapezoidal_yz=True)
    g = cfg.grid()
    n = ng * (ny + 1) * (nz + 1) * nmu * nom
    rng = torch.Generator(device="cuda").manual_seed(5)
    own = [torch.rand(n + shift, device="cuda", dtype=dtype, generator=rng)[shift:] for _ in range(4)]
    w = torch.rand(2 * ng, device="cuda", dtype=torch.float64, generator=rng)
    wy, wz = np.ones(ny + 1), np.ones(nz + 1)
    wy[[0, -1]], wz[[0, -1]] = 0.5, 0.5
    pos = torch.from_numpy((wz[:, None] * wy[None, :]).ravel()).cuda()[None, :, None]
    F0, f0, F1, f1 = [a.double().view(ng, -1, nmu * nom) for a in own]
    k = w.view(ng, 2, 1, 1)
    vol = g.Ly / ny * g.Lz / nz * g.Lu / (nom + 1) * g.Lv / (nmu + 1)
    for second in (True, False):
        out = torch.zeros(2, device="cuda", dtype=torch.float64)
        ptr = [a.data_ptr() for a in own]
        capi.idd_noalloc(g, precision, True, ptr[0], ptr[1], ptr[2] if second else None, ptr[3] if second else None,
                         w.data_ptr(), out.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        psi1, psi2 = (F0 + F1, f0 + f1) if second else (F0, f0)
        want = [float(((k[:, 0] * psi1 + k[:, 1] * psi2) * pos).sum()) * vol, float(f0.sum()) * g.Lg / ng]
        # sums of at most 2e7 positive terms in double: 1e-11 covers any order
        assert np.allclose(out.cpu().numpy(), want, rtol=1e-11, atol=0.0)


# 48 positions and 16-column remainders of the tensor-core output tile, odd angle
# counts, one position tile exactly, one more and one less; bars as for the same
# operator in test_parity_gpu.py
@pytest.mark.parametrize("ny,nz,nmu,nom", [(7, 5, 6, 8), (8, 6, 7, 9), (7, 7, 4, 4), (12, 4, 11, 3), (6, 8, 16, 17)])
def test_tensor_core_source_shapes(ny, nz, nmu, nom):
    cfg = small_cfg(ny=ny, nz=nz, nmu=nmu, nom=nom)
    ctx, ora = build(cfg, precision=capi.PREC_MIXED)
    set_both(ctx, ora, _states(ctx, 45, capi.PREC_MIXED))
    s = ora.source()
    ctx.secondary_source()
    assert np.abs(s).max() > 0
    assert rel_err(ctx.source(), s) < 2e-5


# below the staging size, just above it, a partial last chunk, an odd count
@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("ny,nz,nmu,nom,ng", [(15, 15, 8, 8, 128), (15, 16, 8, 16, 65), (16, 16, 16, 16, 40),
                                              (26, 24, 7, 9, 101)])
def test_state_transfer_round_trip(ny, nz, nmu, nom, ng, precision):
    """Values that both precisions hold come back as they went in."""
    cfg = small_cfg(ny=ny, nz=nz, nmu=nmu, nom=nom, ng=ng, lg=1.475 * ng, beam_energy=1.0 * ng)
    ctx, _ = build(cfg, precision=precision)
    n = int(np.prod(ctx.shape))
    a = (np.arange(n) % 65521).astype(np.float64) * 2.0 ** -20
    b = -a[::-1].copy()
    ctx.set_state(0, 0, a)
    ctx.set_state(1, 1, b)
    ctx.set_state(0, 0, b)
    assert np.array_equal(ctx.get_state(1, 1), b)
    assert np.array_equal(ctx.get_state(0, 0), b)


@pytest.mark.parametrize("n", [255, 256, 257])
def test_step_call_lengths(n):
    """Results of one call around the most steps one export holds, against the
    history of single steps bit for bit (the lite step has no fused forms)."""
    cfg = small_cfg(ny=3, nz=3, nmu=3, nom=3, nx=300, lite_memory=True)
    one, _ = build(cfg)
    idd, prox = one.step(n)
    many, _ = build(cfg)
    got = [many.step(1) for _ in range(n)]
    assert len(idd) == n and np.array_equal(idd, np.concatenate([g[0] for g in got]))
    assert np.array_equal(prox, np.concatenate([g[1] for g in got]))
    assert np.array_equal(one.get_state(0, 0), many.get_state(0, 0))


# the default chunk of the whole-plane kernel changes at 33 points (16, 8 angles)
@pytest.mark.parametrize("ny,nmu,nom", [(20, 5, 4), (24, 3, 6), (32, 5, 4)])
def test_plane_transport_default_chunk(ny, nmu, nom):
    cfg = small_cfg(ny=ny, nz=ny, nmu=nmu, nom=nom, ng=7, lg=1.475 * 7, beam_energy=7.0)
    ctx, ora = build(cfg, precision=capi.PREC_MIXED)
    set_both(ctx, ora, _states(ctx, 46, capi.PREC_MIXED))
    for sp, cf in ((0, 0), (1, 1)):
        ctx.transport(sp, cf, 0.5 * cfg.dt(), cf == 1)
        ora.transport(sp, cf, 0.5 * cfg.dt(), cf == 1)
    assert_states(ctx, ora, 2e-6)


# one step too short for a tuning run, exactly one, one longer (bars of test_bundle_gpu.py)
@pytest.mark.parametrize("n", [5, 6, 7])
def test_bundle_tuning_lengths(n):
    reqs = pick(16, 12, 2, n)
    refs = [alone(r) for r in reqs]
    with capi.Bundle(max_slots=2) as b:
        slots = [b.admit(r.beam()) for r in reqs]
        b.step(1000)
        b.sync()
        assert b.running() == 0
        for s, ref in zip(slots, refs):
            check(b.collect(s), ref)


# classes that no other test uses: the choice is kept for the process
@pytest.mark.parametrize("ny,na,n,call", [(14, 8, 9, 2), (12, 16, 5, 1000)])
def test_bundle_tunes_in_short_runs(ny, na, n, call):
    """Calls of two steps, and beams of five one after another, tune the bundle as
    longer ones do."""
    reqs = pick(ny, na, 2, n)
    with capi.Bundle(max_slots=1) as b:
        assert b.tuning() == "not tuned"
        for r in reqs:
            ref = alone(r)
            slot = b.admit(r.beam())
            while b.running():
                b.step(call)
            check(b.collect(slot), ref)
        assert "lane" in b.tuning()


def test_downloaded_angular_kernel_is_the_one_in_use():
    """Unit values of psi^1, one direction at each position: the source is the
    group's angular kernel times its energy kernel and the group width, product by
    product, so the table a FP64 context returns gives it bit for bit.  Against the
    host's build of that table the entries agree to the last bits of acos, pow and
    exp (a few 1e-16 each, times exponents below 100: 1e-12), but for one within
    those of the threshold 1e-3, which either side may drop."""
    cfg = small_cfg(ny=6, nz=6, nmu=6, nom=8)
    ctx, _ = build(cfg)
    Ng, nyz, NA = ctx.shape
    K = ctx.table(capi.TABLE_KER_V, Ng * NA * NA).reshape(Ng, NA, NA)
    e1 = ctx.table(capi.TABLE_KER_E1, Ng * Ng).reshape(Ng, Ng)
    for s in (2, 7, 20):
        F = np.zeros((Ng, nyz, NA))
        F[s, np.arange(nyz), np.arange(nyz) % NA] = 1.0
        ctx.set_state(0, 0, F.ravel())
        ctx.set_state(0, 1, np.zeros(F.size))
        ctx.secondary_source()
        want = cfg.grid().Lg / Ng * (e1[:, s, None, None] * K[s][np.arange(nyz) % NA][None])
        assert np.count_nonzero(want) > nyz
        assert np.array_equal(ctx.source().reshape(Ng, nyz, NA), want)
    mu, sig = read_tables(table_dir("synthetic500"), cfg.ng)
    H = capi.host_table(cfg.grid(), cfg.phys(), mu, sig, capi.TABLE_KER_V).reshape(K.shape)
    one = (K == 0) != (H == 0)
    assert np.all(np.abs(np.maximum(K, H)[one] - 1e-3) <= 1e-15)
    assert np.all(np.abs(K - H)[~one] <= 1e-12 * H[~one])


def _page_locked_kb():
    """Page-locked host memory that the driver has mapped into this process."""
    kb = 0
    with open("/proc/self/maps") as maps:
        for line in maps:
            if "/dev/zero" in line:
                lo, hi = line.split()[0].split("-")
                kb += (int(hi, 16) - int(lo, 16)) // 1024
    return kb


@pytest.mark.parametrize("precision", PRECISIONS)
def test_step_calls_lock_no_memory(precision):
    """The buffer of a step call's results is no allocation of page-locked memory
    (which takes longer than the step of a small beam); the first calls, which
    copy, and the later ones, which do not, give the history."""
    cfg = small_cfg()
    ctx, _ = build(cfg, precision=precision)
    ctx.step_async(2)
    ctx.sync()
    before = _page_locked_kb()
    got = [ctx.step(n) for n in [1, 256] + [1] * 29 + [3, 2, 1, 256]]
    assert _page_locked_kb() == before
    idd, prox = ctx.history()
    assert np.array_equal(np.concatenate([g[0] for g in got]), idd[2:])
    assert np.array_equal(np.concatenate([g[1] for g in got]), prox[2:])


@pytest.mark.parametrize("precision", PRECISIONS)
def test_large_transfers_lock_no_memory(precision):
    """A context's first large state transfers allocate no page-locked memory
    (which takes longer than the transfer), and later ones through buffers locked
    in place (from 128 MB on) bring the same values."""
    cfg = small_cfg(ny=16, nz=16, nmu=16, nom=16, ng=40)
    ctx, _ = build(cfg, precision=precision)
    before = _page_locked_kb()
    a = (np.arange(int(np.prod(ctx.shape))) % 4093).astype(np.float64)
    for k in range(8):
        ctx.set_state(k // 2 % 2, k % 2, a + k)
        assert np.array_equal(ctx.get_state(k // 2 % 2, k % 2), a + k)
    assert _page_locked_kb() == before
