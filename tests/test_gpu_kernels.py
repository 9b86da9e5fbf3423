"""Kernels at the sizes where they can go wrong: ends of tiles, remainders and
the smallest and largest lengths of each launch shape."""
import numpy as np
import pytest

from oracle import oracle as O
from tests import test_gpu_dropin as D
from tests._helpers import bit_equal, rand_field, rel_l2
from tests.test_gpu_step import STATE, make_case, make_ctx, run_oracle
from vtkmakecompare_b200 import legacy as G
from vtkmakecompare_b200 import solver as S

pytestmark = pytest.mark.gpu


# x lengths of the partitioned lines: the shortest and longest of 4, 8, 16 and 32
# lanes, with equal and unequal partitions; odd y and z lengths.  Tolerance: the
# one every step is held to (test_gpu_step).
@pytest.mark.parametrize("n", [(12, 13, 12), (20, 14, 15), (24, 13, 18), (45, 17, 12),
                               (50, 15, 20), (125, 13, 12), (135, 13, 15), (250, 14, 12),
                               (270, 13, 12), (500, 13, 12)])
def test_x_lines_of_any_length_match_oracle(n):
    g, f, c1, par = make_case(*n)
    assert c1.any()
    ref = run_oracle(g, f, c1, par, 3)
    with make_ctx(g, f, c1, par) as ctx:
        ctx.step(3)
        for k in ("u", "v", "w", "p", "T", "u_ta", "T_pre"):
            assert rel_l2(ctx.download(k), ref.f[k]) < 1e-10, k


# Inside one call, steps that another two follow write only what the next step
# reads (k_correct_step, the wrapped divergence, u_ta from phi under the mask);
# one call per step writes every field every time.  Same bits, with a mask that
# crosses the periodic faces and touches both walls, on grids with remainders of
# the correction's 32 x 8 x 4 tiles and without; replayed and eager steps.
@pytest.mark.parametrize("prec,n", [(S.FP64, (50, 15, 20)), (S.FP64, (64, 16, 12)),
                                    (S.FP64, (90, 14, 25)), (S.MIXED, (96, 17, 15)),
                                    (S.MIXED, (64, 24, 18))])
def test_steps_of_one_call_match_calls_of_one_step(prec, n):
    g, f, _, par = make_case(*n, seed=21)
    X, Y, Z = np.ogrid[:n[0], :n[1], :n[2]]
    c1 = np.asfortranarray(0.5 * ((X < 3) | (X >= n[0] - 2)) + 0.25 * (Z < 2) +
                           0.25 * ((Y < 2) | (Y >= n[1] - 2)) + 0.0 * X)
    out = []
    for calls in ([1] * 13, [13], [2, 3, 4, 4]):
        cfg = S.Config(*n, par["dt"], par["Re"], par["Sc"], 50.0, g["xl"], g["yl"], g["zl"],
                       y0=-1.0, ystretch=2.0, body_force=par["force"], t_bot=par["tbot"],
                       t_solid=par["tsolid"], precision=prec)
        with S.Context(cfg) as ctx:
            for k in ("u", "v", "w", "T"):
                ctx.upload(k, f[k])
            ctx.upload("cellvalue", c1)
            ctx.project()
            ctx.start()
            ctx.set_shapes(0, 0)
            ctx.set_line_shapes(0, 2)
            for m in calls:
                ctx.step(m)
            out.append({k: ctx.download(k) for k in STATE})
    for other in out[1:]:
        for k in STATE:
            assert np.array_equal(out[0][k], other[k]), k


# Level-set sweeps, bit for bit: a rough field (ridges, where both one-sided
# slopes count), zeros (NaN in the reference) and ghosts of its own, on grids with
# remainders of the 32 x 8 blocks; sweep counts below, at and past the replayed graph.
# Values too large for reciprocal quotients and infinities take the dividing form.
@pytest.mark.parametrize("n,nnn,big", [((36, 9, 5), 0, 0), ((30, 8, 3), 1, 0), ((64, 17, 6), 40, 0),
                                       ((6, 5, 4), 128, 0), ((40, 12, 9), 129, 0),
                                       ((32, 8, 4), 200, 0), ((90, 60, 75), 5, 0),
                                       ((30, 8, 5), 30, 1e190), ((30, 8, 5), 3, np.inf),
                                       ((30, 8, 5), 3, 1e-200)])
def test_levelset_sweeps_match_oracle_bit_for_bit(n, nnn, big):
    rng = np.random.default_rng(nnn + n[0])
    g = O.Grid(*n, 2.0, 1.5, 1.0, y0=-0.5, gamma=1.3)
    phi0 = np.asfortranarray(0.3 * rng.standard_normal([m + 2 for m in n]))
    if nnn < 100:
        phi0[3, 3, 2] = 0.0
    if big:
        phi0[5, 4, 3] = big
        phi0[0, 2, 2] = -big
    phi, _ = O.set_levelset(g, phi0, nnn=nnn, dtau=1.0e-3, width=1.5)
    cfg = S.Config(*n, 1e-3, 100.0, 1.0, 1.0, 2.0, 1.5, 1.0, y0=-0.5, ystretch=1.3)
    with S.Context(cfg) as ctx:
        got = ctx.levelset(phi0, nnn=nnn, dtau=1.0e-3, width=1.5)
    assert np.array_equal(got, phi, equal_nan=True)


# Drop-in calls large enough for the pinned slots: rows that fill a slot with and
# without a remainder, few long rows, many short ones.  SET_CONVECT and PHIBC round
# like the oracle, so whole fields and boxes are compared bit for bit; MKP and SPN
# for what they leave alone.
@pytest.mark.parametrize("n", [(90, 61, 50), (500, 7, 12), (20, 80, 90), (64, 62, 64)])
def test_drop_ins_through_pinned_slots(n):
    nx, ny, nz = n
    g, go = D.grid(*n)
    rng = np.random.default_rng(nx)
    ref = [rand_field(rng, *n) for _ in range(7)]
    got = [v.copy(order="F") for v in ref]
    O.set_convect(*ref[:6], 0.01, go)
    G.set_convect(*got[:6], 0.01, nx, ny, nz, g["dx"], g["dy"], g["dz"], g["dx12"], g["dy12"],
                  g["dz12"])
    O.phibc(nx, ny, nz, ref[6])
    G.phibc(nx, ny, nz, got[6])
    for a, b in zip(ref, got):
        assert bit_equal(a, b)
    f = {k: rand_field(rng, *n) for k in ("p", "us", "vs", "ws", "u_ta", "v_ta", "w_ta", "u_ep2",
                                          "v_ep2", "w_ep2", "divu", "u", "v", "w")}
    old = {k: v.copy(order="F") for k, v in f.items()}
    G.mkp(f["p"], f["us"], f["vs"], f["ws"], 0.013, g["dx"], g["dy"], g["dz"], g["dx12"],
          g["dy12"], g["dz12"], 1.0, nx, ny, nz, 1, f["u_ta"], f["v_ta"], f["w_ta"], f["u_ep2"],
          f["v_ep2"], f["w_ep2"], f["divu"], f["u"], f["v"], f["w"], g["xl"], g["zl"])
    for k in f:
        written = np.zeros([m + 2 for m in n], bool)
        if k in ("u", "v", "w", "u_ta", "v_ta", "w_ta"):
            written[:-1, :-1, :-1] = True
        elif k not in ("us", "vs", "ws"):
            written[1:-1, 1:-1, 1:-1] = True
        assert bit_equal(f[k][~written], old[k][~written]), k
        assert not np.any(f[k][written] == old[k][written]) or k == "v", k
    Y = np.asfortranarray(rng.standard_normal((nx // 2 + 1, ny + 2, nz + 2)) + 0j)
    Z = Y.copy(order="F")
    G.spn(*n, *O.mkp_coeffs(go), Z)
    assert bit_equal(Z[:, [0, ny + 1]], Y[:, [0, ny + 1]]) and bit_equal(Z[..., nz:], Y[..., nz:])
    assert np.array_equal(Z[0, :, 0], Y[0, :, 0]) and not np.any(Z[1:, 1:-1, :nz] == Y[1:, 1:-1, :nz])


# SPN by pipelined columns: one row, chunks of 16 rows with and without a
# remainder, the lengths where 32, 16 and 8 systems share a CTA and past them, and
# numbers of systems that leave lanes empty.  Same bits as the same systems
# solved one thread each (an off-boundary array), 1e-13 to the oracle as test_zz_no_alloc.
@pytest.mark.parametrize("n", [(4, 1, 5), (6, 2, 3), (10, 16, 9), (30, 17, 8), (64, 33, 12),
                               (16, 109, 6), (16, 110, 6), (12, 212, 5), (12, 213, 5),
                               (8, 800, 4), (8, 900, 3)])
def test_spn_columns_match_oracle(n):
    import ctypes as C

    import torch
    nx, ny, nz = n
    AC, KXZ = O.mkp_coeffs(O.Grid(nx, ny, nz, 6.0, 2.0, 3.0, y0=-1.0, gamma=1.5))
    rng = np.random.default_rng(ny)
    Y = np.asfortranarray(rng.standard_normal((nx // 2 + 1, ny + 2, nz + 2)) +
                          1j * rng.standard_normal((nx // 2 + 1, ny + 2, nz + 2)))
    ref = Y.copy(order="F")
    O.spn(nx, ny, nz, AC, KXZ, ref)
    f = G.lib().nse_spn_noalloc
    f.argtypes = [C.c_int] * 3 + [C.c_void_p] * 4
    dev = [torch.from_numpy(a.ravel(order="F")).cuda() for a in (AC, KXZ)]
    got = []
    for off in (0, 1):
        raw = torch.zeros(2 * Y.size + 1, dtype=torch.float64, device="cuda")
        d = raw[off:off + 2 * Y.size]
        d.copy_(torch.from_numpy(Y.ravel(order="F").view(np.float64)))
        assert f(nx, ny, nz, dev[0].data_ptr(), dev[1].data_ptr(), d.data_ptr(),
                 torch.cuda.current_stream().cuda_stream) == 0
        got.append(d.cpu().numpy().view(np.complex128).reshape(Y.shape, order="F"))
    assert np.array_equal(got[0], got[1])
    assert rel_l2(got[0], ref) < 1e-13
    assert np.array_equal(got[0][:, [0, ny + 1]], Y[:, [0, ny + 1]])


# The adjoint on recorded steps in place (the lean form) against the one that copies
# (everything on one stream): grids with remainders of the 32 x 4 blocks, segments
# of one, some and all steps, a weight on a field behind the upper wall's row.
# Both are held to 1e-8 of the numpy adjoint (test_gpu_adjoint); to each other, a tenth.
@pytest.mark.parametrize("n,every", [((50, 15, 20), 1), ((64, 13, 18), 4), ((90, 14, 25), 9),
                                     ((33 * 2 - 2, 20, 12), 2)])
def test_adjoint_in_place_matches_copied(n, every):
    g, f, c1, par = make_case(*n, seed=8)
    out = []
    fields = ("u", "v", "w", "T", "u_ta", "v_ta", "w_ta", "u_pre", "v_pre", "w_pre", "T_pre")
    for flags in (0, S.FLAG_ONE_STREAM):
        cfg = S.Config(*n, par["dt"], par["Re"], par["Sc"], 50.0, g["xl"], g["yl"], g["zl"],
                       y0=-1.0, ystretch=2.0, body_force=par["force"], t_bot=1.0,
                       t_solid=par["tsolid"], flags=flags)
        with S.Context(cfg) as ctx:
            for k in ("u", "v", "w", "T"):
                ctx.upload(k, f[k])
            ctx.upload("cellvalue", c1)
            ctx.project()
            ctx.start()
            ctx.step(2)
            with S.Adjoint(ctx, 9, checkpoint_every=every, avg_from=5) as adj:
                rng = np.random.default_rng(3)
                for k in ("v", "u_ta", "T_pre"):
                    adj.set_weight(k, rng.standard_normal(ctx.shape))
                J, grad = adj.gradient()
                init = [adj.initial_adjoint(k)[1:-1, 1:-1, 1:-1]
                        for k in ("u", "v", "w", "T", "u_ta", "w_pre", "T_pre")]
            out.append([np.array(J), grad] + init + [ctx.download(k) for k in fields])
            if not flags:  # the context is left at the state after the steps
                got = [ctx.download(k) for k in STATE]
                for k in ("u", "v", "w", "T"):
                    ctx.upload(k, f[k])
                ctx.project()
                ctx.step_index = 1
                ctx.start()
                ctx.step(2)
                ctx.step(9)
                for k, a in zip(STATE, got):
                    assert np.array_equal(a, ctx.download(k)), k
    for k, (a, b) in enumerate(zip(*out)):
        assert np.linalg.norm(b) > 0
        assert rel_l2(a, b) < 1e-9, k


# The explicit terms with the tuned number of z planes per CTA (2 to 16), bit for
# bit those of 16: every cell is computed alone.  nz below, at and past multiples.
@pytest.mark.parametrize("prec,n", [(S.FP64, (36, 9, 5)), (S.FP64, (50, 15, 20)),
                                    (S.FP64, (64, 62, 64)), (S.FP64, (90, 14, 25)),
                                    (S.MIXED, (64, 24, 18)), (S.MIXED, (96, 17, 15))])
def test_explicit_terms_with_tuned_planes(prec, n):
    g, f, _, par = make_case(*n, seed=5)
    out = []
    for flags in (S.FLAG_NO_AUTOTUNE, 0):
        cfg = S.Config(*n, par["dt"], par["Re"], par["Sc"], 50.0, g["xl"], g["yl"], g["zl"],
                       y0=-1.0, ystretch=2.0, body_force=par["force"], t_bot=par["tbot"],
                       t_solid=par["tsolid"], precision=prec, flags=flags)
        with S.Context(cfg) as ctx:
            for k in ("u", "v", "w", "T"):
                ctx.upload(k, f[k])
            ctx.start()
            ctx.step(1)
            out.append([ctx.download(k) for k in ("u_pre", "v_pre", "w_pre", "T_pre")])
    for a, b in zip(*out):
        assert a.any() and np.array_equal(a, b)


# Transforms of two register stages: every radix in either place, odd counts of
# rows and columns off the tiles of 8, and lengths of three stages (250, 216).
# Tolerance: that of the other transforms (test_gpu_dropin).
@pytest.mark.parametrize("n", [(4, 1, 9), (6, 2, 10), (12, 3, 15), (20, 2, 25), (36, 3, 40),
                               (45, 2, 54), (64, 3, 72), (80, 2, 81), (90, 3, 100),
                               (96, 2, 108), (120, 2, 120), (128, 2, 135), (144, 2, 150),
                               (160, 3, 160), (180, 1, 192), (192, 2, 225), (240, 2, 240),
                               (250, 2, 216)])
def test_transforms_of_two_stages(n):
    nx, ny, nz = n
    FP = rand_field(np.random.default_rng(nx), nx, ny, nz)
    F1 = np.full((nx // 2 + 1, ny + 2, nz + 2), 7.0 + 3.0j, order="F")
    F2 = F1.copy(order="F")
    O.p2s(FP, nx, ny, nz, F1)
    G.p2s(FP, F2, nx, ny, nz)
    sl = (slice(None), slice(1, ny + 1), slice(0, nz))
    assert rel_l2(F2[sl], F1[sl]) < 1e-14
    F2[sl] = F1[sl]
    assert np.array_equal(F1, F2)  # nothing else written
    P1 = O.field(nx, ny, nz, -9.0)
    P2 = P1.copy(order="F")
    O.s2p(F1, nx, ny, nz, P1)
    G.s2p(F1, P2, nx, ny, nz)
    box = (slice(0, nx + 1), slice(1, ny + 1), slice(0, nz + 1))
    assert rel_l2(P2[box], P1[box]) < 1e-14
    P2[box] = P1[box]
    assert np.array_equal(P1, P2)


# The forward transform's division by NX NZ, a reciprocal with a correction, gives
# the bits of the division: an impulse at the origin has the one value everywhere.
@pytest.mark.parametrize("nx,nz", [(20, 25), (81, 9), (90, 100), (225, 240), (96, 256),
                                   (64, 128)])
def test_transform_divides_exactly(nx, nz):
    v = np.random.default_rng(nx + nz).standard_normal(400) * 10.0 ** np.arange(-200, 200)
    v[:8] = [0.0, -0.0, 5e-324, -1e-310, 3e-290, 1e290, -8e307, 2.2250738585072014e-308]
    FP = np.zeros((nx + 2, v.size + 2, nz + 2), order="F")
    FP[0, 1:-1, 0] = v
    F = np.zeros((nx // 2 + 1, v.size + 2, nz + 2), complex, order="F")
    G.p2s(FP, F, nx, v.size, nz)
    want = np.broadcast_to((v / (nx * nz))[None, :, None], (nx // 2 + 1, v.size, nz))
    assert np.array_equal(F[:, 1:-1, :nz].real, want)


# SPN on tiles: every remainder of the rows its sweeps and the mean mode's march run
# ahead (from the least number of rows that split, 4), against the form that loads
# each row as it needs it: same bits.  Tiles of 12 columns, whole and partial.
@pytest.mark.parametrize("ny", [4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 17, 18, 19, 20, 27, 256])
def test_spn_tiles_of_any_height(ny):
    nx, nz = (45, 5) if ny % 2 else (64, 6)
    rhs = rand_field(np.random.default_rng(ny), nx, ny, nz)
    out = []
    for form in (0, S.FLAG_SPN_CPASYNC):
        cfg = S.Config(nx, ny, nz, 1.0, 1.0, 1.0, 0.0, 2.0, 2.0, 3.0, y0=-1.0, ystretch=2.0,
                       flags=S.FLAG_NO_AUTOTUNE | form)
        with S.Context(cfg) as ctx:
            ctx.upload("phi", rhs)
            ctx.poisson()
            out.append(ctx.download("phi"))
    assert out[0].any() and np.array_equal(out[0], out[1])


# The adjoint's recorded steps start from device memory that held something else
# before and must not read a cell that no one wrote.  Blocks below 1 MB share the
# driver's 2 MB chunks, so holes between live blocks of NaN are what the adjoint's
# fields get.  Same bits as with a checkpoint before every step, whose start state
# is a copy of the context's fields.
@pytest.mark.parametrize("n,every", [((12, 13, 12), 2), ((12, 13, 12), 4), ((16, 14, 15), 3)])
def test_adjoint_on_recycled_memory(n, every):
    import ctypes as C

    import torch
    cu = C.CDLL("libcuda.so.1")
    g, f, c1, par = make_case(*n, seed=8)
    out = []
    for k in (1, every):
        cfg = S.Config(*n, par["dt"], par["Re"], par["Sc"], 50.0, g["xl"], g["yl"], g["zl"],
                       y0=-1.0, ystretch=2.0, body_force=par["force"], t_bot=1.0,
                       t_solid=par["tsolid"])
        with S.Context(cfg) as ctx:
            for name in ("u", "v", "w", "T"):
                ctx.upload(name, f[name])
            ctx.upload("cellvalue", c1)
            ctx.project()
            ctx.start()
            ctx.step(2)
            ctx.sync()
            torch.cuda.synchronize()
            blocks = []
            for fields in (4, 7 * k, 10, 11, 16 * k):
                for _ in range(16):
                    p, size = C.c_uint64(), C.c_size_t(fields * f["u"].nbytes)
                    assert cu.cuMemAlloc_v2(C.byref(p), size) == 0
                    blocks.append(p)
                    assert cu.cuMemsetD8_v2(p, C.c_ubyte(255), size) == 0
            torch.cuda.synchronize()
            for p in blocks[::2]:
                assert cu.cuMemFree_v2(p) == 0
            with S.Adjoint(ctx, 9, checkpoint_every=k, avg_from=5) as adj:
                adj.set_weight("v", f["w"])
                J, grad = adj.gradient()
                out.append([np.array(J), grad] + [adj.initial_adjoint(q)[1:-1, 1:-1, 1:-1]
                                                  for q in ("u", "v", "w", "T", "u_ta", "w_pre")])
            for p in blocks[1::2]:
                assert cu.cuMemFree_v2(p) == 0
    for q, (a, b) in enumerate(zip(*out)):
        assert np.linalg.norm(a) > 0 and np.array_equal(a, b), q


# Transforms of two register stages are no further from the 80-bit ones than the
# radix-4/2/3/5 stages were on the same samples (the bounds are those stages' errors).
@pytest.mark.parametrize("n,forward,inverse", [(32, 1.930e-16, 1.854e-16), (64, 2.147e-16, 2.051e-16),
                                               (72, 2.540e-16, 2.490e-16), (96, 2.427e-16, 2.393e-16),
                                               (128, 2.372e-16, 2.310e-16)])
def test_transform_error_against_80_bits(n, forward, inverse):
    ny, h = max(8, 200000 // n ** 2), n // 2 + 1
    FP = rand_field(np.random.default_rng(1001 * n), n, ny, n)
    F = np.zeros((h, ny + 2, n + 2), complex, order="F")
    G.p2s(FP, F, n, ny, n)
    S1 = F[:, 1:-1, :n].astype(np.clongdouble)
    want = np.fft.fft2(FP[:n, 1:-1, :n].astype(np.longdouble), axes=(0, 2))[:h] / n ** 2
    assert np.linalg.norm(abs(S1 - want)) <= forward * np.linalg.norm(abs(want))
    full = np.empty((n, ny, n), np.clongdouble)
    full[:h] = S1
    for i in range(h, n):
        full[i] = np.conj(np.roll(S1[n - i][:, ::-1], 1, axis=-1))
    want = np.fft.ifft2(full, axes=(0, 2)).real * n ** 2
    P = O.field(n, ny, n)
    G.s2p(F, P, n, ny, n)
    assert np.linalg.norm(P[:n, 1:-1, :n] - want) <= inverse * np.linalg.norm(want)


# Graphs of steps are made where they are used often: a call of 5 steps makes those of
# the steps in between, and a call of 20 or 21 after it none; the ones that begin
# and end a call come with its third use, a mask change starts over.
@pytest.mark.parametrize("prec", [S.FP64, S.MIXED])
@pytest.mark.parametrize("steps", [20, 21])
def test_long_call_after_a_short_one_makes_no_graph(prec, steps):
    g, f, c1, par = make_case(64, 24, 18, seed=4)
    cfg = S.Config(64, 24, 18, par["dt"], par["Re"], par["Sc"], par["eta"], g["xl"], g["yl"],
                   g["zl"], y0=-1.0, ystretch=2.0, precision=prec)
    with S.Context(cfg) as ctx:
        for k in ("u", "v", "w", "T"):
            ctx.upload(k, f[k])
        ctx.upload("cellvalue", c1)
        ctx.project()
        ctx.start()
        made = []
        for m in [5] + [steps] * 9:
            n0 = S.graph_count()
            ctx.step(m)
            made.append(S.graph_count() - n0)
        assert made[0] == (2 if prec == S.FP64 else 1) and made[1] == 0 and made[-1] == 0, made
        assert sum(made[2:]) > 0
        ctx.upload("cellvalue", np.asfortranarray(1.0 * (c1 > 0.5)))
        n0, r0 = S.graph_count(), S.graph_count(True)
        ctx.step(steps)
        assert S.graph_count() - n0 == made[0]
        assert S.graph_count(True) - r0 == steps - 3


# SPN by pipelined columns at the edges of its chunks of 8 rows: one row less, whole
# chunks, one and two rows more.
@pytest.mark.parametrize("ny", [7, 8, 9, 10, 15, 23, 24, 25, 26])
def test_spn_columns_at_chunk_edges(ny):
    test_spn_columns_match_oracle((10, ny, 9))


# The explicit terms, full and lean form, with every number of z planes per CTA that the
# tuning tries, and one and five, in every launch shape, bit for bit those of 16 planes in
# the first: whole and partial tiles, nz below, at and past multiples, an obstacle.
@pytest.mark.parametrize("prec,n", [(S.FP64, (64, 17, 45)), (S.FP64, (50, 15, 20)),
                                    (S.MIXED, (96, 17, 15))])
def test_explicit_terms_with_each_plane_count(prec, n):
    g, f, c1, par = make_case(*n, seed=6)
    ref = None
    for shape in range(7):
        for planes in (16, 12, 8, 5, 4, 2, 1):
            cfg = S.Config(*n, par["dt"], par["Re"], par["Sc"], 50.0, g["xl"], g["yl"], g["zl"],
                           y0=-1.0, ystretch=2.0, body_force=par["force"], t_bot=par["tbot"],
                           t_solid=par["tsolid"], precision=prec, flags=S.FLAG_NO_AUTOTUNE)
            with S.Context(cfg) as ctx:
                ctx.set_shapes(rhs=shape, correct=0)
                ctx.set_rhs_planes(planes)
                for k in ("u", "v", "w", "T"):
                    ctx.upload(k, f[k])
                ctx.upload("cellvalue", c1)
                ctx.start()
                ctx.step(1)
                ctx.step(4)  # two lean steps and two full ones
                got = [ctx.download(k) for k in STATE]
            ref = ref or got
            for k, a, b in zip(STATE, ref, got):
                assert np.isfinite(a).all() and np.array_equal(a, b), (k, shape, planes)


def test_plane_counts_out_of_range_are_refused():
    from vtkmakecompare_b200 import NseError
    g, _, _, par = make_case(36, 9, 10, seed=6)
    cfg = S.Config(36, 9, 10, par["dt"], par["Re"], par["Sc"], 50.0, g["xl"], g["yl"], g["zl"])
    with S.Context(cfg) as ctx:
        with pytest.raises(NseError):
            ctx.set_rhs_planes(8)  # no shape fixed yet
        ctx.set_shapes(rhs=1)
        for planes in (0, 17, -1):
            with pytest.raises(NseError):
                ctx.set_rhs_planes(planes)
        ctx.set_rhs_planes(16)


# Level-set sweeps that march 4 and 8 cells a thread (from 600k and 2.5M cells), and 2
# and 4 in replayed graphs, with nz off their multiples.
@pytest.mark.parametrize("n,nnn", [((90, 60, 75), 130), ((96, 80, 81), 3), ((96, 80, 81), 129),
                                   ((160, 128, 125), 3), ((150, 135, 135), 2)])
def test_levelset_marches_match_oracle_bit_for_bit(n, nnn):
    test_levelset_sweeps_match_oracle_bit_for_bit(n, nnn, 0)


# Rounding of x lines of any length: one step of heat conduction along x alone (no flow,
# cells 1e11 wide in y and z), so T is (I - b D)^-1 (I + b D) T0 with b D of order 0.1,
# against long doubles.  Of T's roundings the right-hand side makes three and a solve that
# adds its corrections up before it adds them to T one, sqrt(4 / 12) = 0.58 units in
# the last place in the mean square; one that rounds T in every operation has 5 to 13
# more a row, 0.9 units and above.  Bound: half way.
@pytest.mark.parametrize("nx", [20, 36, 50, 75, 90, 100, 125, 150, 225, 270, 405, 500])
def test_x_lines_of_any_length_round_once(nx):
    ny, nz = 13, 12
    cfg = S.Config(nx, ny, nz, 0.2, 1.0, 1.0, 1.0, float(nx), 1e11 * ny, 1e11 * nz,
                   body_force=0.0, heat_source=0.0)
    rng = np.random.default_rng(nx)
    T = np.asfortranarray(1.0 + rng.random((nx + 2, ny + 2, nz + 2)))
    with S.Context(cfg) as ctx:
        ctx.upload("T", T)
        ctx.start()
        ctx.step(1)
        got = ctx.download("T")[1:-1, 1:-1, 1:-1]
    T0 = T[1:-1, 1:-1, 1:-1].reshape(nx, -1).astype(np.longdouble)
    D = lambda x: np.roll(x, 1, 0) - 2 * x + np.roll(x, -1, 0)
    b = np.longdouble(0.2) / 2
    r = T0 + b * D(T0)
    M = np.eye(nx) - float(b) * D(np.eye(nx))
    x = np.zeros_like(r)
    for _ in range(4):
        x += np.linalg.solve(M, (r - (x - b * D(x))).astype(float))
    err = (got.reshape(nx, -1) - x).astype(float) / 2.0 ** -52
    assert np.sqrt(np.mean(err ** 2)) < 0.75, np.sqrt(np.mean(err ** 2))
