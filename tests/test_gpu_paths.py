"""Edges of the GPU kernels behind the solvers, the network's training and the layout
conversion: column counts of the three-pass orthonormalisation, blocks of right-hand
sides that share reliable updates, 16-bit iterations, pairs beyond one group of the
network's layers, the operator on reference-layout arrays, device arrays that are not
16-byte aligned, and a device without room."""
import numpy as np
import pytest

import oracle
from qqtest import golden_gauge, random_half

pytestmark = pytest.mark.gpu

DIMS, BC = (4, 4, 4, 8), (1, 1, 1, -1)
KAPPA = (0.130, 0.01)


@pytest.fixture(scope="module")
def pair():
    import baylorlqcd_b200 as qq

    ol = oracle.OracleLattice(*DIMS, bc=BC)
    _, u = golden_gauge(DIMS, ol.ntotal, seed=41, eps=0.3)
    ol.set_gauge(u)
    lat = qq.Lattice(*DIMS, bc=BC)
    lat.gauge_upload(u, recon=18)
    yield ol, lat
    lat.close()


def interior_rel(a, b, nv):
    return np.linalg.norm((a - b)[..., :nv, :]) / np.linalg.norm(b[..., :nv, :])


@pytest.mark.parametrize("m,k", [(2, 1), (9, 3), (17, 6), (66, 20), (127, 40)])
def test_gmresdr_column_counts(pair, m, k):
    """Every column count up to m is orthonormalised, so the sizes cross the kernel's
    splits at 8, 16, 32 and 64 vectors (lanes in one to eight groups, eight or sixteen
    columns a lane) and reach the largest.  Both solve to 1e-11, and the operator's
    condition at this kappa is below 1e2: solutions agree to 1e-8."""
    ol, lat = pair
    be, bo = random_half(ol.ntotal, ol.nvhalf, 5), random_half(ol.ntotal, ol.nvhalf, 6)
    xe, xo, info = lat.fermprop(be, bo, KAPPA, inverter=5, resmax=1e-11, nGMRES=(m, k))
    we, wo, st, _ = ol.fermprop(be, bo, KAPPA, inverter=5, resmax=1e-11, nGMRES=(30, 10))
    assert info.status == 0 and st == 0
    assert interior_rel(xe, we, ol.nvhalf) < 1e-8 and interior_rel(xo, wo, ol.nvhalf) < 1e-8


def gram_error(lat, defl):
    """max |V^H V - 1| of a deflation space's vectors."""
    import torch

    v = torch.stack([torch.from_numpy(defl.vector(j)[..., : lat.nvhalf, :]).cuda().flatten() for j in range(defl.k + 1)])
    v = torch.complex(v[:, 0::2], v[:, 1::2])
    return (v.conj() @ v.T - torch.eye(defl.k + 1, device="cuda")).abs().max().item()


@pytest.mark.parametrize("m,k", [(9, 4), (17, 12), (33, 28), (66, 60), (127, 60)])
def test_restarted_basis_is_orthonormal(m, k):
    """A restart's vectors are combinations of the whole basis with orthonormal
    coefficients, so their Gram matrix shows the basis's: classical Gram-Schmidt done
    twice leaves rounding, m products of length 24576 (below 1e-13 with m <= 127)."""
    import baylorlqcd_b200 as qq

    lat = qq.Lattice(8, 8, 8, 8, bc=BC)
    lat.heatbath(6.0, 30, seed=4)
    b, kappa = random_half(lat.ntotal, lat.nvhalf, 12), (0.156, 0.0)
    defl = lat.deflation(m, k)
    x, info = lat.gmresdr(b, lat.new_half(), (m, k), 1e-10, kappa=kappa, defl=defl)
    assert info.status == 0 and info.ncycles > 1 and defl.k == k
    r = (b - lat.hdbletm(x, 0, kappa))[..., : lat.nvhalf, :]
    err = gram_error(lat, defl)
    defl.close()
    lat.close()
    assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(b) and err < 1e-13


@pytest.mark.parametrize("nt", [32, 48])
def test_large_bases(nt):
    """65,536 and 98,304 sites of a parity: past 2^19 elements a vector (both in FP64, the
    second in FP32 too), where the first products of 32 and more vectors are another
    kernel's.  Each solve is judged by its FP64 residual through the operator."""
    import baylorlqcd_b200 as qq

    lat = qq.Lattice(16, 16, 16, nt, bc=BC)
    lat.heatbath(6.0, 20, seed=6)
    b, kappa = random_half(lat.ntotal, lat.nvhalf, 13), (0.150, 0.01)
    defl = lat.deflation(66, 30)
    x, info = lat.gmresdr(b, lat.new_half(), (66, 30), 1e-10, kappa=kappa, defl=defl)
    assert info.status == 0 and info.ncycles > 1 and gram_error(lat, defl) < 1e-13
    r = (b - lat.hdbletm(x, 0, kappa))[..., : lat.nvhalf, :]
    assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(b)
    defl.close()
    half = np.stack([b, random_half(lat.ntotal, lat.nvhalf, 14)])
    _, _, infos = lat.fermprop_batch(half, half[::-1].copy(), kappa, tol=1e-10)  # FP32 basis, m = 60
    lat.close()
    assert all(i.status == 0 and i.true_rel <= 1e-10 and i.finished_by == 0 for i in infos)


@pytest.mark.parametrize("m,k", [(9, 3), (17, 6), (40, 12), (60, 20), (100, 40), (127, 40)])
def test_deflated_batch_column_counts(pair, m, k):
    """The FP32 basis behind a deflated batch, on both sides of the same splits; 60 and 20
    are the call's defaults.  Solutions agree with the oracle's as those of the FP64
    basis do."""
    ol, lat = pair
    be = np.stack([random_half(ol.ntotal, ol.nvhalf, 20 + i) for i in range(2)])
    bo = np.stack([random_half(ol.ntotal, ol.nvhalf, 25 + i) for i in range(2)])
    xe, xo, infos = lat.fermprop_batch(be, bo, KAPPA, m=m, k=k, tol=1e-10)
    for i in range(2):
        assert infos[i].status == 0 and infos[i].true_rel <= 1e-10 and infos[i].finished_by == 0
        we, wo, st, _ = ol.fermprop(be[i], bo[i], KAPPA, inverter=5, resmax=1e-12, nGMRES=(30, 10))
        assert interior_rel(xe[i], we, ol.nvhalf) < 1e-8 and interior_rel(xo[i], wo, ol.nvhalf) < 1e-8


@pytest.mark.parametrize("m", [40, 100])
def test_gmresdr_past_the_krylov_degree(m):
    """On a unit gauge field the operator has few distinct eigenvalues, so the basis is
    complete well before m and the rest of the cycle orthogonalises rounding noise: the
    corrections are as large as the vectors, and the norm is summed directly.  The solve
    converges in its first cycle with a residual far below its tolerance's 1e-10."""
    import baylorlqcd_b200 as qq

    lat = qq.Lattice(4, 4, 4, 8, bc=(1, 1, 1, 1))
    u = np.zeros(lat.gauge_shape)
    u[:, :, :, : lat.nvhalf, [0, 8, 16]] = 1.0
    lat.gauge_upload(u)
    b = random_half(lat.ntotal, lat.nvhalf, 9)
    x, info = lat.gmresdr(b, lat.new_half(), (m, 8), 1e-10, kappa=(0.11, 0.02))
    r = b - lat.hdbletm(x, 0, (0.11, 0.02))
    lat.close()
    assert info.status == 0 and info.ncycles == 1
    assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("nrhs,block,precision", [(1, 1, 32), (5, 3, 32), (33, 32, 32), (5, 8, 16), (3, 2, 64)])
def test_batch_blocks_share_updates(pair, nrhs, block, precision):
    """Every right-hand side of every block, with the last block short: converged by the
    batched iteration (16 bits may be finished by FP32) and equal to the oracle's solution
    to the tolerance times the operator's condition."""
    ol, lat = pair
    be = np.stack([random_half(ol.ntotal, ol.nvhalf, 50 + i) for i in range(nrhs)])
    bo = np.stack([random_half(ol.ntotal, ol.nvhalf, 150 + i) for i in range(nrhs)])
    xe, xo, infos = lat.fermprop_batch(be, bo, KAPPA, precision=precision, rhs_block=block, tol=1e-10, deflate=0)
    for i in range(nrhs):
        assert infos[i].status == 0 and infos[i].true_rel <= 1e-10 and infos[i].finished_by in (0, 32)
    for i in {0, nrhs - 1}:
        we, wo, st, _ = ol.fermprop(be[i], bo[i], KAPPA, inverter=5, resmax=1e-12, nGMRES=(30, 10))
        assert interior_rel(xe[i], we, ol.nvhalf) < 1e-8 and interior_rel(xo[i], wo, ol.nvhalf) < 1e-8


@pytest.mark.parametrize("precision", [16, -16])
@pytest.mark.parametrize("nrhs", [1, 5])
def test_easy_16bit_solves_need_no_other_precision(pair, precision, nrhs):
    """Far from critical kappa the 16-bit iteration converges by itself, so long as the
    products that a reliable update resumes from are those of the residual it stored: no
    hand-over to FP32, no restart."""
    ol, lat = pair
    be = np.stack([random_half(ol.ntotal, ol.nvhalf, 250 + i) for i in range(nrhs)])
    bo = np.stack([random_half(ol.ntotal, ol.nvhalf, 350 + i) for i in range(nrhs)])
    _, _, infos = lat.fermprop_batch(be, bo, (0.08, 0.0), precision=precision, tol=1e-10, deflate=0)
    for i in infos:
        assert i.status == 0 and i.true_rel <= 1e-10 and i.finished_by == 0 and i.restarts == 0


def test_launch_counter_of_the_graph_loop(pair):
    """The counter knows how often the loop's two bodies ran.  Two equal right-hand sides
    at several tolerances give the launches of a call, an iteration and an update (three
    unknowns, five calls); two unlike ones then launch an update for every iteration after
    which either was updated."""
    import baylorlqcd_b200 as qq

    ol, lat = pair
    noise = random_half(ol.ntotal, ol.nvhalf, 31), random_half(ol.ntotal, ol.nvhalf, 32)
    point = lat.pointsource((1, 1, 1, 1), 1, 1)

    def run(a, b, tol):
        be, bo = np.stack([a[0], b[0]]), np.stack([a[1], b[1]])
        n0 = qq.launch_count()
        _, _, infos = lat.fermprop_batch(be, bo, KAPPA, precision=32, tol=tol, deflate=0)
        n = qq.launch_count() - n0
        its = [set((i.hist_mvp - np.arange(len(i.hist_mvp)) - 2) // 2) for i in infos]  # at each update
        return n, max(i.itercount for i in infos), len(its[0] | its[1]), max(map(len, its))

    run(noise, point, 1e-4)  # tunes the hops
    same = [run(noise, noise, 10.0 ** -k) for k in (2, 4, 6, 8, 10)]
    fit = np.array([(1, it, upd) for _, it, upd, _ in same], float)
    per = np.linalg.lstsq(fit, np.array([n for n, *_ in same], float), rcond=None)[0]
    assert np.abs(per - np.rint(per)).max() < 1e-6 and np.array_equal(fit @ np.rint(per), [n for n, *_ in same])
    n, it, upd, most = run(noise, point, 1e-10)
    assert upd > most and n == np.rint(per) @ (1, it, upd)


@pytest.mark.parametrize("precision,tol", [(16, 2e-3), (-16, 1.5e-2)])
@pytest.mark.parametrize("nrhs", [1, 3, 5, 12, 24, 32])
@pytest.mark.parametrize("shape", [307, 308])
def test_copy_ring_16bit(pair, shape, nrhs, precision, tol):
    """The 16-bit copy ring against the oracle's FP64 Hsingle, with the tolerances of the
    other 16-bit shapes (11 and 8 significant bits against a site's norm); 5 right-hand
    sides leave the last block partly empty.  128 sites of a parity."""
    ol, lat = pair
    gin = np.stack([random_half(ol.ntotal, ol.nvhalf, 500 + i) for i in range(nrhs)])
    for idag, gblclr in ((0, 1), (1, 2)):
        out = lat.hsingle_block(gin, idag, gblclr, precision=precision, shape=shape)
        for k in {0, nrhs - 1}:
            ref = ol.hsingle(gin[k], idag, gblclr)[..., : ol.nvhalf, :]
            assert np.abs(out[k][..., : ol.nvhalf, :] - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize("recon", [12, 18])
@pytest.mark.parametrize("shape", [1, 2, 4, 5, 6, 64])
def test_fp64_single(monkeypatch, shape, recon):
    """The shapes of one FP64 right-hand side, 1280 sites of a parity.  An output
    component sums 8 hops of 3 products of normal deviates: 1e-13 is 450 rounding errors
    of the largest."""
    import baylorlqcd_b200 as qq

    dims = (4, 8, 4, 20)
    ol = oracle.OracleLattice(*dims, bc=BC)
    _, u = golden_gauge(dims, ol.ntotal, seed=43, eps=0.3)
    ol.set_gauge(u)
    monkeypatch.setenv("QQ_FORCE_TPS", str(shape))
    lat = qq.Lattice(*dims, bc=BC)
    lat.gauge_upload(u, recon=recon)
    gin = random_half(ol.ntotal, ol.nvhalf, 600)
    for idag, gblclr in ((0, 1), (1, 2)):
        out = lat.hsingle(gin, idag, gblclr)[..., : ol.nvhalf, :]
        ref = ol.hsingle(gin, idag, gblclr)[..., : ol.nvhalf, :]
        assert np.abs(out - ref).max() < 1e-13 * np.abs(ref).max()
    lat.close()


@pytest.mark.parametrize("recon", [12, 18])
@pytest.mark.parametrize("shape", [5, 6, 96])
def test_fp64_blocks(monkeypatch, shape, recon):
    """The FP64 shapes offered to blocks only by the autotuner's choice, forced on three
    right-hand sides (42 sites a block of 128 threads, the last one partly empty).  The
    residual that the solve is judged by is another kernel's."""
    import baylorlqcd_b200 as qq

    dims = (4, 8, 4, 20)
    ol = oracle.OracleLattice(*dims, bc=BC)
    _, u = golden_gauge(dims, ol.ntotal, seed=43, eps=0.3)
    monkeypatch.setenv("QQ_FORCE_TPS", str(shape))
    lat = qq.Lattice(*dims, bc=BC)
    lat.gauge_upload(u, recon=recon)
    be = np.stack([random_half(ol.ntotal, ol.nvhalf, 610 + i) for i in range(3)])
    bo = np.stack([random_half(ol.ntotal, ol.nvhalf, 620 + i) for i in range(3)])
    _, _, infos = lat.fermprop_batch(be, bo, KAPPA, precision=64, tol=1e-12, deflate=0)
    lat.close()
    for i in infos:
        assert i.status == 0 and i.true_rel <= 1e-12 and i.finished_by == 0 and i.restarts == 0


@pytest.mark.parametrize("channels", [(4, 4), (4, 8, 16, 4), (4, 16, 16, 4)])
def test_gradient_of_more_pairs_than_a_group(pair, channels):
    """Pairs go through the layers in groups of at most eight.  The loss and the gradient
    of nine are the means of the single ones: the FP32 fields are the same but for the
    residual's scale 1/9 (a relative 2^-24 per element), and the sums are FP64."""
    import baylorlqcd_b200 as qq

    ol, lat = pair
    net = qq.Net(channels, seed=3)
    b = np.stack([random_half(ol.ntotal, ol.nvhalf, 300 + i) for i in range(9)])
    x = np.stack([random_half(ol.ntotal, ol.nvhalf, 400 + i) for i in range(9)])
    loss, grad = net.loss_grad(lat, b, x)
    one = [net.loss_grad(lat, b[i:i + 1], x[i:i + 1]) for i in range(9)]
    net.close()
    want = np.mean([g for _, g in one], axis=0)
    assert abs(loss - np.mean([v for v, _ in one])) <= 1e-12 * abs(loss)
    assert np.abs(grad - want).max() <= 1e-6 * np.abs(want).max()


@pytest.mark.parametrize("dims", [(8, 8, 8, 32), (8, 8, 12, 28)])
@pytest.mark.parametrize("channels", [(4, 4), (4, 16, 8, 4)])
def test_layers_on_both_sides_of_the_split(dims, channels):
    """16384 and 21504 sites: a thread per colour and a thread per site.  FP32 against
    numpy's FP64 with the bound of the small lattices: a site's sums are as long there."""
    import baylorlqcd_b200 as qq
    import netref
    from qqtest import half_to_lex, random_gauge

    ol = oracle.OracleLattice(*dims, bc=BC)
    links, u = random_gauge(dims, ol.ntotal, seed=4)
    net = qq.Net(channels, seed=2)
    g = random_half(ol.ntotal, ol.nvhalf, seed=7)
    lat = qq.Lattice(*dims, bc=BC)
    lat.gauge_upload(u, recon=18)
    out = net.apply(lat, g)
    lat.close()
    w, ch, ws = net.get_weights(), net.channels, []
    for i in range(len(ch) - 1):
        n = 9 * ch[i + 1] * ch[i]
        ws.append(w[:n].reshape(9, ch[i + 1], ch[i]))
        w = w[n:]
    net.close()
    ref = netref.apply(ws, links, half_to_lex(g, dims, 1), BC)
    assert np.abs(half_to_lex(out, dims, 1) - ref).max() < 2e-5 * np.abs(ref).max()


@pytest.mark.parametrize("dims,bc,recon", [((4, 4, 4, 8), (1, 1, 1, -1), 12), ((4, 4, 4, 8), (0, -1, 1, 0), 18),
                                           ((8, 8, 8, 12), (1, -1, 1, -1), 18), ((8, 8, 8, 16), (1, 1, 1, -1), 12),
                                           ((12, 20, 4, 28), (-1, 1, 0, 1), 18),
                                           ((16, 16, 8, 32), (1, 0, 1, -1), 18), ((16, 8, 16, 40), (1, 1, 1, -1), 12),
                                           ((24, 24, 24, 24), (1, 1, 1, -1), 12), ((24, 24, 24, 24), (1, 1, 1, -1), 18)])
def test_operator_on_reference_arrays(dims, bc, recon):
    """Hsingle and Hdbletm read and write the reference layout directly: each number of
    threads per site its rule picks (256 and 3072 sites of a parity: four; 4096 and 13,440:
    two; 32,768 and more: one), both link storages, fixed and antiperiodic boundaries; FP64
    against the oracle at its other tests' 1e-13."""
    import baylorlqcd_b200 as qq

    ol = oracle.OracleLattice(*dims, bc=bc)
    _, u = golden_gauge(dims, ol.ntotal, seed=43, eps=0.6)
    ol.set_gauge(u)
    lat = qq.Lattice(*dims, bc=bc)
    lat.gauge_upload(u, recon=recon)
    g = random_half(ol.ntotal, ol.nvhalf, 8)
    for idag, gblclr in ((0, 1), (1, 2)):
        want = ol.hsingle(g, idag, gblclr)[..., : ol.nvhalf, :]
        got = lat.hsingle(g, idag, gblclr)
        assert np.abs(got[..., : ol.nvhalf, :] - want).max() <= 1e-13 * np.abs(want).max()
        assert not got[..., ol.nvhalf:, :].any()
    for kappa in ((0.15, 0.0), (0.15, 0.02)):
        want = ol.hdbletm(g, 0, kappa)[..., : ol.nvhalf, :]
        got = lat.hdbletm(g, 0, kappa)[..., : ol.nvhalf, :]
        assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
    same = g.copy()  # in place: through the GPU layout
    lat.hdbletm(same, 0, kappa, out=same)
    assert np.abs(same[..., : ol.nvhalf, :] - want).max() <= 1e-13 * np.abs(want).max()
    lat.close()


def test_unaligned_device_arrays(pair):
    """Reference-layout device arrays 8 bytes off a 16-byte boundary, in and out, take the
    path through the GPU layout; aligned ones are read and written directly.  The same
    values but for the order of the 24 products a component sums in each of the two hops:
    2 * 24 * 2^-53 of the sum of their magnitudes, itself below 20 times the largest
    component, is 1e-13 of that.  Halo slots are zeroed on both."""
    import torch

    ol, lat = pair
    g = random_half(ol.ntotal, ol.nvhalf, 7)
    want = lat.hdbletm(g, 0, KAPPA)
    n = g.size
    gin = torch.zeros(n + 1, dtype=torch.float64, device="cuda")
    out = torch.full((n + 1,), 3.0, dtype=torch.float64, device="cuda")
    gin[1:] = torch.from_numpy(g).cuda().flatten()
    torch.cuda.synchronize()
    lat.hdbletm(gin[1:], 0, KAPPA, out=out[1:])
    got = out[1:].cpu().numpy().reshape(g.shape)
    assert np.abs(got - want).max() <= 1e-13 * np.abs(want).max()
    assert not got[..., ol.nvhalf:, :].any() and not want[..., ol.nvhalf:, :].any()
    assert out[0].item() == 3.0


def test_a_full_device_is_an_error():
    """A call whose fields do not fit on the device reports it, and the next one, with the
    memory free again, gives the values of a fresh context (the order of a component's
    sums is the autotuner's choice: 1e-12 of the largest value)."""
    import torch

    import baylorlqcd_b200 as qq

    dims = (16, 16, 16, 32)  # the eight fields of the call take 100 MB

    def lattice():
        lat = qq.Lattice(*dims, bc=BC)
        lat.heatbath(6.0, 2, seed=3)
        return lat

    lat = lattice()
    v = [torch.from_numpy(random_half(lat.ntotal, lat.nvhalf, 70 + i)).cuda() for i in range(4)]
    want = lat.average(*v, 0.15, nsub=4, nmom=1, nop=9)
    lat.close()
    lat, held = lattice(), []
    while (free := torch.cuda.mem_get_info()[0] - (48 << 20)) > 0:
        held.append(torch.empty(min(free, 1 << 30), dtype=torch.uint8, device="cuda"))
    with pytest.raises(qq.QQError, match="memory"):
        lat.average(*v, 0.15, nsub=4, nmom=1, nop=9)
    held.clear()
    torch.cuda.empty_cache()
    got = lat.average(*v, 0.15, nsub=4, nmom=1, nop=9)
    lat.close()
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
