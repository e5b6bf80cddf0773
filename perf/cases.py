"""Performance cases: the work a user of this framework has it do, through its public calls.

A lattice-QCD program holds a lattice with a quenched SU(3) configuration on the GPU and
asks for Dirac-operator applications, propagators (batched mixed-precision, plain FP64
GMRES-DR, deflated GMRES-Proj on further right-hand sides), loop operators of a noise
vector, and training runs of the learned preconditioner.  Every array stays on the GPU in
the reference's layout; configurations come from the package's own heatbath at beta = 6.0,
kappas, masses, extents, GMRES(m, k) and RHS blocks from the repository's benchmark
configurations (8^4 to 24^3 x 48).

A case is a dict of plain values; ``kind`` says which call it makes:
  operator  one Hdbletm (Wilson for mu = 0, twisted otherwise)
  batch     Lattice.fermprop_batch: nrhs propagators to 1e-10, inner precision FP32 or
            16 bits (16 FP16, -16 BF16), FP64 true residual
  gmresdr   Lattice.fermprop with the FP64 GMRES-DR(m, k)
  gmresproj Lattice.gmresproj on a further right-hand side of the even-site system,
            deflated by the space a first GMRES-DR solve left
  train     a Net of the given width trained for some Adam steps on (source, solution)
            pairs: forward, backward and update
  average   the Wilson loop operators of one noise at subtraction levels 1..nsub
"""
import math

import numpy as np
import torch

import baylorlqcd_b200 as qq

BC = (1, 1, 1, -1)
TOL = 1e-10


def listed():
    return [
        # One application of the operator on the smallest lattice of the configurations:
        # the call a host code makes inside its own inverter.
        dict(name="operator 8^4", kind="operator", nx=8, ny=8, nz=8, nt=8, kappa=0.150, mu=0.0, idag=0),
        # The same on an odd-shaped lattice whose rows and slices are no multiple of a warp.
        dict(name="operator 12x20x4x28 dagger", kind="operator", nx=12, ny=20, nz=4, nt=28, kappa=0.155, mu=0.0,
             idag=1),
        # The same on the largest configuration, twisted mass.
        dict(name="operator 24^3x48 twisted", kind="operator", nx=24, ny=24, nz=24, nt=48, kappa=0.1566, mu=0.0025,
             idag=0),
        # The 12 spin-colour columns of a point propagator on a small lattice: latency.
        dict(name="batch 8^3x16", kind="batch", nx=8, ny=8, nz=8, nt=16, kappa=0.150, mu=0.0, nrhs=12, block=12,
             precision=32, source="point", iters=105),
        # The point propagator at 16^3x32, several hundred iterations.
        dict(name="batch 16^3x32", kind="batch", nx=16, ny=16, nz=16, nt=32, kappa=0.155, mu=0.0, nrhs=12, block=12,
             precision=32, source="point", iters=350),
        # Noise solves of a disconnected-loop run on the largest configuration, twisted mass.
        dict(name="batch 24^3x48 twisted", kind="batch", nx=24, ny=24, nz=24, nt=48, kappa=0.150, mu=0.0025, nrhs=12,
             block=12, precision=32, source="z4", iters=100),
        # A ragged batch (5 noises) in FP16 storage on the second lattice of the uneven batch.
        dict(name="batch 12^3x24 fp16", kind="batch", nx=12, ny=12, nz=12, nt=24, kappa=0.145, mu=0.0, nrhs=5, block=8,
             precision=16, source="z4", iters=150),
        # The plain method of the first configuration: point source, GMRES-DR(30, 10).
        dict(name="gmresdr 8^4", kind="gmresdr", nx=8, ny=8, nz=8, nt=8, kappa=0.150, mu=0.0, m=30, k=10, iters=140),
        # The plain method at 16^3x32 with the larger subspace.
        dict(name="gmresdr 16^3x32 twisted", kind="gmresdr", nx=16, ny=16, nz=16, nt=32, kappa=0.1566, mu=0.005, m=60,
             k=20, iters=1220),
        # A further right-hand side of the loop run, deflated by the first one's eigenvectors.
        dict(name="gmresproj 16^3x32 twisted", kind="gmresproj", nx=16, ny=16, nz=16, nt=32, kappa=0.1566, mu=0.005,
             m=60, k=30, iters=435),
        # A training run of the learned preconditioner: two pairs, twenty Adam steps.
        dict(name="train 8^3x16 4-8-8-4", kind="train", nx=8, ny=8, nz=8, nt=16, kappa=0.1566, mu=0.0025, width=8,
             pairs=2, steps=20),
        # The loop operators of one noise, all subtraction levels and momenta.
        dict(name="average 16^3x32", kind="average", nx=16, ny=16, nz=16, nt=32, kappa=0.155, mu=0.0, nsub=6, nmom=5),
    ]


def _extents(rng, low, high):
    """Four extents, each a multiple of 4, whose volume is spread over [low, high] in its logarithm."""
    want = math.exp(rng.uniform(math.log(low), math.log(high)))
    for _ in range(1000):
        n = [rng.choice((4, 8, 12, 16, 20, 24)) for _ in range(3)] + [rng.choice((8, 12, 16, 20, 24, 28, 32, 40, 48))]
        v = n[0] * n[1] * n[2] * n[3]
        if low <= v <= high and 0.7 < v / want < 1.4:
            return n
    return [8, 8, 8, 8]


def draw(rng):
    kind = rng.choice(("operator", "operator", "batch", "batch", "batch", "gmresdr", "gmresproj", "train", "average"))
    top = {"operator": 24 ** 3 * 48, "batch": 20 ** 3 * 40, "gmresdr": 16 ** 3 * 32, "gmresproj": 16 ** 3 * 32,
           "train": 16 ** 3 * 32, "average": 20 ** 3 * 40}[kind]
    n = _extents(rng, 2048 if kind == "operator" else 4096, top)
    c = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], nt=n[3])
    # solves stay below the kappas where a configuration can be exceptional
    mu = round(rng.uniform(0.0025, 0.02), 4) if rng.random() < 0.5 else 0.0
    kappa = rng.choice((0.150, 0.155, 0.1566) if kind == "operator" else (0.145, 0.148, 0.150))
    if kind == "operator":
        c.update(kappa=kappa, mu=mu, idag=rng.randrange(2))
    elif kind == "batch":
        prec = rng.choice((32, 32, 32, 16, -16))
        if prec != 32:  # 16-bit storage: well away from critical, where it converges by itself
            kappa = rng.choice((0.140, 0.145))
        c.update(kappa=kappa, mu=mu, nrhs=rng.choice((1, 2, 3, 5, 8, 11, 12, 12, 16, 24, 32)),
                 block=rng.choice((8, 12, 16, 32)), precision=prec, source=rng.choice(("point", "z4")), iters=100)
    elif kind in ("gmresdr", "gmresproj"):
        m = rng.choice((30, 40, 60))
        c.update(kappa=kappa, mu=mu, m=m, k=m // rng.choice((2, 3)),
                 iters=160)
    elif kind == "train":
        c.update(kappa=0.1566, mu=0.0025, width=rng.choice((4, 8, 8, 16)), pairs=rng.choice((1, 2, 3)),
                 steps=rng.choice((5, 10, 20)))
    else:
        c.update(kappa=rng.choice((0.150, 0.155)), mu=0.0, nsub=rng.choice((2, 4, 6)), nmom=rng.choice((1, 3, 5)))
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _dims(c):
    return c["nx"], c["ny"], c["nz"], c["nt"]


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 11)


def _lattice(c, seed):
    lat = qq.Lattice(*_dims(c), bc=BC)
    u = torch.zeros(lat.gauge_shape, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    lat.heatbath(6.0, 40, seed=int(seed) + 1, u_out=u)
    return lat, u


def _half(lat, n=None):
    return torch.zeros(lat.half_shape if n is None else (n,) + lat.half_shape, dtype=torch.float64, device="cuda")


def _gauss_half(lat, gen):
    h = _half(lat)
    h[:, :, :, : lat.nvhalf] = torch.randn(8, 2, 4, lat.nvhalf, 6, generator=gen, dtype=torch.float64, device="cuda")
    return h


def _z4_half(lat, gen):
    """Every complex entry uniform on {1, i, -1, -i}."""
    h = _half(lat)
    k = torch.randint(0, 4, (8, 2, 4, lat.nvhalf, 3), generator=gen, device="cuda")
    h[:, :, :, : lat.nvhalf, 0::2] = (k == 0).double() - (k == 2).double()
    h[:, :, :, : lat.nvhalf, 1::2] = (k == 1).double() - (k == 3).double()
    return h


def _sources(c, lat, gen, n, source):
    be, bo = _half(lat, n), _half(lat, n)
    if source == "z4":
        for i in range(n):
            be[i], bo[i] = _z4_half(lat, gen), _z4_half(lat, gen)
        return be, bo
    # point sources: the spin-colour columns of one site after another
    r = torch.randint(0, 1 << 30, (n, 2), generator=gen, device="cuda").cpu().numpy()
    for i in range(n):
        ieo, isite = int(r[i // 12, 0]) % 2, int(r[i // 12, 1]) % lat.nvhalf
        be[i, 0, ieo, (i // 3) % 4, isite, 2 * (i % 3)] = 1.0
    return be, bo


def _widths(c):
    return 4, c["width"], c["width"], 4


def _weights(c, gen):
    """Start weights: near the kappa^2 the operator's diagonal asks for, every other path small."""
    ch, out = _widths(c), []
    for ci, co in zip(ch, ch[1:]):
        w = 0.005 * torch.randn(9, co, ci, 2, generator=gen, dtype=torch.float64, device="cuda")
        w[0, range(4), range(4), 0] += c["kappa"] ** (2.0 / 3.0)
        out.append(torch.view_as_complex(w).flatten())
    return torch.cat(out).cpu().numpy()


def prepare(case, seed):
    c, gen = case, _generator(seed)
    lat, u = _lattice(c, seed)
    s = dict(case=dict(c), lat=lat, kappa=(c["kappa"], c["mu"]))
    kind = c["kind"]
    if kind == "operator":
        s.update(g=_gauss_half(lat, gen), h=_half(lat))
    elif kind in ("batch", "gmresdr"):
        n = c.get("nrhs", 1)
        be, bo = _sources(c, lat, gen, n, c.get("source", "point"))
        if kind == "gmresdr":
            be, bo = be[0].clone(), bo[0].clone()
        s.update(be=be, bo=bo, xe=torch.zeros_like(be), xo=torch.zeros_like(bo))
    elif kind == "gmresproj":
        first, b = _z4_half(lat, gen), _z4_half(lat, gen)
        defl = lat.deflation(c["m"], c["k"])
        x = _half(lat)
        torch.cuda.synchronize()
        lat.gmresdr(first, x, (c["m"], c["k"]), TOL, kappa=s["kappa"], defl=defl)
        s.update(defl=defl, b=b, x=_half(lat))
    elif kind == "train":
        x = torch.stack([_gauss_half(lat, gen) for _ in range(c["pairs"])])
        b = torch.zeros_like(x)
        torch.cuda.synchronize()
        for i in range(c["pairs"]):
            lat.hdbletm(x[i], 0, s["kappa"], out=b[i])
        s.update(b=b, x=x, w0=_weights(c, gen))
    else:
        be, bo = _z4_half(lat, gen), _z4_half(lat, gen)
        xe, xo = _gauss_half(lat, gen), _gauss_half(lat, gen)
        s.update(be=be, bo=bo, xe=xe, xo=xo, momfac=qq.momfacs(_dims(c))[:, : c["nmom"] - 1] if c["nmom"] > 1 else None)
        if s["momfac"] is not None:
            s["momfac"] = np.ascontiguousarray(s["momfac"])
    torch.cuda.synchronize()
    del u
    return s


# ---------------------------------------------------------------------------
# The calls
# ---------------------------------------------------------------------------
def run(s):
    c, lat = s["case"], s["lat"]
    kind = c["kind"]
    if kind == "operator":
        return lat.hdbletm(s["g"], c["idag"], s["kappa"], out=s["h"])
    if kind == "batch":
        xe, xo, _ = lat.fermprop_batch(s["be"], s["bo"], s["kappa"], precision=c["precision"], rhs_block=c["block"],
                                       tol=TOL, deflate=0, xe=s["xe"], xo=s["xo"])
        return xe, xo
    if kind == "gmresdr":
        xe, xo, _ = lat.fermprop(s["be"], s["bo"], s["kappa"], inverter=5, resmax=TOL, nGMRES=(c["m"], c["k"]),
                                 xe=s["xe"], xo=s["xo"])
        return xe, xo
    if kind == "gmresproj":
        s["x"].zero_()
        torch.cuda.synchronize()
        x, _ = lat.gmresproj(s["b"], s["x"], (c["m"] - c["k"], c["k"]), TOL, kappa=s["kappa"], defl=s["defl"])
        return x
    if kind == "train":
        net = qq.Net(_widths(c))
        net.set_weights(s["w0"])
        losses = net.train_pairs(lat, s["b"], s["x"], nsteps=c["steps"], lr=1e-3)
        w = net.get_weights()
        net.close()
        return losses, w
    return lat.average(s["be"], s["bo"], s["xe"], s["xo"], c["kappa"], nsub=c["nsub"], nmom=c["nmom"], nop=9,
                       momfac=s["momfac"])


# ---------------------------------------------------------------------------
# What a pass cannot do without, and how far two correct answers may lie apart
# ---------------------------------------------------------------------------
def work(case):
    """Bytes and flops.  A half spinor has vh sites; the links are counted as their two
    independent rows, 8 per site of a parity.  Solves count one nominal number of
    iterations (``iters``, as the present method needs on such fields): per iteration the
    operator's links and spinors once, and for GMRES the basis once per projection and
    once per update."""
    c = case
    nx, ny, nz, nt = _dims(c)
    vh = nx * ny * nz * nt // 2
    kind = c["kind"]
    dbl_flops = 2 * 1320.0 * vh + 96.0 * vh
    if kind == "operator":
        return {"bytes": vh * (2 * 192.0 + 8 * 96.0), "flops": dbl_flops}
    if kind == "batch":
        n, b = c["nrhs"], min(c["block"], c["nrhs"])
        size = 96.0 if c["precision"] == 32 else 52.0
        links = 2 * 2 * 8 * 48.0 * math.ceil(n / b)   # four hops, every link once per block
        vectors = n * size * (2 * 5 + 3 + 4 + 7)      # two operators and the three vector updates
        its = c["iters"]
        return {"bytes": vh * (its * (links + vectors) + n * 4 * 192.0), "flops": its * n * (2 * dbl_flops + 400.0 * vh)}
    if kind in ("gmresdr", "gmresproj"):
        its, m, k = c["iters"], c["m"], c["k"]
        cols = (m + k) / 2 if kind == "gmresdr" else (m - k) / 2
        return {"bytes": its * vh * (2 * 8 * 96.0 + 5 * 192.0 + 2 * cols * 192.0),
                "flops": its * (dbl_flops + vh * 2 * 2 * cols * 96.0)}
    if kind == "train":
        w = c["width"]
        layers = ((4, w), (w, w), (w, 4))
        # per layer and site: 9 paths, SU(3) transport of every input channel and the channel
        # mixing, forward, weight gradient and (but for the first layer) adjoint
        flops = sum(ci * 8 * 66.0 + 9 * 24.0 * ci * co + (ci * 8 * 66.0 + 9 * 24.0 * ci * co)
                    + (co * 8 * 66.0 + 9 * 24.0 * ci * co if l else 0) for l, (ci, co) in enumerate(layers))
        moved = sum((8 * 48.0 + 24.0 * (ci + co)) * (3 if l else 2) for l, (ci, co) in enumerate(layers))
        return {"bytes": c["steps"] * c["pairs"] * 2 * vh * moved, "flops": c["steps"] * c["pairs"] * 2 * vh * flops}
    powers = c["nsub"] + 1 if c["nsub"] > 1 else 0
    return {"bytes": 2 * vh * (4 * 192.0 + 4 * 96.0 + (5 * 4 * 8.0 if c["nmom"] > 1 else 0)),
            "flops": 2 * vh * (1320.0 * powers + c["nsub"] * 4 * 2 * (4 * 66.0 + 200.0))}


def tolerance(case):
    """Operators and loop sums are FP64 sums of some hundred terms (loop sums cancel over the
    sites of a slice).  Propagators are solved to a residual of 1e-10: two solutions differ by
    up to that times the condition of the operator.  Training runs in FP32 and normalises its
    steps by the gradients' own sizes."""
    kind = case["kind"]
    if kind == "operator":
        return {"rel": 1e-14}
    if kind == "average":
        return {"rel": 1e-12}
    if kind == "train":
        return {"rel": 1e-4}
    return {"rel": 1e-7}


# ---------------------------------------------------------------------------
# 64-bit statements in plain torch.  Fields are complex (..., t, z, y, x, spin, colour).
# ---------------------------------------------------------------------------
def _site_map(dims):
    """The reference's blocked site map: parity and the indices (ibl, ieo, isite) of each site."""
    nx, ny, nz, nt = dims
    t, z, y, x = np.meshgrid(np.arange(nt), np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    xb, yb, zb, tb = x >> 1, y >> 1, z >> 1, t >> 1
    isite = (xb >> 1) + yb * (nx // 4) + zb * (nx * ny // 8) + tb * (nx * ny * nz // 16)
    ibl = (x & 1) + 2 * (y & 1) + 4 * (z & 1) + 8 * (t & 1)
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda()
            for a in ((x + y + z + t) & 1, ibl, (xb + yb + zb + tb) & 1, isite)]


def _links(u, sm):
    m = torch.view_as_complex(u.view(u.shape[:-1] + (9, 2)).contiguous())
    return [m[sm[1], sm[2], mu, sm[3]].reshape(sm[1].shape + (3, 3)) for mu in range(4)]


def _lex(halves, sm):
    """Reference halves {parity: (8, 2, 4, ntotal, 6)} -> full field, zeros elsewhere."""
    out = torch.zeros(sm[0].shape + (4, 3), dtype=torch.complex128, device="cuda")
    for p, h in halves.items():
        m = sm[0] == p
        v = h[sm[1][m] // 2, sm[2][m], :, sm[3][m], :]  # (sites, spin, 6)
        out[m] = torch.view_as_complex(v.reshape(-1, 4, 3, 2).contiguous())
    return out


def _ref(psi, sm, parity, shape):
    """Full field -> reference half of one parity."""
    m = sm[0] == parity
    out = torch.zeros(shape, dtype=torch.float64, device="cuda")
    v = torch.view_as_real(psi[m].contiguous()).flatten(-2)
    for d in range(4):
        out[sm[1][m] // 2, sm[2][m], d, sm[3][m], :] = v[:, d]
    return out


_PERM = ((3, 2, 1, 0), (3, 2, 1, 0), (2, 3, 0, 1), (0, 1, 2, 3))
_FAC = ((1, 1, 1, 1), (-1j, 1j, -1j, 1j), (1, -1, 1, -1), (1, 1, -1, -1))


def _gamma(mu, v):
    f = torch.tensor(_FAC[mu], dtype=torch.complex128, device="cuda")[:, None]
    return v[..., list(_PERM[mu]), :] * f


def _twist(v):
    """i gamma_5."""
    return torch.cat((v[..., 2:, :], -v[..., :2, :]), dim=-2)


def _shift(f, mu, d, tail):
    """f(x + d mu) with the boundary factor; `tail` dimensions follow the site's."""
    ax = f.dim() - tail - 1 - mu
    g = torch.roll(f, -d, dims=ax)
    if BC[mu] != 1:
        g.select(ax, f.shape[ax] - 1 if d > 0 else 0).mul_(BC[mu])
    return g


def _mul(u, v):
    """u (..., 3, 3) on v (..., spin or channel, 3)."""
    return sum(u[..., None, :, b] * v[..., :, b, None] for b in range(3))


def _plain_shift(u, mu):
    return torch.roll(u, 1, dims=3 - mu)


def _hop(links, psi, idag=0):
    s = 1 if idag == 0 else -1
    out = torch.zeros_like(psi)
    for mu in range(4):
        f = _mul(links[mu], _shift(psi, mu, 1, 2))
        out += f - s * _gamma(mu, f)
        ub = _plain_shift(links[mu], mu)
        f = _mul(ub.conj().transpose(-1, -2), _shift(psi, mu, -1, 2))
        out += f + s * _gamma(mu, f)
    return out


def _dot(a, b):
    return (a.conj() * b).flatten(-6).sum(-1)


def _solve(links, b, kappa, mu, tol=1e-13, most=4000):
    """(1 + 2 kappa mu J - kappa H) x = b by BiCGStab on the even-odd preconditioned form,
    every right-hand side on its own scalars, restarted from the true residual."""
    tk = 2.0 * kappa * mu

    def op(v):  # M v, preconditioned by the diagonal's inverse
        d = v + tk * _twist(v) - kappa * _hop(links, v)
        return (d - tk * _twist(d)) / (1.0 + tk * tk)

    rhs = (b - tk * _twist(b)) / (1.0 + tk * tk)
    lead = (Ellipsis,) + (None,) * 6
    x = torch.zeros_like(b)
    bn = _dot(rhs, rhs).real.sqrt()
    for _ in range(6):
        r = rhs - op(x)
        if bool((_dot(r, r).real.sqrt() <= tol * bn).all()):
            break
        goal = torch.clamp(1e-9 * _dot(r, r).real.sqrt(), min=0.3 * tol * float(bn.max()))
        rhat, p = r.clone(), r.clone()
        rho = _dot(rhat, r)
        for it in range(most):
            v = op(p)
            alpha = rho / _dot(rhat, v)
            r = r - alpha[lead] * v
            t = op(r)
            omega = _dot(t, r) / (_dot(t, t) + 1e-300)
            x = x + alpha[lead] * p + omega[lead] * r
            r = r - omega[lead] * t
            if it % 8 == 7 and bool((_dot(r, r).real.sqrt() <= goal).all()):
                break
            new = _dot(rhat, r)
            beta = (new / rho) * (alpha / omega)
            rho = new
            p = r + beta[lead] * (p - omega[lead] * v)
    return x


def _exact_average(c, links, b, x, mf, sm):
    kappa, nsub, nmom, nt = c["kappa"], c["nsub"], c["nmom"], c["nt"]
    out = torch.zeros(9, nmom, nsub, nt, dtype=torch.complex128, device="cuda")
    powers = [b]
    if nsub > 1:
        for _ in range(nsub + 1):
            powers.append(_hop(links, powers[-1]))
    fac = None if mf is None else torch.from_numpy(mf).cuda()[:, :, sm[1], sm[2], sm[3]]
    total = lambda v: v.sum(dim=(1, 2, 3))  # noqa: E731
    dot = lambda a, d: (a.conj() * d).sum(dim=(-1, -2))  # noqa: E731
    for k in range(1, nsub + 1):
        y = x - sum((kappa ** n * powers[n] for n in range(k + 2)), torch.zeros_like(b)) if k > 1 else x
        ops = []
        for mu in range(4):
            udb = _mul(links[mu].conj().transpose(-1, -2), b)
            ubn = _mul(links[mu], _shift(b, mu, 1, 2))
            a = dot(_shift(y, mu, 1, 2), udb - _gamma(mu, udb)) - dot(y, ubn + _gamma(mu, ubn))
            ops.append(a.conj())
        ops.append(dot(y, b).conj() + (12.0 if k > 1 else 0.0))
        ops += [dot(y, _gamma(mu, b)).conj() for mu in range(4)]
        for i in range(9):
            out[i, 0, k - 1] = total(ops[i])
        for im in range(nmom - 1):
            f = fac[:, im]
            for i, (re, im_) in enumerate(((2, 1), (0, 2), (1, 0))):
                out[i, im + 1, k - 1] = torch.complex(total(f[re] * ops[i].imag), total(f[im_] * ops[i].imag))
            out[3, im + 1, k - 1] = total(f[3] * ops[3])
            out[4, im + 1, k - 1] = total(f[4] * ops[4])
    out[:4] *= kappa
    return torch.view_as_real(out).cpu().numpy()


def _exact_train(c, links, b, x, w0, even):
    """The whole training run in 64 bits: autograd through the layers, Adam on the real and
    imaginary parts of the weights (0.9, 0.999, 1e-12)."""
    ch = _widths(c)
    back = [_plain_shift(links[mu], mu).conj().transpose(-1, -2) for mu in range(4)]
    w = torch.view_as_real(torch.from_numpy(w0).cuda()).clone()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    losses = []
    for step in range(1, c["steps"] + 1):
        w.requires_grad_(True)
        wc, at, layers = torch.view_as_complex(w), 0, []
        for l in range(3):
            n = 9 * ch[l] * ch[l + 1]
            layers.append(wc[at: at + n].view(9, ch[l + 1], ch[l]))
            at += n
        loss = 0.0
        for i in range(c["pairs"]):
            f = b[i]
            for W in layers:
                g = torch.einsum("oc,...ca->...oa", W[0], f)
                for mu in range(4):
                    g = g + torch.einsum("oc,...ca->...oa", W[1 + 2 * mu], _mul(links[mu], _shift(f, mu, 1, 2)))
                    g = g + torch.einsum("oc,...ca->...oa", W[2 + 2 * mu], _mul(back[mu], _shift(f, mu, -1, 2)))
                f = g
            d = (f - x[i]) * even[..., None, None]
            loss = loss + (d.abs() ** 2).sum() / (x[i].abs() ** 2).sum() / c["pairs"]
        grad, = torch.autograd.grad(loss, w)
        losses.append(float(loss))
        w = w.detach()
        m = 0.9 * m + 0.1 * grad
        v = 0.999 * v + 0.001 * grad * grad
        w = w - 1e-3 * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-12)
    return np.array(losses), torch.view_as_complex(w.contiguous()).cpu().numpy()


def exact(case, seed):
    c = case
    kind = c["kind"]
    nx, ny, nz, nt = _dims(c)
    vol = nx * ny * nz * nt
    if kind in ("batch", "gmresdr", "gmresproj") and vol * c.get("nrhs", 1) * c["iters"] > 4e7:
        return None  # the plain solve would take too long
    if kind == "train" and vol * c["pairs"] * c["steps"] * c["width"] > 2e7:
        return None
    s = prepare(c, seed)
    _, u = _lattice(c, seed)
    sm = _site_map(_dims(c))
    links = _links(u, sm)
    del u
    shape = s["lat"].half_shape
    kappa, mu = s["kappa"]
    tk = 2.0 * kappa * mu
    if kind == "operator":
        g = _lex({0: s["g"]}, sm)
        h = _hop(links, g, c["idag"])
        h = _hop(links, h - tk * _twist(h), c["idag"])
        return _ref((g + tk * _twist(g)) / kappa ** 2 - h / (1.0 + tk * tk), sm, 0, shape)
    if kind in ("batch", "gmresdr"):
        be, bo = (s["be"], s["bo"]) if kind == "batch" else (s["be"][None], s["bo"][None])
        xs = [_solve(links, _lex({0: e, 1: o}, sm)[None], kappa, mu)[0] for e, o in zip(be, bo)]
        e = torch.stack([_ref(x, sm, 0, shape) for x in xs])
        o = torch.stack([_ref(x, sm, 1, shape) for x in xs])
        return (e, o) if kind == "batch" else (e[0], o[0])
    if kind == "gmresproj":
        x = _solve(links, (_lex({0: s["b"]}, sm) * kappa ** 2)[None], kappa, mu)[0]
        return _ref(x, sm, 0, shape)
    if kind == "train":
        b = [_lex({0: v}, sm) for v in s["b"]]
        x = [_lex({0: v}, sm) for v in s["x"]]
        return _exact_train(c, links, b, x, s["w0"], (sm[0] == 0).double())
    b, x = _lex({0: s["be"], 1: s["bo"]}, sm), _lex({0: s["xe"], 1: s["xo"]}, sm)
    return _exact_average(c, links, b, x, s["momfac"], sm)
