"""What a program that uses this engine spends its time on, as cases that can
be timed: Monte Carlo sweeps, sweeps with measurements, batches of lattices,
measurements on a stored configuration, and smearing.

Each case is one call sequence of the Python API.  `prepare` builds the
lattices and their links, `run` is one pass of a program's inner loop on them,
`exact` the same observables or links in 64-bit torch without the engine, and
`work` the bytes and operations a pass cannot do without.

The links are made by torch from the seed: A_mu(x) = an SU(N) matrix near 1,
then a Haar-random gauge transformation, so single links are spread over the
group while plaquettes sit near the value of the coupling, as in a thermalized
configuration.
"""
import math

import numpy as np
import torch

from sun_b200 import api

BETA = {2: 2.5, 3: 6.0, 4: 11.1, 6: 25.0}      # the couplings of the benchmark workloads
SPREAD = {2: 0.41, 3: 0.34, 4: 0.28, 6: 0.22}  # distance from 1 that gives their plaquettes
LAYOUT = {"SOA": api.SOA, "SOA12": api.SOA12}
APE_W, STOUT_W, HITS, TOL = 0.2, 0.1, 10, 1e-10
HYP = (0.75, 0.6, 0.3)


def _case(kind, N, dims, prec, layout="SOA", order="eo", **more):
    x, y, z, t = dims
    return dict(kind=kind, N=N, x=x, y=y, z=z, t=t, prec=prec, layout=layout, order=order, **more)


def listed():
    return [
        # plaquette and Polyakov loop of a small stored configuration: two
        # calls with a host result each, launch latency
        _case("measure", 3, (8, 8, 8, 8), "f64", name="measure_su3_8x4_f64"),
        # the plain small chain: both observables after every sweep
        _case("sweep_measure", 3, (8, 8, 8, 8), "f64", sweeps=10, name="chain_su3_8x4_f64"),
        # the production sweep (1 heatbath + 4 overrelaxation) on the
        # benchmark lattice, compressed FP32 links
        _case("sweep", 3, (32, 32, 32, 32), "f32", "SOA12", name="sweep_su3_32x4_f32"),
        # the same in full FP64 links on a lattice with four different extents
        _case("sweep", 3, (22, 18, 14, 26), "f64", name="sweep_su3_22.18.14.26_f64"),
        # the other gauge groups in FP32
        _case("sweep", 2, (24, 24, 24, 24), "f32", name="sweep_su2_24x4_f32"),
        _case("sweep", 4, (24, 24, 24, 24), "f32", name="sweep_su4_24x4_f32"),
        _case("sweep", 6, (24, 24, 24, 24), "f32", name="sweep_su6_24x4_f32"),
        # an ensemble of uneven lattices advanced together, L in {8, 12, 16},
        # T in {L, 2L}, with the plaquettes read back
        _case("batch", 3, (8, 8, 8, 8), "f32", "SOA12", lattices=12, sweeps=2, name="batch_su3_12_f32"),
        # observables of the benchmark lattice
        _case("measure", 3, (32, 32, 32, 32), "f32", "SOA12", name="measure_su3_32x4_f32"),
        # Wilson loops to 4 x 4, the static-potential measurement
        _case("wilson", 3, (24, 24, 24, 24), "f32", "SOA12", R=4, T=4, name="wilson_su3_24x4_f32"),
        # smearing a copy of a configuration before such a measurement: APE
        # steps in the reference's own storage, and one HYP step
        _case("ape", 3, (24, 24, 24, 24), "f64", "SOA", "lex", steps=3, name="ape_su3_24x4_f64"),
        _case("hyp", 3, (24, 24, 24, 24), "f32", "SOA12", steps=1, name="hyp_su3_24x4_f32"),
    ]


def _dims(rng, least, most_sites):
    """Four even extents from `least` up, the volume spread over its logarithm."""
    goal = math.exp(rng.uniform(math.log(least ** 4), math.log(most_sites)))
    while True:
        d = [2 * round(goal ** 0.25 * math.exp(rng.uniform(-0.5, 0.5)) / 2) for _ in range(4)]
        v = d[0] * d[1] * d[2] * d[3]
        if min(d) >= least and max(d) <= 64 and 0.5 * goal <= v <= most_sites:
            return d


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep_measure", "batch", "measure", "measure", "wilson", "wilson",
                       "ape", "stout", "hyp"])
    N = 3 if kind in ("stout", "batch") else rng.choice([2, 3, 3, 3, 4, 6] if kind == "sweep" else [2, 3, 3, 3, 3, 4])
    prec = rng.choice(["f32", "f32", "f64"])
    layout = rng.choice(["SOA", "SOA12", "SOA12"]) if N == 3 and prec == "f32" else "SOA"
    order = rng.choice(["eo", "lex"]) if kind in ("measure", "wilson", "ape", "stout", "hyp") else "eo"
    # the largest listed sweep costs as much as 24^4 of SU(6) in FP32
    most = 24 ** 4 if N < 6 else 24 ** 4 * (1.0 if prec == "f32" else 0.45)
    if kind in ("sweep", "measure") and N == 3 and prec == "f32":
        most = 32 ** 4
    if kind == "sweep_measure":
        return _case(kind, N, _dims(rng, 4, 14 ** 4), prec, layout, order, sweeps=rng.randint(1, 12))
    if kind == "batch":
        lattices = rng.randint(2, {"SOA12": 16, "SOA": 10 if prec == "f32" else 5}[layout])
        return _case(kind, N, _dims(rng, 4, 8 ** 4), prec, layout, order, lattices=lattices, sweeps=rng.randint(1, 2))
    if kind == "wilson":
        return _case(kind, N, _dims(rng, 6, most / (3 if N == 4 else 1)), prec, layout, order, R=rng.randint(1, 5), T=rng.randint(1, 5))
    if kind in ("ape", "stout"):
        return _case(kind, N, _dims(rng, 4, most), prec, layout, order, steps=rng.randint(1, 3))
    if kind == "hyp":
        return _case(kind, N, _dims(rng, 4, most / (3 if N == 4 else 1)), prec, layout, order, steps=1)
    return _case(kind, N, _dims(rng, 4, most), prec, layout, order)


# -- links in torch: [V, 4, N, N] complex128, lexicographic sites, x fastest ---
def _extents(case):
    return (case["x"], case["y"], case["z"], case["t"])


def _mul(A, B):
    return sum(A[..., :, k, None] * B[..., None, k, :] for k in range(A.shape[-1]))


def _dag(A):
    return A.conj().transpose(-1, -2)


def _shift(F, dims, mu, n=1):
    """F(x + n mu) for F [V, ...]."""
    X, Y, Z, T = dims
    return torch.roll(F.reshape(T, Z, Y, X, *F.shape[1:]), -n, 3 - mu).reshape(F.shape)


def _special_unitary(M):
    """Gram-Schmidt over rows, then the determinant's phase spread over them."""
    rows = []
    for i in range(M.shape[-1]):
        v = M[..., i, :]
        for r in rows:
            v = v - (r.conj() * v).sum(-1, keepdim=True) * r
        rows.append(v / v.abs().square().sum(-1, keepdim=True).sqrt())
    U = torch.stack(rows, -2)
    det = torch.ones_like(U[..., 0, 0])
    W = U.clone()
    for k in range(W.shape[-1]):  # elimination; the leading minors of these matrices do not vanish
        det = det * W[..., k, k]
        f = W[..., k + 1:, k] / W[..., k, k, None]
        W[..., k + 1:, :] -= f[..., None] * W[..., k, None, :]
    return U * torch.polar(torch.ones_like(det.real), -det.angle() / U.shape[-1])[..., None, None]


def _links(N, dims, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    V = dims[0] * dims[1] * dims[2] * dims[3]

    def gauss(*shape):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=torch.complex64).to(torch.complex128)

    G = _special_unitary(gauss(V, N, N))
    one = torch.eye(N, device="cuda", dtype=torch.complex128)
    U = torch.empty(V, 4, N, N, device="cuda", dtype=torch.complex128)
    for mu in range(4):
        A = _special_unitary(one + SPREAD[N] * gauss(V, N, N))
        U[:, mu] = _mul(_mul(G, A), _dag(_shift(G, dims, mu)))
    return U


def _sites(dims, order):
    """Lexicographic site of each site in storage order."""
    V = dims[0] * dims[1] * dims[2] * dims[3]
    s = torch.arange(V, device="cuda")
    if order == "lex":
        return s
    X, Y, Z, _ = dims
    odd = (s % X + s // X % Y + s // (X * Y) % Z + s // (X * Y * Z)) % 2
    return torch.cat([s[odd == 0], s[odd == 1]])


def _image(U, dims, prec, layout, order):
    """The device image of links [V, 4, N, N]: [elements, 4, V]."""
    rows = U[:, :, :2] if layout == "SOA12" else U
    flat = rows.reshape(rows.shape[0], 4, -1)[_sites(dims, order)]
    return flat.permute(2, 1, 0).to(torch.complex64 if prec == "f32" else torch.complex128).contiguous()


def _stored(case, seed):
    """The links as the lattice holds them, in 64 bits."""
    U = _links(case["N"], _extents(case), seed)
    if case["prec"] == "f32":
        U = U.to(torch.complex64).to(torch.complex128)
    if case["layout"] == "SOA12":
        U[:, :, 2] = torch.linalg.cross(U[:, :, 0], U[:, :, 1]).conj()
    return U


# -- lattices -----------------------------------------------------------------
_context = None


def _ctx():
    global _context
    if _context is None:
        _context = api.Context(0)
    return _context


class _Device:
    def __init__(self, g):
        self.lattice = g  # a tensor on the image keeps the lattice
        self.__cuda_array_interface__ = dict(shape=(g.Bytes() // (4 if g.prec == "f32" else 8),), version=3,
                                             typestr="<f4" if g.prec == "f32" else "<f8", data=(g.GetPtr(), False),
                                             strides=None)


def _view(g):
    """The lattice's device image as real numbers, without a copy."""
    return torch.as_tensor(_Device(g), device="cuda")


def _lattice(case, dims, seed, layout=None, fill=True):
    layout = layout or case["layout"]
    N = case["N"]
    g = api.gauge(_ctx(), N=N, dims=dims, beta=BETA[N], atype=LAYOUT[layout], evenodd=case["order"] == "eo",
                  prec=case["prec"], seed=seed, reunit_every=10)
    if fill:
        img = _image(_links(N, dims, seed), dims, case["prec"], layout, case["order"])
        _view(g).copy_(torch.view_as_real(img).reshape(-1))
        torch.cuda.synchronize()
    return g


def _ensemble(case):
    """The extents of a batch: L, L + L/2 and 2 L in turn, T as drawn or twice that."""
    X = _extents(case)
    out = []
    for i in range(case["lattices"]):
        f = (2, 3, 4)[i % 3]
        d = [2 * ((e * f + 2) // 4) for e in X]
        out.append((d[0], d[1], d[2], d[3] * (1 + i // 3 % 2)))
    return out


def prepare(case, seed):
    kind, dims = case["kind"], _extents(case)
    state = dict(case=case)
    if kind == "batch":
        state["lattices"] = [_lattice(case, d, seed + 7919 * i) for i, d in enumerate(_ensemble(case))]
        state["batch"] = api.Batch(_ctx())
        for g in state["lattices"]:
            state["batch"].add(g)
    else:
        state["g"] = _lattice(case, dims, seed)
        if kind in ("ape", "stout", "hyp"):  # smearing works in place: on a second lattice
            state["smeared"] = _lattice(case, dims, seed, fill=False)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "sweep":
        api.Sweep(state["g"], 1, 4, 1)
        return _view(state["g"])
    if kind == "sweep_measure":
        plaq, poly = api.SweepMeasure(state["g"], 1, 4, case["sweeps"])
        return {"plaquette": plaq, "polyakov": poly, "links": _view(state["g"])}
    if kind == "batch":
        state["batch"].sweep(1, 4, case["sweeps"], graph=True)
        return {"plaquette": state["batch"].plaquette(), "links": [_view(g) for g in state["lattices"]]}
    if kind == "measure":
        p, l = api.PlaquetteCUB(state["g"]).Run(), api.OnePolyakovLoop(state["g"]).Run()
        return np.array([p.real, p.imag, l.real, l.imag])
    if kind == "wilson":
        return api.WilsonLoop(state["g"], case["R"], case["T"])
    s = state["smeared"]
    s.Copy(state["g"])
    if kind == "ape":
        api.ApplyAPEinSpace(s, APE_W, case["steps"], HITS, TOL)
    elif kind == "stout":
        api.ApplyStoutinSpace(s, STOUT_W, case["steps"])
    else:
        api.ApplyHYPinSpace(s, case["steps"], HITS, TOL, api.ParamHYP(*HYP))
    return _view(s)


def work(case):
    """Bytes: an update phase (parity, mu) reads every link of three directions
    and all of direction mu and writes half of the latter, so 9 link records
    per update; a measurement reads its links once; a smearing step reads the
    four directions and writes the spatial three (HYP also each level's 12
    links per site once each way), a copy reads and writes all.
    Operations: complex multiply-adds (8) of the matrix products."""
    N, kind = case["N"], case["kind"]
    elems = 6 if case["layout"] == "SOA12" else N * N
    size = 8 if case["prec"] == "f32" else 16
    rec, full = elems * size, N * N * size
    prod = 8.0 * N ** 3
    pairs = N * (N - 1) // 2
    V = float(case["x"] * case["y"] * case["z"] * case["t"])
    if kind in ("sweep", "sweep_measure", "batch"):
        if kind == "batch":
            V = float(sum(d[0] * d[1] * d[2] * d[3] for d in _ensemble(case)))
        n = case.get("sweeps", 1)
        return {"bytes": n * 20 * V * 9 * rec, "flops": n * 20 * V * (12 * prod + pairs * 64.0 * N)}
    if kind == "measure":
        return {"bytes": 4 * V * rec, "flops": V * (6 * (2 * prod + 8.0 * N * N) + prod)}
    if kind == "wilson":
        R, T = case["R"], case["T"]
        lines = 3 * (R - 1) + (T - 1)              # longer lines from shorter ones
        loops = 3 * R * T * (2 * prod + 8.0 * N * N)
        return {"bytes": 4 * V * rec, "flops": V * (lines * prod + loops)}
    steps = case["steps"]
    hits = HITS * pairs * 64.0 * N
    if kind == "ape":
        return {"bytes": V * rec * (8 + 7 * steps), "flops": steps * 3 * V * (8 * prod + hits)}
    if kind == "stout":
        return {"bytes": V * rec * (8 + 7 * steps), "flops": steps * 3 * V * (8 * prod + 3 * prod)}
    return {"bytes": V * (rec * 8 + steps * (7 * rec + 48 * full)),
            "flops": steps * V * (12 * (4 * prod + hits) + 12 * (8 * prod + hits) + 3 * (12 * prod + hits))}


# -- the same in 64-bit torch -----------------------------------------------------
def _trace(A):
    return A.diagonal(dim1=-2, dim2=-1).sum(-1)


def _trace_nd(A, B):
    return (A * B.conj()).sum((-1, -2))


def _plane_staple(R, A, dims, a, r):
    """R(x) A(x+r) R(x+a)^dag + R(x-r)^dag A(x-r) R(x-r+a)."""
    Ra = _shift(R, dims, a)
    up = _mul(_mul(R, _shift(A, dims, r)), _dag(Ra))
    return up + _shift(_mul(_mul(_dag(R), A), Ra), dims, r, -1)


def _project(W, Q, hits, tol):
    """Cabibbo-Marinari maximisation of Re tr W Q^dag from W; tol > 0: each
    matrix stops once Re tr(W Q) changes by at most tol."""
    N = W.shape[-1]
    W = W.clone()
    live = torch.ones_like(W[..., 0, 0].real, dtype=torch.bool)
    old = _trace(_mul(W, Q)).real if tol > 0 else None
    for _ in range(hits):
        new = W.clone()
        for gap in range(1, N):
            for p in range(N - gap):
                q = p + gap
                up, uq = new[..., p, :].clone(), new[..., q, :].clone()
                b = [(u * Q[..., k, :].conj()).sum(-1) for u in (up, uq) for k in (p, q)]
                r = torch.stack([(b[0] + b[3]).real, (b[1] + b[2]).imag, (b[1] - b[2]).real, (b[0] - b[3]).imag], -1)
                c = r / r.square().sum(-1, keepdim=True).sqrt()
                d = torch.complex(c[..., 0], -c[..., 3])[..., None]
                o = torch.complex(-c[..., 2], -c[..., 1])[..., None]
                new[..., p, :] = d * up + o * uq
                new[..., q, :] = d.conj() * uq - o.conj() * up
        W = torch.where(live[..., None, None], new, W)
        if tol > 0:
            now = _trace(_mul(W, Q)).real
            live = live & ((now - old) / old > tol)
            old = now
    return W


def _exact_measure(U, dims):
    V, _, N, _ = U.shape
    sums = [0.0, 0.0]
    for mu in range(3):
        for nu in range(mu + 1, 4):
            P = _mul(U[:, mu], _shift(U[:, nu], dims, mu))
            Q = _mul(U[:, nu], _shift(U[:, mu], dims, nu))
            sums[nu == 3] += _trace_nd(P, Q).real.sum().item()
    X, Y, Z, T = dims
    L = U[:, 3].reshape(T, X * Y * Z, N, N)
    P = L[0]
    for t in range(1, T):
        P = _mul(P, L[t])
    loop = _trace(P).sum().item() / (N * X * Y * Z)
    return np.array([sums[0] / (3 * N * V), sums[1] / (3 * N * V), loop.real, loop.imag])


def _exact_wilson(U, dims, R, T):
    V, _, N, _ = U.shape
    one = torch.eye(N, device=U.device, dtype=U.dtype).expand(V, N, N)
    time = [one]
    for t in range(T):
        time.append(_mul(time[t], _shift(U[:, 3], dims, 3, t)))
    out = np.zeros((R + 1, T + 1), dtype=np.complex128)
    for mu in range(3):
        line = one
        for r in range(R + 1):
            if r:
                line = _mul(line, _shift(U[:, mu], dims, mu, r - 1))
            for t in range(T + 1):
                P = _mul(line, _shift(time[t], dims, mu, r))
                Q = _mul(time[t], _shift(line, dims, 3, t))
                out[r, t] += _trace_nd(P, Q).sum().item()
    return out / (3 * N * V)


def _exact_ape(U, dims):
    N, new = U.shape[-1], U.clone()
    for mu in range(3):
        S = sum(_plane_staple(U[:, nu], U[:, mu], dims, mu, nu) for nu in range(3) if nu != mu)
        Q = (U[:, mu] + APE_W * S) / (1 + 6 * APE_W)
        if N == 3:
            new[:, mu] = _project(torch.eye(3, device=U.device, dtype=U.dtype).expand_as(Q), Q, HITS, 0.0)
        else:
            new[:, mu] = _project(U[:, mu], Q, HITS, TOL)
    return new


def _exact_stout(U, dims):
    new = U.clone()
    one = torch.eye(3, device=U.device, dtype=U.dtype)
    for mu in range(3):
        S = sum(_plane_staple(U[:, nu], U[:, mu], dims, mu, nu) for nu in range(3) if nu != mu)
        Om = _mul(STOUT_W * S, _dag(U[:, mu]))
        Q = 0.5j * (_dag(Om) - Om)
        X = 1j * (Q - _trace(Q)[:, None, None] / 3 * one) / 64
        E, term = one + X, X
        for k in range(2, 14):
            term = _mul(term, X) / k
            E = E + term
        for _ in range(6):
            E = _mul(E, E)
        new[:, mu] = _mul(E, U[:, mu])
    return new


def _exact_hyp(U, dims):
    a1, a2, a3 = (float(np.float32(a)) for a in HYP)
    bar, til, new = {}, {}, U.clone()
    for m in range(4):
        for e in range(4):
            if e != m:
                S = _plane_staple(U[:, e], U[:, m], dims, m, e)
                bar[m, e] = _project(U[:, m], (1 - a3) * U[:, m] + 0.5 * a3 * S, HITS, TOL)
    for a in range(4):
        for b in range(4):
            if b != a:
                S = 0
                for r in range(4):
                    if r not in (a, b):
                        s = 6 - a - b - r
                        S = S + _plane_staple(bar[r, s], bar[a, s], dims, a, r)
                til[a, b] = _project(U[:, a], (1 - a2) * U[:, a] + 0.25 * a2 * S, HITS, TOL)
    for m in range(3):
        S = sum(_plane_staple(til[n, m], til[m, n], dims, m, n) for n in range(4) if n != m)
        new[:, m] = _project(U[:, m], (1 - a1) * U[:, m] + a1 / 6 * S, HITS, TOL)
    return new


def exact(case, seed):
    kind, dims = case["kind"], _extents(case)
    if kind in ("sweep", "sweep_measure", "batch"):
        return None  # random draws with accept / reject decisions
    U = _stored(case, seed)
    if kind == "measure":
        return _exact_measure(U, dims)
    if kind == "wilson":
        return _exact_wilson(U, dims, case["R"], case["T"])
    for _ in range(case["steps"]):
        if kind == "ape":
            U = _exact_ape(U, dims)
        elif kind == "stout":
            U = _exact_stout(U, dims)
        else:
            U = _exact_hyp(U, dims)
    return torch.view_as_real(_image(U, dims, "f64", case["layout"], case["order"])).reshape(-1)
