"""Timed cases of the bimetric TreePM engine: what a simulation program has it do.

A case is one call pattern of a program that uses the engine:

* ``step``      KDK steps of one box that stays on the device, then the state
                and the accelerations read into device arrays (a run that
                analyses or saves every few steps);
* ``forces``    positions handed over in device arrays, accelerations handed
                back (an external integrator; TreePMForce.update +
                compute_all_forces with device memory);
* ``host``      one step of a box whose state lives in pinned host memory;
* ``batch``     one step of many uneven boxes in one batch (parameter scans);
* ``rcompat``   the reference solver's call shape and formulas
                (GpuNBodyTwoPass): drift-kick-drift steps, forces, readback.

Sizes, box lengths, grids, mass ratio, cut and softening rules are those of
bench.py and the tests: 2 x 16^3 .. 2 x 224^3 particles, PM 32^3 .. 512^3,
r_s = 1.25 cells, cut 4.5 r_s or widened by cut_tail_ppm = 440, softening
spacing / 30.  Time steps are small, so that the particle distribution a case
stands for does not change over the passes that time it; the cost of a step
does not depend on dt.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "janus-sim_b200"))
import janus_treepm as J  # noqa: E402

HUBBLE = 0.3          # 1/Gyr, drag of the kicks
DEVICE = "cuda"


# ---------------------------------------------------------------- the cases
def _case(name, kind, ic, n_p, n_m, L, M, **kw):
    c = dict(name=name, kind=kind, ic=ic, n_p=n_p, n_m=n_m, L=float(L), M=M, theta=0.5, tail=0, mu=19.0,
             dt=1.0e-4, steps=1, lam=0.0, boxes=1, order=0, interlace=0)
    c.update(kw)
    return c


def listed():
    n224, n128, n112, n96, n64, n48 = 224 ** 3, 128 ** 3, 112 ** 3, 96 ** 3, 64 ** 3, 48 ** 3
    return [
        # the smallest box of a scan: launches and host latency count
        _case("step_2x16", "step", "lattice", 16 ** 3, 16 ** 3, 60.0, 32, steps=4),
        # the smallest workload of the bench and the tests: uniform random, PM 64^3
        _case("step_2x32_uniform", "step", "uniform", 32 ** 3, 32 ** 3, 64.0, 64, steps=2),
        # positions in, accelerations out; mu realised as a count ratio (N-/N+ = 19), odd counts
        _case("forces_ragged", "forces", "uniform", 30011, 570209, 100.0, 128, mu=570209 / 30011),
        # the reference's call shape and formulas, as a program ported to this engine first runs
        _case("rcompat_2x48", "rcompat", "lattice", n48, n48, 96.0, 128),
        # opposite-species pairs Yukawa-screened (two sources, two sets of grids)
        _case("step_2x64_screened", "step", "lattice", n64, n64, 120.0, 128, lam=5.0),
        # the largest box of a scan, one handle
        _case("step_2x96", "step", "lattice", n96, n96, 150.0, 256, steps=2),
        # a scan: 24 uneven boxes, 16^3 .. 96^3 per species, PM 32^3 .. 256^3, one launch per stage
        _case("batch_24", "batch", "lattice", 16 ** 3, n96, 50.0, 256, boxes=24),
        # state held in pinned host memory between steps
        _case("host_2x112", "host", "lattice", n112, n112, 125.0, 256, tail=440),
        # collapsed structures at a tight opening angle: the tree walk with its multipoles
        _case("clustered_2x64_theta03", "step", "plummer", n64, n64, 50.0, 128, theta=0.3, dt=2.0e-6),
        # collapsed structures at the bench's size and accuracy setting
        _case("clustered_2x128", "step", "plummer", n128, n128, 100.0, 256, tail=440, dt=2.0e-6),
        # the production step at the config's cut
        _case("step_2x224", "step", "lattice", n224, n224, 250.0, 512),
        # the production step at the accuracy setting of the bench's headline
        _case("step_2x224_tail", "step", "lattice", n224, n224, 250.0, 512, tail=440),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid_for(n):
    """PM grid of n particles per species: the next power of two >= 2 n^(1/3), 32 .. 512."""
    return min(512, max(32, 1 << math.ceil(math.log2(2.0 * n ** (1.0 / 3.0)) - 1e-9)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "forces", "batch", "host", "rcompat", "clustered", "screened"])
    kw = dict(tail=rng.choice([0, 440]), mu=rng.uniform(5.0, 30.0), steps=rng.choice([1, 2, 3]))
    ic = "uniform" if kind == "forces" else rng.choice(["lattice", "lattice", "uniform"])
    top = {"step": 200 ** 3, "forces": 128 ** 3, "batch": 96 ** 3, "host": 140 ** 3, "rcompat": 64 ** 3,
           "clustered": 110 ** 3, "screened": 96 ** 3}[kind]
    n_p = _log_int(rng, 16 ** 3, top)
    n_m = max(1, int(n_p * rng.uniform(0.8, 1.2)))
    L = rng.uniform(50.0, 300.0)
    if kind == "forces":
        n_p, n_m = max(64, n_p // 19), n_p
        kw["mu"] = n_m / n_p
    if kind in ("step", "forces"):
        kw["order"], kw["interlace"] = rng.choice([(0, 0), (0, 0), (0, 0), (3, 0), (2, 2), (4, 2)])
    M = _grid_for(max(n_p, n_m))
    if kind == "rcompat":
        # its cut is rounded down to whole Mpc: keep it at several
        kw.update(tail=0, steps=1)
        L = rng.uniform(90.0, 200.0) * M / 128
        ic = "lattice"
    elif kind == "batch":
        kw.update(boxes=rng.randint(3, 24), steps=1, tail=0)
        n_m = max(n_p, 24 ** 3)
        n_p, L, M = 16 ** 3, 50.0, _grid_for(n_m)
        ic = "lattice"
    elif kind == "clustered":
        kind, ic = "step", "plummer"
        kw.update(theta=rng.choice([0.3, 0.5, 0.7]), dt=2.0e-6, steps=1)
        L = rng.uniform(0.7, 1.1) * 100.0 * n_p ** (1.0 / 3.0) / 128.0
    elif kind == "screened":
        kind = "step"
        kw.update(lam=rng.uniform(1.0, 20.0), steps=1)
    elif kind == "host":
        kw.update(steps=1)
    c = _case("", kind, ic, n_p, n_m, L, M, **kw)
    del c["name"]
    return c


def _batch_boxes(case):
    """The boxes of a batch case: per-species side log-uniform over the range
    the case gives, L U(50, 300), PM the next power of two >= 2 n, mu U(5, 30)."""
    rng = np.random.default_rng(case["n_m"] + 131 * case["boxes"])
    lo, hi = round(case["n_p"] ** (1 / 3)), round(case["n_m"] ** (1 / 3))
    out = []
    for _ in range(case["boxes"]):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        out.append(dict(case, kind="step", n_p=n ** 3, n_m=n ** 3, L=float(rng.uniform(50.0, 300.0)),
                        M=max(32, 1 << math.ceil(math.log2(2 * n))), mu=float(rng.uniform(5.0, 30.0)), boxes=1))
    return out


# ---------------------------------------------------------------- inputs
def _wrap(x, L):
    y = torch.remainder(x + 0.5 * L, L) - 0.5 * L
    return torch.where(y >= 0.5 * L, y - L, y)


def _lattice(n, L, sign, gen, noise_seed):
    """n particles on the lattice of side ceil(n^(1/3)) (a random subset when n
    is no cube) with Zel'dovich displacements, P(k) ~ k^-2.5 exp(-(k/k_c)^2), rms
    0.3 spacing; the m- species half a cell off with the opposite displacement."""
    s = round(n ** (1.0 / 3.0))
    s += 1 if s ** 3 < n else 0
    a = L / s
    g2 = torch.Generator(DEVICE).manual_seed(noise_seed)
    dk = torch.fft.rfftn(torch.randn(s, s, s, generator=g2, device=DEVICE))
    k1 = 2 * math.pi * torch.fft.fftfreq(s, d=a, device=DEVICE)
    kr = 2 * math.pi * torch.fft.rfftfreq(s, d=a, device=DEVICE)
    kz, ky, kx = k1[:, None, None], k1[None, :, None], kr[None, None, :]
    k2 = kz * kz + ky * ky + kx * kx
    k2[0, 0, 0] = 1.0
    kc = 0.5 * math.pi / a
    dk = dk * k2 ** -0.625 * torch.exp(-0.5 * k2 / kc ** 2) / k2
    dk[0, 0, 0] = 0.0
    if sign < 0:
        ph = 0.5 * a * (kx + ky + kz)
        dk = -dk * torch.complex(torch.cos(ph), torch.sin(ph))
    psi = torch.stack([torch.fft.irfftn(1j * k * dk, s=(s, s, s)) for k in (kx, ky, kz)], -1).reshape(-1, 3)
    psi = psi * (0.3 * a / psi.square().sum(1).mean().sqrt())
    g = (torch.arange(s, device=DEVICE) + 0.5) * a - 0.5 * L + (0.5 * a if sign < 0 else 0.0)
    Z, Y, X = torch.meshgrid(g, g, g, indexing="ij")
    pos = _wrap(torch.stack([X, Y, Z], -1).reshape(-1, 3) + psi, L)
    vel = 0.05 * psi
    if n < s ** 3:
        keep = torch.randperm(s ** 3, generator=gen, device=DEVICE)[:n].sort().values
        pos, vel = pos[keep], vel[keep]
    return pos.contiguous(), vel.contiguous()


def _plummer(n, L, species, gen, centres, scales):
    """80 % of the particles in every second Plummer sphere, 20 % background."""
    mine = torch.arange(species, len(scales), 2, device=DEVICE)
    n_bg = n // 5
    n_cl = n - n_bg
    which = mine[torch.randint(len(mine), (n_cl,), generator=gen, device=DEVICE)]
    u = torch.rand(n_cl, generator=gen, device=DEVICE).clamp_(1e-6, 1.0 - 1e-6)
    r = torch.minimum(scales[which] / torch.sqrt(u ** (-2.0 / 3.0) - 1.0), 10.0 * scales[which])
    d = torch.randn(n_cl, 3, generator=gen, device=DEVICE)
    d = d / d.norm(dim=1, keepdim=True)
    bg = (torch.rand(n_bg, 3, generator=gen, device=DEVICE) - 0.5) * L
    pos = _wrap(torch.cat([centres[which] + d * r[:, None], bg]), L)
    pos = pos[torch.randperm(n, generator=gen, device=DEVICE)].contiguous()
    return pos, 0.05 * torch.randn(n, 3, generator=gen, device=DEVICE)


def _inputs(case, seed):
    """(pos_p, vel_p, pos_m, vel_m) float32 (n, 3) on the device."""
    gen = torch.Generator(DEVICE).manual_seed(seed)
    L, n = case["L"], (case["n_p"], case["n_m"])
    out = []
    if case["ic"] == "plummer":
        # the bench's density of spheres: 512 in a box of 100 Mpc
        k = max(8, 2 * round(256 * (L / 100.0) ** 3))
        centres = (torch.rand(k, 3, generator=gen, device=DEVICE) - 0.5) * L
        scales = torch.exp(torch.rand(k, generator=gen, device=DEVICE) * math.log(20.0) + math.log(0.05))
        for s in (0, 1):
            out += _plummer(n[s], L, s, gen, centres, scales)
    else:
        for s in (0, 1):
            if case["ic"] == "lattice":
                out += _lattice(n[s], L, 1 - 2 * s, gen, seed)
            else:
                out += [_wrap((torch.rand(n[s], 3, generator=gen, device=DEVICE) - 0.5) * L, L),
                        0.05 * torch.randn(n[s], 3, generator=gen, device=DEVICE)]
    # no particle within 1e-4 L of a face: one that rounding carries through it
    # comes back at the other side, a difference of L between equal results
    for a in out[0::2]:
        a.clamp_(-0.4999 * L, 0.4999 * L)
    return out


# ---------------------------------------------------------------- plan
def _config(case):
    L, M = case["L"], case["M"]
    n = case["n_p"] + case["n_m"]
    r_s = 1.25 * L / M
    spacing = L / (0.5 * n) ** (1.0 / 3.0)
    return J.Config(box_L=L, pm_grid=M, theta=case["theta"], softening=L / n ** (1.0 / 3.0) / 30.0, r_s=r_s,
                    r_cut=4.5 * r_s, mu=case["mu"], G_mass_plus=1.0e-3 * (spacing / (250.0 / 224.0)) ** 3,
                    pm_order=case["order"], pm_interlace=case["interlace"], cut_tail_ppm=case["tail"])


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _ok(code, what):
    if code != 0:
        raise J.JanusError(code, what)


def _rcompat_cut(case):
    return max(2.0, float(math.floor(4.5 * 1.25 * case["L"] / case["M"])))


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "batch":
        B = J.Batch()
        ids, outs = [], []
        for i, bx in enumerate(_batch_boxes(case)):
            x = _inputs(bx, seed * 1000 + i)
            ids.append(B.add(_config(bx), *[a.cpu().numpy() for a in x]))
            outs.append([torch.empty_like(a) for a in (x[0], x[1], x[0], x[2], x[3], x[2])])
        B.forces(ids)
        st.update(batch=B, ids=ids, out=outs)
        return st
    x = _inputs(case, seed)
    torch.cuda.synchronize()
    if kind == "rcompat":
        pos = torch.cat([x[0], x[2]]).cpu().numpy()
        vel = torch.cat([x[1], x[3]]).cpu().numpy()
        signs = np.concatenate([np.ones(case["n_p"], np.int8), -np.ones(case["n_m"], np.int8)])
        g = J.GpuNBodyTwoPass.with_custom_ics(pos, vel, signs, case["L"], pm_grid=case["M"])
        g.compute_forces(_rcompat_cut(case))
        st["sim"] = g
        return st
    s = J.Solver(_config(case))
    s.set_state_device(*x)
    if case["lam"] > 0.0:
        s.set_screening(case["lam"])
    # pos, vel, acc per species
    out = [torch.empty_like(a) for a in (x[0], x[1], x[0], x[2], x[3], x[2])]
    s.accel_device(out[2], out[5])
    st.update(solver=s, out=out)
    if kind == "forces":
        st["pos"] = (x[0], x[2])
    if kind == "host":
        pin = [a.cpu().pin_memory().numpy() for a in (x[0], x[1], out[2], x[2], x[3], out[5])]
        st["host"] = pin
    return st


# ---------------------------------------------------------------- one pass
def run(st):
    case = st["case"]
    kind = case["kind"]
    lib = J.library()
    if kind == "batch":
        B = st["batch"]
        B.step(st["ids"], case["dt"], HUBBLE, 1.0, case["steps"])
        for i, o in zip(st["ids"], st["out"]):
            _ok(lib.jt_batch_get_state(B._b, i, _p(o[0]), _p(o[1]), _p(o[3]), _p(o[4]), J.JT_MEM_DEVICE), "state")
            _ok(lib.jt_batch_get_accel(B._b, i, _p(o[2]), _p(o[5]), J.JT_MEM_DEVICE), "accel")
        # one tensor per quantity and species, boxes in order
        return [torch.cat([o[k] for o in st["out"]]) for k in range(6)]
    if kind == "rcompat":
        g = st["sim"]
        g.step_treepm_gpu(case["dt"], _rcompat_cut(case), HUBBLE, 1.0)
        acc = g.compute_forces(_rcompat_cut(case))
        pos, vel, _ = g.get_particles()
        return [pos, vel, acc]
    s, o = st["solver"], st["out"]
    if kind == "forces":
        s.set_state_device(st["pos"][0], None, st["pos"][1], None)
        s.accel_device(o[2], o[5])
        return [o[2], o[5]]
    if kind == "host":
        s.step_host(*st["host"], case["dt"], HUBBLE, 1.0)
        return st["host"]
    s.step(case["dt"], HUBBLE, 1.0, case["steps"])
    _ok(lib.jt_get_state(s._h, _p(o[0]), _p(o[1]), _p(o[3]), _p(o[4]), J.JT_MEM_DEVICE), "state")
    _ok(lib.jt_get_accel(s._h, _p(o[2]), _p(o[5]), J.JT_MEM_DEVICE), "accel")
    return o


# ---------------------------------------------------------------- work
def _cut(case):
    return J.short_cut(_config(case))


def work(case):
    if case["kind"] == "batch":
        w = [work(b) for b in _batch_boxes(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    n, M = case["n_p"] + case["n_m"], case["M"]
    G = M ** 3
    ref = case["kind"] == "rcompat"
    order = 2 if ref else (case["order"] or 4)
    ng = 1 if ref or case["interlace"] == 2 else 2
    ns = 2 if case["lam"] > 0 else 1
    rc = _rcompat_cut(case) if ref else _cut(case)
    # pairs inside the cut at the mean density (a lower bound for clustered data), 40 flops each
    pairs = n * n / case["L"] ** 3 * 4.0 / 3.0 * math.pi * rc ** 3
    ffts = ns * (2 if ref else 4 * ng)
    flops = 40.0 * pairs + ffts * 2.5 * G * math.log2(G) + ns * ng * n * order ** 3 * (2.0 + 6.0)
    if case["kind"] == "forces":
        return {"bytes": 24.0 * n, "flops": flops}
    if ref:
        return {"bytes": 72.0 * n, "flops": 2.0 * flops}
    # per step: positions, velocities and accelerations read and written once
    return {"bytes": 72.0 * n * case["steps"], "flops": flops * case["steps"]}


def tolerance(case):
    """Accelerations set it (positions and velocities agree to 1e-7).  Against
    exact() the relative error of the accelerations is 1e-5 .. 1.2e-4 on
    lattices and uniform boxes (single-precision FFTs, the pair table and the
    rounding of near-cancelling lattice forces) and up to 2e-4 on clustered
    boxes at theta 0.5 (multipoles; about three times that at 0.7); the same
    inputs twice differ by 1e-7.  The compatibility mode's sums are 32-bit in a
    fixed order."""
    if case["kind"] == "rcompat":
        return {"rel": 1.0e-5, "max": 1.0e-3}
    if case["ic"] == "plummer":
        return {"rel": 3.0e-3 if case["theta"] > 0.6 else 1.0e-3, "max": 0.1}
    return {"rel": 5.0e-4, "max": 0.02}


# ---------------------------------------------------------------- 64-bit result
def _stencil(g, order):
    """First node and weights of the assignment of order 2 (CIC), 3 (TSC), 4 (PCS)."""
    if order == 2:
        f = torch.floor(g)
        t = g - f
        return f.long(), [1 - t, t]
    if order == 3:
        c = torch.floor(g + 0.5)
        d = g - c
        return c.long() - 1, [0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2]
    f = torch.floor(g)
    t = g - f
    s = 1 - t
    return f.long() - 1, [s ** 3 / 6, 2 / 3 - t * t + t ** 3 / 2, 2 / 3 - s * s + s ** 3 / 2, t ** 3 / 6]


def _stencil_terms(pos, L, M, order, shift):
    st = [_stencil((pos[:, a] + 0.5 * L) * (M / L) - shift, order) for a in range(3)]
    for c in range(order):
        for b in range(order):
            w_zy = st[2][1][c] * st[1][1][b]
            row = (torch.remainder(st[2][0] + c, M) * M + torch.remainder(st[1][0] + b, M)) * M
            for a in range(order):
                yield row + torch.remainder(st[0][0] + a, M), w_zy * st[0][1][a]


def _pm_exact(pos, q, L, M, r_s, order, ng, kappa, source):
    """Acceleration of a unit m+ particle from the mesh: the Gaussian-filtered
    Green's function with the assignment deconvolved, spectral gradient,
    interlaced grids.  source 0: the signed source's response, 1: the unsigned
    one's (screened boxes)."""
    h = L / M
    dev = pos.device
    k1 = 2 * math.pi * torch.fft.fftfreq(M, d=h, device=dev, dtype=torch.float64)
    kr = 2 * math.pi * torch.fft.rfftfreq(M, d=h, device=dev, dtype=torch.float64)
    axes = (kr[None, None, :], k1[None, :, None], k1[:, None, None])   # x, y, z
    rho = None
    for g in range(ng):
        grid = torch.zeros(M ** 3, dtype=torch.float64, device=dev)
        for idx, w in _stencil_terms(pos, L, M, order, 0.5 * g):
            grid.index_add_(0, idx, w * q)
        f = torch.fft.rfftn(grid.view(M, M, M) / h ** 3)
        del grid
        if g == 1:
            for k in axes:
                f = f * torch.polar(torch.ones_like(k), -0.5 * h * k)
        rho = f if rho is None else 0.5 * (rho + f)
    k2 = axes[0] ** 2 + axes[1] ** 2 + axes[2] ** 2
    k2[0, 0, 0] = 1.0
    for k in axes:
        u = torch.special.sinc(k * (h / (2 * math.pi)))
        rho = rho * (torch.exp(-k * k * r_s * r_s) / u ** (2 * order))
    green = -4 * math.pi / k2
    if kappa > 0:
        gy = green * (k2 / (k2 + kappa ** 2)) * math.exp(-(kappa * r_s) ** 2)
        green = 0.5 * (green - gy) if source else 0.5 * (green + gy)
    rho = rho * green
    rho[0, 0, 0] = 0.0
    half = M // 2
    rho[half, :, :] = 0.0
    rho[:, half, :] = 0.0
    rho[:, :, half] = 0.0
    acc = torch.zeros_like(pos)
    for g in range(ng):
        ph = rho
        if g == 1:
            for k in axes:
                ph = ph * torch.polar(torch.ones_like(k), 0.5 * h * k)
        for a in range(3):
            field = torch.fft.irfftn(-1j * axes[a] * ph, s=(M, M, M)).reshape(-1)
            for idx, w in _stencil_terms(pos, L, M, order, 0.5 * g):
                acc[:, a] += w * field[idx] / ng
            del field
    return acc


def _short_exact(pos, q, L, r_s, rc, eps, kappa):
    """sum_j s_i s_j m_j S(r_p / 2 r_s) d / r_p^3 over |d| < rc, times s_i left
    out (q = s m): every pair, over a cell list with periodic ghosts."""
    dev = pos.device
    n = len(pos)
    nb = max(1, int(L / rc))
    side = L / nb
    # sources with ghosts one cell around the box
    src, sq = [], []
    for i in (-1, 0, 1):
        for j in (-1, 0, 1):
            for k in (-1, 0, 1):
                p = pos + torch.tensor([i * L, j * L, k * L], dtype=torch.float64, device=dev)
                m = (p.abs() < 0.5 * L + side).all(1) if (i or j or k) else slice(None)
                src.append(p[m])
                sq.append(q[m])
    src, sq = torch.cat(src), torch.cat(sq)
    w = nb + 2
    cell = torch.floor((src + 0.5 * L) / side).long().clamp_(-1, nb) + 1
    key = (cell[:, 2] * w + cell[:, 1]) * w + cell[:, 0]
    key, order = key.sort()
    src, sq = src[order].contiguous(), sq[order].contiguous()
    first = torch.searchsorted(key, torch.arange(w ** 3 + 1, device=dev))
    del key, order, cell
    tc = torch.floor((pos + 0.5 * L) / side).long().clamp_(0, nb - 1) + 1
    acc = torch.zeros(n, 3, dtype=torch.float64, device=dev)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            row = ((tc[:, 2] + dz) * w + tc[:, 1] + dy) * w + tc[:, 0]
            lo, hi = first[row - 1], first[row + 2]
            cnt, by = (hi - lo).sort()
            lo = lo[by]
            cnt_h = cnt.cpu().numpy()
            at = int(np.searchsorted(cnt_h, 1))
            while at < n:
                # as many targets as keep the padded pair matrix at 2^25 entries
                k = max(1, (1 << 25) // max(1, int(cnt_h[min(n - 1, at + 4095)])))
                end = min(n, at + k)
                while int(cnt_h[end - 1]) * (end - at) > (1 << 26) and end - at > 1:
                    end = at + (end - at) // 2
                t = by[at:end]
                cols = torch.arange(int(cnt_h[end - 1]), device=dev)
                ok = cols[None, :] < cnt[at:end, None]
                idx = torch.where(ok, lo[at:end, None] + cols[None, :], 0)
                d = [src[:, a][idx] - pos[t, a][:, None] for a in range(3)]
                r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
                ok &= r2 < rc * rc
                ok &= r2 > 0
                rp2 = r2 + eps * eps
                rp = rp2.sqrt()
                x = rp / (2 * r_s)
                gauss = (2 / math.sqrt(math.pi)) * x * torch.exp(-x * x)
                S = torch.erfc(x) + gauss
                qq = sq[idx]
                if kappa > 0:
                    b = kappa * r_s
                    em, ep = torch.exp(-kappa * rp) * torch.erfc(x - b), torch.exp(kappa * rp) * torch.erfc(x + b)
                    Sy = 0.5 * (em + ep) + b * x * (em - ep) + gauss * math.exp(-b * b)
                    S = torch.where(qq * q[t][:, None] < 0, Sy, S)
                f = torch.where(ok, qq * S / (rp2 * rp), 0.0)
                for a in range(3):
                    acc[t, a] += (f * d[a]).sum(1)
                at = end
    return acc


def _forces_exact(pos, q, case):
    cfg = _config(case)
    order = case["order"] or 4
    ng = 1 if case["interlace"] == 2 else 2
    kappa = 1.0 / case["lam"] if case["lam"] > 0.01 else 0.0
    s = torch.sign(q)[:, None]
    a = s * _short_exact(pos, q, cfg.box_L, cfg.r_s, _cut(case), cfg.softening, kappa)
    a += s * _pm_exact(pos, q, cfg.box_L, cfg.pm_grid, cfg.r_s, order, ng, kappa, 0)
    if kappa > 0:
        a += _pm_exact(pos, q.abs(), cfg.box_L, cfg.pm_grid, cfg.r_s, order, ng, kappa, 1)
    return a


def _exact_box(case, seed):
    x = [a.double() for a in _inputs(case, seed)]
    L, n_p, n_m = case["L"], case["n_p"], case["n_m"]
    m_p = _config(case).G_mass_plus
    m_m = case["mu"] * m_p * n_p / n_m
    q = torch.cat([torch.full((n_p,), m_p, dtype=torch.float64, device=DEVICE),
                   torch.full((n_m,), -m_m, dtype=torch.float64, device=DEVICE)])
    pos, vel = torch.cat([x[0], x[2]]), torch.cat([x[1], x[3]])
    a = _forces_exact(pos, q, case)
    if case["kind"] == "forces":
        return [a[:n_p], a[n_p:]]
    h = 0.5 * case["dt"]
    for _ in range(case["steps"]):
        vel = vel + (a - HUBBLE * vel) * h
        pos = _wrap(pos + vel * case["dt"], L)
        a = _forces_exact(pos, q, case)
        vel = vel + (a - HUBBLE * vel) * h
    return [pos[:n_p], vel[:n_p], a[:n_p], pos[n_p:], vel[n_p:], a[n_p:]]


def exact(case, seed):
    if case["kind"] == "rcompat":
        return None   # defined by the reference's own single-precision formulas and walk order
    if case["kind"] == "batch":
        boxes = [_exact_box(b, seed * 1000 + i) for i, b in enumerate(_batch_boxes(case))]
        return [torch.cat([b[k] for b in boxes]) for k in range(6)]
    if case["ic"] == "plummer" and case["n_p"] > 80 ** 3:
        return None   # direct pairs inside the clumps: minutes
    return _exact_box(case, seed)
