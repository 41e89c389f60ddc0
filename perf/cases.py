"""Performance cases: the work a user has this framework do, through its public entry points.

Every case is one call pattern of the host API (`llg-sim_b200/llg_b200.py`) on films, hierarchies
or training batches of the sizes and materials of `workloads.py`, `sp4.py`, `bench.py` and the tests.
`exact` restates a pass in FP64 with plain torch / numpy: the demag kernel by the face-charge
integration, zero-padded FFT convolution, the local terms with their ghost rules, the steppers.

Integrator cases cap the step size (dt_max), as a run sampled at fixed times does, where the
error-limited step is longer than the cap: the number of steps, and so the work, is then given.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "llg-sim_b200"))

import llg_b200 as L  # noqa: E402
import workloads as W  # noqa: E402

GAMMA = W.GAMMA
MU0 = 4.0 * math.pi * 1e-7

# Materials of the repository's workloads: Ms, A, Ku (+z), D, alpha, cell, m0.
#  dmi: the 1024x1024 benchmark film (random m0); soft: the mixed batch and the 128x32 flow;
#  sp4: the standard-problem-4 film; holey: the warm-start films (Ms 8e5, D 0..2e-3, holes).
MATERIALS = {
    "dmi": dict(ms=5.8e5, a=1.5e-11, ku=8e5, dmi=3e-3, alpha=0.3, cell=(2e-9, 2e-9, 2e-9), b=(0.0, 0.0, 0.0)),
    "soft": dict(ms=8e5, a=1.3e-11, ku=0.0, dmi=None, alpha=0.02, cell=(4e-9, 4e-9, 3e-9), b=(0.012, 0.016, 0.0)),
    "sp4": dict(ms=8e5, a=1.3e-11, ku=0.0, dmi=None, alpha=0.02, cell=(2.5e-9, 2.5e-9, 3e-9),
                b=(-24.6e-3, 4.3e-3, 0.0)),
    "holey": dict(ms=8e5, a=1.3e-11, ku=0.0, dmi=1e-3, alpha=0.5, cell=(4e-9, 4e-9, 3e-9), b=(0.01, -0.005, 0.0)),
}


def listed():
    return [
        # one host-driven adaptive step with the state passed in and out (the drop-in binding of
        # step(&mut m, ...)): the smallest call, launches and latency count
        dict(name="step_128x32_f64", kind="step", nx=128, ny=32, mat="soft", f64=True, dt=2e-13),
        # a sample window of the SP4 driver on its 200x50 film (no power of two in either direction)
        dict(name="window_200x50_f32", kind="window", nx=200, ny=50, mat="sp4", f64=False, dt=8e-14, steps=60,
             random=False),
        # the benchmark film: random start, adaptive steps, until a given time
        dict(name="window_1024x1024_f32", kind="window", nx=1024, ny=1024, mat="dmi", f64=False, dt=3e-14, steps=40,
             random=True),
        # a double-precision run of a mid-sized film
        dict(name="window_512x256_f64", kind="window", nx=512, ny=256, mat="soft", f64=True, dt=2e-13, steps=25,
             random=False),
        # parameter sweep: films of mixed sizes and materials advanced together
        dict(name="batch_64_f32", kind="batch", n=64, f64=False, dt=2e-13, steps=20),
        # relaxation of holey films with random start (energy descent, RK23 with torque sums)
        dict(name="relax_16x128_f32", kind="relax", n=16, size=128, f64=False, dt=2e-14, steps=45),
        # damping-only minimiser on a square film
        dict(name="minimize_256x256_f32", kind="minimize", nx=256, ny=256, mat="dmi", f64=False, iters=60),
        # field, energy and torque of a given state: post-processing of a ragged film in double precision
        dict(name="field_250x125_f64", kind="field", nx=250, ny=125, mat="dmi", f64=True),
        # demag field on device arrays inside another framework's loop
        dict(name="demag_dev_1000x400_f32", kind="demag_dev", nx=1000, ny=400),
        # AMR with the flattened fine grid (8x the 192x192 base), on device arrays
        dict(name="allfft_1536x1536_f64", kind="allfft", nx=192, ny=192, ratio=8, masked=False),
        # AMR with the coarse-FFT demag, hierarchy on the host
        dict(name="coarse_192x192_f64", kind="coarse", nx=192, ny=192),
        # one backward pass of the warm-start network on a minibatch of 128x128 films
        dict(name="train_16x128_bf16", kind="train", n=16, size=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """A film side: a power of two (the usual choice), a round number, or (up to 200 cells) any length."""
    v, r = _log_int(rng, lo, hi), rng.random()
    if r < 0.4:
        v = 1 << int(round(math.log2(v)))
    elif r < 0.8 or v > 200:
        q = 20 if v > 200 else 5
        v = q * int(round(v / q))
    return min(max(v, lo), hi)


def draw(rng):
    kind = rng.choice(["step", "window", "window", "window", "batch", "relax", "minimize", "field", "demag_dev",
                       "allfft", "coarse", "train"])
    f64 = rng.random() < 0.4
    if kind == "step":
        return dict(kind=kind, nx=_side(rng, 16, 256), ny=_side(rng, 16, 128), mat="soft", f64=f64, dt=2e-13)
    if kind == "window":
        nx, ny = _side(rng, 32, 1024), _side(rng, 16, 1024)
        mat = rng.choice(["soft", "sp4"])
        return dict(kind=kind, nx=nx, ny=ny, mat=mat, f64=f64, dt=2e-13 if mat == "soft" else 8e-14,
                    steps=rng.randint(10, 30), random=False)
    if kind == "batch":
        return dict(kind=kind, n=_log_int(rng, 4, 64), f64=f64, dt=2e-13, steps=rng.randint(8, 20))
    if kind == "relax":
        return dict(kind=kind, n=_log_int(rng, 1, 16), size=rng.choice([64, 96, 100, 128, 150]), f64=f64, dt=2e-14,
                    steps=3 * rng.randint(5, 15))
    if kind == "minimize":
        return dict(kind=kind, nx=_side(rng, 32, 512), ny=_side(rng, 32, 512), mat="dmi", f64=f64,
                    iters=rng.randint(20, 60))
    if kind == "field":
        return dict(kind=kind, nx=_side(rng, 32, 512), ny=_side(rng, 16, 512), mat=rng.choice(["dmi", "soft", "sp4"]),
                    f64=f64)
    if kind == "demag_dev":
        return dict(kind=kind, nx=_side(rng, 64, 1024), ny=_side(rng, 64, 1024))
    if kind == "allfft":
        n = rng.choice([64, 80, 96, 100, 128])
        return dict(kind=kind, nx=n, ny=rng.choice([48, 64, 96, 100]), ratio=rng.choice([4, 8]),
                    masked=rng.random() < 0.5)
    if kind == "coarse":
        return dict(kind=kind, nx=rng.choice([128, 160, 192, 200, 256]), ny=rng.choice([128, 150, 192, 256]))
    return dict(kind=kind, n=_log_int(rng, 2, 16), size=rng.choice([64, 96, 128]))


# ------------------------------------------------------------------ inputs


def _film(case):
    m = MATERIALS[case["mat"]]
    dx, dy, dz = m["cell"]
    return L.Grid2D(case["nx"], case["ny"], dx, dy, dz), L.Material(m["ms"], m["a"], m["ku"], (0, 0, 1), m["dmi"], True)


def _m0(n, seed, random):
    if random:
        return L.init_random(n, seed + 1)
    return L.init_uniform_with_noise(n, (1.0, 0.1, 0.05), 0.1, seed + 1)


def _prec(case):
    return L.FP64 if case["f64"] else L.FP32


def _batch_films(case, seed):
    """Sizes by the case alone; materials and fields by the seed."""
    films = W.mixed_film_batch(n=case["n"], seed=seed + 4)[0]
    for f, g in zip(films, W.mixed_film_batch(n=case["n"], seed=3)[0]):
        f.nx, f.ny = g.nx, g.ny
    return films


def _holey_films(case, seed):
    films = W.holey_film_batch(case["n"], size=case["size"], seed=seed + 5)[0]
    for i, f in enumerate(films):
        f.m0 = L.init_random(f.n, (seed + 5) * 1000 + i)
        f.m0[f.mask == 0] = 0.0
    return films


def _train_inputs(case, seed):
    """Random start, a smooth target of unit vectors, disk holes and in-plane fields, He-scaled weights."""
    rng = np.random.default_rng(seed + 17)
    n, s = case["n"], case["size"]
    films = W.holey_film_batch(n, size=s, seed=seed + 5)[0]
    mask = np.stack([f.mask for f in films]).astype(np.uint8)
    m0 = rng.standard_normal((n, 3, s * s))
    m0 *= mask[:, None] / np.linalg.norm(m0, axis=1, keepdims=True)
    X, Y = np.meshgrid(np.arange(s) / s, np.arange(s) / s)
    ph = rng.uniform(0, 2 * math.pi, (n, 1))
    a = (2 * math.pi * X.reshape(1, -1) + ph, 2 * math.pi * Y.reshape(1, -1) - ph)
    tgt = np.stack([np.cos(a[0]) * np.cos(a[1]), np.sin(a[0]) * np.cos(a[1]), np.sin(a[1])], axis=1)
    bext = np.array([f.b_ext for f in films])
    params = []
    for ci, co in L.WarmStartNet.LAYERS:
        params.append(rng.normal(0.0, math.sqrt(2.0 / (9 * ci)), co * 9 * ci))
        params.append(np.zeros(co))
    return (np.concatenate(params).astype(np.float32), m0.astype(np.float32), mask, bext,
            (tgt * mask[:, None]).astype(np.float32))


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).pin_memory()


def _single(case, seed):
    g, mat = _film(case)
    m0 = _pinned(_m0(g.n_cells(), seed, case.get("random", case["kind"] in ("minimize", "field"))))
    s = L.Solver(g, mat, _prec(case))
    return dict(case=case, s=s, m0=m0, out=torch.empty_like(m0).pin_memory())


def _batch(case, films):
    b = L.Batch([f.grid(L) for f in films], [f.material(L) for f in films], _prec(case),
                masks=[f.mask for f in films] if films[0].mask is not None else None)
    return dict(case=case, b=b, films=films)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "window", "minimize", "field"):
        return _single(case, seed)
    if kind == "batch":
        films = _batch_films(case, seed)
        for i, f in enumerate(films):
            f.m0 = L.init_uniform_with_noise(f.n, (1.0, 0.0, 0.0), 0.1, seed + 1 + i)
        return _batch(case, films)
    if kind == "relax":
        return _batch(case, _holey_films(case, seed))
    if kind == "demag_dev":
        m = MATERIALS["soft"]
        nx, ny = case["nx"], case["ny"]
        g = L.Grid2D(nx, ny, *m["cell"])
        s = L.Solver(g, L.Material(m["ms"], m["a"], demag=True), L.FP32)
        planes = torch.from_numpy(s.kernel_kspace()).cuda()
        s.close()
        m0 = torch.from_numpy(_m0(nx * ny, seed, False)).float().cuda().reshape(ny, nx, 3).permute(2, 0, 1)
        return dict(case=case, m=m0.contiguous(), planes=planes, b=torch.empty(3, ny, nx, device="cuda"))
    if kind == "allfft":
        base = L.Grid2D(case["nx"], case["ny"], 4e-9, 4e-9, 3e-9)
        r = case["ratio"]
        fine = L.Grid2D(base.nx * r, base.ny * r, base.dx / r, base.dy / r, base.dz)
        m, mask = _fine_state(case, seed)
        d = dict(case=case, base=base, op=L.DemagOp(fine), mat=L.Material(8e5, 1.3e-11, demag=True),
                 m=torch.from_numpy(m).cuda(), mask=None if mask is None else torch.from_numpy(mask).cuda())
        d["bf"] = torch.empty_like(d["m"])
        d["bc"] = torch.empty(base.nx * base.ny, 3, dtype=torch.float64, device="cuda")
        return d
    if kind == "coarse":
        base = L.Grid2D(case["nx"], case["ny"], 4e-9, 4e-9, 3e-9)
        mc, ps = W.amr_vortex_hierarchy(case["nx"], case["ny"], seed=seed + 13)
        patches = [L.AmrPatch(p.i0, p.j0, p.cnx, p.cny, p.ratio, p.ghost, p.m) for p in ps]
        return dict(case=case, h=L.AmrDemag(base), mat=L.Material(8e5, 1.3e-11, demag=True), mc=mc, patches=patches)
    params, m0, mask, bext, tgt = _train_inputs(case, seed)
    s = case["size"]
    up = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    return dict(case=case, t=L.WarmStartTrainer(params, case["n"] * s * s), m0=up(m0), mask=up(mask), bext=up(bext),
                tgt=up(tgt))


def _fine_state(case, seed):
    nx, ny = case["nx"] * case["ratio"], case["ny"] * case["ratio"]
    dx = 4e-9 / case["ratio"]
    rng = np.random.default_rng(seed + 23)
    m = W.amr_fine_vortex(nx, ny, dx, dx) + 0.02 * rng.standard_normal((nx * ny, 3))
    m /= np.linalg.norm(m, axis=1, keepdims=True)
    if not case["masked"]:
        return m, None
    mask = W.disk_holes_mask(nx, ny, dx, dx, [(0.2 * nx * dx, 0.1 * ny * dx, 0.15 * ny * dx)]).astype(np.uint8)
    return m * mask[:, None], mask


# ------------------------------------------------------------------ one pass


def _params(case):
    m = MATERIALS[case["mat"]]
    return L.LLGParams(GAMMA, m["alpha"], case.get("dt", 1e-13), m["b"])


def _film_params(case, films):
    return [L.LLGParams(GAMMA, f.alpha, case["dt"], f.b_ext) for f in films]


def _own_precision(case, m):
    """A state or field at the film's own precision (the host arrays are double for both)."""
    return m if case["f64"] else m.float()


def _minimize_settings(case):
    return L.MinimizeSettings.default(max_iters=case["iters"], torque_threshold=0.0, dm_stop=None, lambda0=2e-4,
                                      lambda_min=1e-5, lambda_max=1e-3, stall_iters=10 ** 9)


def _relax_settings(case):
    return L.RelaxSettings.default(torque_threshold=1e-6, max_err=1e-3, headroom=0.8, dt_min=1e-18,
                                   dt_max=case["dt"], max_accepted_steps=case["steps"])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "window", "minimize", "field"):
        s = state["s"]
        p = _params(case)
        s.set_state_ptr(state["m0"].data_ptr())
        if kind == "field":
            b = torch.from_numpy(s.build_h_eff(p, L.FULL))
            e = s.compute_energy(p.b_ext)
            return dict(b=_own_precision(case, b), torque=s.torque_metric(p, L.FULL, L.TORQUE_RMS),
                        energy=[e.exchange, e.anisotropy, e.zeeman, e.dmi, e.demag]) if case["f64"] else dict(
                            b=_own_precision(case, b),
                            torque=np.float32(s.torque_metric(p, L.FULL, L.TORQUE_RMS)),
                            energy=np.float32([e.exchange, e.anisotropy, e.zeeman, e.dmi, e.demag]))
        if kind == "step":
            s.step_rk45(p, L.FULL, 1e-5, 0.8, 1e-18, case["dt"])
        elif kind == "window":
            s.run_rk45(p, L.FULL, 1e-5, 0.8, 1e-18, case["dt"] if not case["random"] else 1e-11,
                       t_end=case["steps"] * case["dt"])
        else:
            s.minimize(p, L.FULL, _minimize_settings(case))
        s.get_state_ptr(state["out"].data_ptr())
        return _own_precision(case, state["out"])
    if kind in ("batch", "relax"):
        b, films = state["b"], state["films"]
        for i, f in enumerate(films):
            b.set_state(i, f.m0)
        P = _film_params(case, films)
        if kind == "batch":
            b.run_rk45(P, L.FULL, 1e-5, 0.8, 1e-18, case["dt"], t_end=case["steps"] * case["dt"])
        else:
            b.relax(P, L.FULL, _relax_settings(case))
        return [_own_precision(case, torch.from_numpy(b.get_state(i))) for i in range(len(films))]
    if kind == "demag_dev":
        L.demag_field_noalloc(case["nx"], case["ny"], MATERIALS["soft"]["ms"], state["m"].data_ptr(),
                              state["planes"].data_ptr(), state["b"].data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
        return state["b"]
    if kind == "allfft":
        mask = state["mask"]
        L.allfft_demag_device(state["op"], state["mat"], state["m"].data_ptr(), 0 if mask is None else mask.data_ptr(),
                              state["base"], state["bf"].data_ptr(), state["bc"].data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
        return dict(bf=state["bf"], bc=state["bc"])
    if kind == "coarse":
        bc, bp = state["h"].compute(state["mat"], state["mc"], state["patches"])
        return dict(bc=bc, bp=bp)
    s = case["size"]
    loss, grad = state["t"].gradients(case["n"], s, s, state["m0"].data_ptr(), state["mask"].data_ptr(),
                                      state["bext"].data_ptr(), state["tgt"].data_ptr())
    return dict(loss=np.float32(loss), grad=grad)


# ------------------------------------------------------------------ work


def _eval_flops(nx, ny):
    """One field evaluation: pruned 2-D transforms of 3 real components there and back, kernel
    product, local terms and torque."""
    row = 2 * 1.5 * 2 * ny * 5.0 * nx * math.log2(max(nx, 2))
    col = 12 * (nx + 1) * 5.0 * ny * math.log2(max(ny, 2))
    return row + col + 2 * (nx + 1) * ny * 20.0 + 120.0 * nx * ny


def _film_bytes(nx, ny, w):
    """State in and out on the host (double), kernel spectrum in."""
    return 48.0 * nx * ny + 4.0 * w * (nx + 1) * (ny + 1)


def work(case):
    kind = case["kind"]
    w = 8 if case.get("f64", kind in ("allfft", "coarse")) else 4
    if kind in ("step", "window", "minimize", "field"):
        nx, ny = case["nx"], case["ny"]
        evals = {"step": 7, "field": 3}.get(kind) or (case["iters"] if kind == "minimize" else 6 * case["steps"] + 1)
        return dict(bytes=_film_bytes(nx, ny, w), flops=evals * _eval_flops(nx, ny))
    if kind in ("batch", "relax"):
        if kind == "relax":
            sizes, evals = [(case["size"], case["size"])] * case["n"], 3 * case["steps"] + case["steps"] // 3 + 1
        else:
            sizes, evals = [(f.nx, f.ny) for f in _batch_films(case, 0)], 6 * case["steps"] + 1
        return dict(bytes=sum(_film_bytes(x, y, w) for x, y in sizes),
                    flops=sum(evals * _eval_flops(x, y) for x, y in sizes))
    nx, ny = case.get("nx", 0), case.get("ny", 0)
    if kind == "demag_dev":
        return dict(bytes=24.0 * nx * ny + 32.0 * (nx + 1) * (ny + 1), flops=_eval_flops(nx, ny))
    if kind == "allfft":
        r = case["ratio"]
        return dict(bytes=48.0 * nx * ny * r * r + 32.0 * (nx * r + 1) * (ny * r + 1) + 24.0 * nx * ny,
                    flops=_eval_flops(nx * r, ny * r))
    if kind == "coarse":
        cells = sum(p.pnx * p.pny for p in W.amr_vortex_hierarchy(nx, ny)[1])
        return dict(bytes=48.0 * (nx * ny + cells) + 32.0 * (nx + 1) * (ny + 1), flops=_eval_flops(nx, ny))
    cells = case["n"] * case["size"] ** 2
    per = sum(2.0 * 9 * ci * co for ci, co in L.WarmStartNet.LAYERS)
    return dict(bytes=cells * 25.0, flops=3 * per * cells)


# ------------------------------------------------------------------ FP64 restatement


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _unit(v):
    n = (v * v).sum(0).sqrt()
    z = torch.zeros_like(v)
    z[2] = 1.0
    return torch.where(n > 0, v / torch.where(n > 0, n, torch.ones_like(n)), z)


def _count(x):
    return np.floor(np.maximum(x, 1.0) + 0.5).astype(np.int64)


def _quadrant(nx, ny, cell):
    """Face-charge integration of mu0 N for displacements 0..nx-1, 0..ny-1: [4, ny, nx] (xx, xy, yy, zz)."""
    cell = np.asarray(cell, dtype=np.float64)
    sx, sy = np.meshgrid(np.arange(nx), np.arange(ny))
    ax, ay = np.maximum(sx - 1, 0) * cell[0], np.maximum(sy - 1, 0) * cell[1]
    d = np.sqrt(ax * ax + ay * ay)
    d[d == 0] = cell.min()
    ms = d / 10.0
    cnt = np.stack([_count(cell[k] / ms) for k in range(3)], -1).reshape(-1, 3)
    keys, inv = np.unique(cnt, axis=0, return_inverse=True)
    inv = inv.reshape(-1)
    out = torch.zeros(4, ny * nx, dtype=torch.float64, device="cuda")
    centre = np.stack([sx.reshape(-1) * cell[0], sy.reshape(-1) * cell[1], np.zeros(nx * ny)], 1)

    def points(n, c):
        return -0.5 * c + c / (2.0 * n) + np.arange(n) * (c / n)

    for k, key in enumerate(keys):
        ids = np.nonzero(inv == k)[0]
        obs = np.stack(np.meshgrid(*[points(int(key[q]), cell[q]) for q in range(3)], indexing="ij"), -1).reshape(-1, 3)
        for u, take in ((0, ((0, 0),)), (1, ((1, 0), (2, 1))), (2, ((3, 2),))):
            v, w = (u + 1) % 3, (u + 2) % 3
            nv, nw = 2 * int(key[v]), 2 * int(key[w])
            face = np.zeros((nv * nw, 3))
            pv, pw = np.meshgrid(points(nv, cell[v]), points(nw, cell[w]), indexing="ij")
            face[:, v], face[:, w] = pv.reshape(-1), pw.reshape(-1)
            dif = torch.from_numpy((obs[:, None] - face[None]).reshape(-1, 3)).cuda()
            q = cell[v] * cell[w] / dif.shape[0] / (4.0 * math.pi)
            step = max(1, (1 << 24) // dif.shape[0])
            for a in range(0, len(ids), step):
                part = torch.from_numpy(ids[a:a + step]).cuda()
                r = torch.from_numpy(centre[ids[a:a + step]]).cuda()[:, None] + dif[None]
                h = 0.0
                for sgn in (1.0, -1.0):
                    rr = r.clone()
                    rr[..., u] -= sgn * 0.5 * cell[u]
                    n2 = (rr * rr).sum(-1, keepdim=True)
                    h = h + (sgn * q * rr / (n2 * n2.sqrt())).sum(1)
                for row, comp in take:
                    out[row, part] = MU0 * h[:, comp]
    return out.reshape(4, ny, nx)


class _Demag:
    def __init__(self, nx, ny, cell, ms):
        q = _quadrant(nx, ny, cell)
        K = torch.zeros(4, 2 * ny, 2 * nx, dtype=torch.float64, device="cuda")
        K[:, :ny, :nx] = q
        K[:, :ny, nx + 1:] = q[:, :, 1:].flip(2)
        K[:, ny + 1:, :nx] = q[:, 1:].flip(1)
        K[:, ny + 1:, nx + 1:] = q[:, 1:, 1:].flip(1, 2)
        K[1, :ny, nx + 1:] *= -1
        K[1, ny + 1:, :nx] *= -1
        K[1, 0], K[1, :, 0] = 0.0, 0.0
        self.k, self.nx, self.ny, self.ms = torch.fft.rfft2(K).real, nx, ny, ms

    def __call__(self, m):
        f = torch.fft.rfft2(self.ms * m, s=(2 * self.ny, 2 * self.nx))
        k = self.k
        b = torch.stack([k[0] * f[0] + k[1] * f[1], k[1] * f[0] + k[2] * f[1], k[3] * f[2]])
        return torch.fft.irfft2(b, s=(2 * self.ny, 2 * self.nx))[:, :self.ny, :self.nx]


class _Film:
    """Effective field, torques and steppers of one film; m [3, ny, nx] FP64."""

    def __init__(self, nx, ny, cell, ms, a, ku, dmi, b, alpha, mask=None, demag=None):
        self.nx, self.ny, self.cell, self.ms, self.a, self.ku, self.alpha = nx, ny, cell, ms, a, ku, alpha
        self.d = 0.0 if dmi is None else dmi
        self.b = torch.tensor(b, dtype=torch.float64, device="cuda").reshape(3, 1, 1)
        self.mask = None if mask is None else torch.from_numpy(np.asarray(mask).reshape(ny, nx) != 0).cuda()
        self.demag = demag or _Demag(nx, ny, cell, ms)

    def neighbour(self, m, dim, sgn, vacuum_ghost):
        """m of the neighbour at +-1 along x (dim 2) or y (dim 1): a chiral ghost at film edges, and at
        vacuum cells either a chiral ghost (exchange) or a copy of the centre (DMI)."""
        n = m.shape[dim]
        t = torch.roll(m, -sgn, dim)
        edge = torch.zeros(m.shape[1:], dtype=torch.bool, device="cuda")
        edge.select(dim - 1, n - 1 if sgn > 0 else 0)[:] = True
        ghost = m.clone()
        eta, comp, h = self.d / (2.0 * self.a), (0 if dim == 2 else 1), self.cell[0 if dim == 2 else 1]
        if n > 1:
            ghost[comp] = m[comp] - sgn * h * eta * m[2]
            ghost[2] = m[2] + sgn * h * eta * m[comp]
        t = torch.where(edge, ghost, t)
        if self.mask is not None:
            vac = ~torch.roll(self.mask, -sgn, dim - 1) & ~edge
            t = torch.where(vac, ghost if vacuum_ghost else m, t)
        return t

    def local(self, m):
        b = self.b.expand_as(m).clone()
        inside = 1.0 if self.mask is None else self.mask.double()
        ex = 0.0
        for dim, h in ((2, self.cell[0]), (1, self.cell[1])):
            if m.shape[dim] > 1:
                ex = ex + (self.neighbour(m, dim, 1, True) - 2 * m + self.neighbour(m, dim, -1, True)) / (h * h)
        b = b + 2 * self.a / self.ms * ex * inside
        b[2] += 2 * self.ku / self.ms * m[2]
        if self.d:
            b = b + self.dmi_field(m, False) * inside
        return b

    def dmi_field(self, m, vacuum_ghost):
        pref, dx, dy = 2 * self.d / self.ms, 2 * self.cell[0], 2 * self.cell[1]
        gx = (self.neighbour(m, 2, 1, vacuum_ghost) - self.neighbour(m, 2, -1, vacuum_ghost)) / dx
        gy = (self.neighbour(m, 1, 1, vacuum_ghost) - self.neighbour(m, 1, -1, vacuum_ghost)) / dy
        if m.shape[2] == 1:
            gx = torch.zeros_like(gx)
        if m.shape[1] == 1:
            gy = torch.zeros_like(gy)
        return pref * torch.stack([gx[2], gy[2], -(gx[0] + gy[1])])

    def field(self, m):
        return self.local(m) + self.demag(m)

    def energy(self, m):
        v = self.cell[0] * self.cell[1] * self.cell[2]
        ex = ((m[:, :, 1:] - m[:, :, :-1]) ** 2).sum() / self.cell[0] ** 2
        ex = ex + ((m[:, 1:] - m[:, :-1]) ** 2).sum() / self.cell[1] ** 2
        dm = self.dmi_field(m, True) if self.d else torch.zeros_like(m)
        return [float(self.a * ex * v), float(self.ku * (1 - m[2] ** 2).sum() * v),
                float(-self.ms * (m * self.b).sum() * v), float(-0.5 * self.ms * (m * dm).sum() * v),
                float(-0.5 * self.ms * (m * self.demag(m)).sum() * v)]

    def rhs(self, m, relax=False):
        t = _cross(m, self.field(m))
        pref = -GAMMA / (1 + self.alpha ** 2)
        return pref * self.alpha * _cross(m, t) if relax else pref * (t + self.alpha * _cross(m, t))

    def norm(self, m):
        m = _unit(m)
        return m if self.mask is None else torch.where(self.mask, m, torch.zeros_like(m))

    def rk45(self, m, dt, dt_max, t_end, max_err=1e-5, headroom=0.8, dt_min=1e-18, attempts=None):
        A = ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
             (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
             (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
             (35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
        E = (35 / 384 - 5179 / 57600, 0, 500 / 1113 - 7571 / 16695, 125 / 192 - 393 / 640,
             -2187 / 6784 + 92097 / 339200, 11 / 84 - 187 / 2100, -1 / 40)
        t, n = 0.0, 0
        k1 = self.rhs(m)
        dt = min(dt, t_end)
        while t + 1e-18 < t_end and (attempts is None or n < attempts):
            k, x = [k1], m
            for row in A:
                x = self.norm(m + sum(dt * c * q for c, q in zip(row, k) if c))
                k.append(self.rhs(x))
            eps = float(sum(c * q for c, q in zip(E, k) if c).abs().max()) * dt
            if eps <= max_err or dt <= dt_min * 1.0000000001:
                m, k1, t = x, k[6], t + dt
            dt = dt * headroom * (max_err / eps) ** 0.2 if eps > 0 else 2 * dt
            dt = min(max(dt, dt_min), dt_max, t_end - t if t_end > t else dt_max)
            n += 1
        return m

    def rk23_relax(self, m, dt, steps):
        k1 = self.rhs(m, True)
        for _ in range(steps):
            k2 = self.rhs(self.norm(m + dt / 2 * k1), True)
            k3 = self.rhs(self.norm(m + dt * 3 / 4 * k2), True)
            m = self.norm(m + dt * (2 / 9 * k1 + 1 / 3 * k2 + 4 / 9 * k3))
            k1 = self.rhs(m, True)
        return m

    def minimize(self, m, st):
        lam, prev = st.lambda0, math.inf
        for _ in range(st.max_iters):
            q = _cross(m, self.field(m))
            mean = float((q * q).sum(0).sqrt().mean())
            m = self.norm(m + lam * _cross(q, m))
            lam = min(lam * st.grow, st.lambda_max) if mean < prev else max(lam * st.shrink, st.lambda_min)
            prev = mean
        return m


def _planes(m, nx, ny):
    return torch.from_numpy(np.ascontiguousarray(m)).cuda().reshape(ny, nx, 3).permute(2, 0, 1).contiguous()


def _aos(m):
    return m.permute(1, 2, 0).reshape(-1, 3).cpu()


def _bilinear(f, dx, dy, x, y):
    """Bilinear samples of f [ny, nx, 3] (cell centres at (i + 0.5) dx) at points x, y."""
    ny, nx = f.shape[:2]
    fx, fy = x / dx - 0.5, y / dy - 0.5
    i, j = np.floor(fx), np.floor(fy)
    tx, ty = (fx - i)[:, None], (fy - j)[:, None]
    i0, i1 = np.clip(i, 0, nx - 1).astype(int), np.clip(i + 1, 0, nx - 1).astype(int)
    j0, j1 = np.clip(j, 0, ny - 1).astype(int), np.clip(j + 1, 0, ny - 1).astype(int)
    return (f[j0, i0] * (1 - tx) + f[j0, i1] * tx) * (1 - ty) + (f[j1, i0] * (1 - tx) + f[j1, i1] * tx) * ty


def _centres(nx, ny, dx, dy):
    X, Y = np.meshgrid((np.arange(nx) + 0.5) * dx, (np.arange(ny) + 0.5) * dy)
    return X.reshape(-1), Y.reshape(-1)


def _exact_film(case):
    m = MATERIALS[case["mat"]]
    return _Film(case["nx"], case["ny"], m["cell"], m["ms"], m["a"], m["ku"], m["dmi"], m["b"], m["alpha"])


def _exact_train(case, seed):
    params, m0, mask, bext, tgt = _train_inputs(case, seed)
    s, n = case["size"], case["n"]
    p = torch.from_numpy(params).double().cuda().requires_grad_()
    inside = torch.from_numpy(mask).double().cuda().reshape(n, 1, s, s)
    x = torch.cat([torch.from_numpy(m0).double().cuda().reshape(n, 3, s, s) * inside, inside,
                   (torch.from_numpy(bext).cuda() / 0.05).reshape(n, 3, 1, 1).expand(n, 3, s, s)], 1)
    o = 0
    for i, (ci, co) in enumerate(L.WarmStartNet.LAYERS):
        w = p[o:o + co * 9 * ci].reshape(co, 3, 3, ci).permute(0, 3, 1, 2)
        o += co * 9 * ci
        x = torch.nn.functional.conv2d(x, w, p[o:o + co], padding=1)
        o += co
        if i < 5:
            x = torch.relu(x)
    u = x / x.norm(dim=1, keepdim=True)
    t = torch.from_numpy(tgt).double().cuda().reshape(n, 3, s, s)
    loss = ((1 - (u * t).sum(1, keepdim=True)) * inside).sum() / inside.sum()
    loss.backward()
    return dict(loss=float(loss.detach()), grad=p.grad.cpu())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "window", "minimize", "field"):
        f = _exact_film(case)
        m = _planes(_m0(f.nx * f.ny, seed, case.get("random", kind in ("minimize", "field"))), f.nx, f.ny)
        if kind == "field":
            b = f.field(m)
            return dict(b=_aos(b), energy=f.energy(m), torque=float((_cross(m, b) ** 2).sum(0).mean().sqrt())) \
                if case["f64"] else dict(b=_aos(b), energy=np.array(f.energy(m)),
                                         torque=float((_cross(m, b) ** 2).sum(0).mean().sqrt()))
        if kind == "step":
            return _aos(f.rk45(m, case["dt"], case["dt"], math.inf, attempts=1))
        if kind == "window":
            return _aos(f.rk45(m, case["dt"], 1e-11 if case["random"] else case["dt"], case["steps"] * case["dt"]))
        return _aos(f.minimize(m, _minimize_settings(case)))
    if kind in ("batch", "relax"):
        films = _batch_films(case, seed) if kind == "batch" else _holey_films(case, seed)
        out, ops = [], {}
        for i, f in enumerate(films):
            if kind == "batch":
                f.m0 = L.init_uniform_with_noise(f.n, (1.0, 0.0, 0.0), 0.1, seed + 1 + i)
            key = (f.nx, f.ny)
            ops[key] = ops.get(key) or _Demag(f.nx, f.ny, (f.dx, f.dy, f.dz), 1.0)
            x = _Film(f.nx, f.ny, (f.dx, f.dy, f.dz), f.ms, f.a_ex, f.k_u, f.dmi, f.b_ext, f.alpha, f.mask,
                      lambda m, op=ops[key], ms=f.ms: ms * op(m))
            m = _planes(f.m0, f.nx, f.ny)
            m = x.rk45(m, case["dt"], case["dt"], case["steps"] * case["dt"]) if kind == "batch" else \
                x.rk23_relax(m, case["dt"], case["steps"])
            out.append(_aos(m))
        return out
    nx, ny = case.get("nx"), case.get("ny")
    if kind == "demag_dev":
        m = MATERIALS["soft"]
        m0 = torch.from_numpy(_m0(nx * ny, seed, False)).float().double().cuda().reshape(ny, nx, 3).permute(2, 0, 1)
        return _Demag(nx, ny, m["cell"], m["ms"])(m0).contiguous()
    if kind == "allfft":
        r = case["ratio"]
        m, mask = _fine_state(case, seed)
        b = _Demag(nx * r, ny * r, (4e-9 / r, 4e-9 / r, 3e-9), 8e5)(_planes(m, nx * r, ny * r))
        bf = _aos(b).numpy() if mask is None else _aos(b).numpy() * mask[:, None]
        x, y = _centres(nx, ny, 4e-9, 4e-9)
        return dict(bf=bf, bc=_bilinear(bf.reshape(ny * r, nx * r, 3), 4e-9 / r, 4e-9 / r, x, y))
    if kind == "coarse":
        mc, ps = W.amr_vortex_hierarchy(nx, ny, seed=seed + 13)
        e = mc.reshape(ny, nx, 3).copy()
        for p in ps:
            g, r = p.ghost, p.ratio
            inner = p.m.reshape(p.pny, p.pnx, 3)[g:p.pny - g, g:p.pnx - g]
            e[p.j0:p.j0 + p.cny, p.i0:p.i0 + p.cnx] = inner.reshape(p.cny, r, p.cnx, r, 3).mean((1, 3))
        b = _aos(_Demag(nx, ny, (4e-9, 4e-9, 3e-9), 8e5)(_planes(e, nx, ny))).numpy()
        bp = []
        for p in ps:
            d = 4e-9 / p.ratio
            X, Y = np.meshgrid((p.i0 * p.ratio + np.arange(p.pnx) - p.ghost + 0.5) * d,
                               (p.j0 * p.ratio + np.arange(p.pny) - p.ghost + 0.5) * d)
            bp.append(_bilinear(b.reshape(ny, nx, 3), 4e-9, 4e-9, X.reshape(-1), Y.reshape(-1)))
        return dict(bc=b, bp=bp)
    return _exact_train(case, seed)
