"""The work that users of fastreg_gb300 have it do, as cases to be timed and compared.

Whole registrations with either solver (one pair, a cohort of uneven pairs), the
differentiated registration that weights are tuned with, and the standalone field
operations (warp, its adjoint, sampling a vector field), each through the entry point that
a program calls, from volumes of a few ten thousand voxels to cohorts of tens of millions.

Inputs are the synthetic pairs that the tests and the benchmark use, made on the GPU from
the seed: a clipped sum of Gaussian blobs, and a source that is the target warped by the
exponential of a smooth random velocity, with threshold labels.

``exact`` restates each operation in 64-bit torch, independent of the package.
"""
from __future__ import annotations

import ctypes
import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from fastreg_gb300 import FastReg, Params, _native, interpolate_field, warp
from fastreg_gb300.hypertune import sobolev_loss_grad

# voxel-iterations up to which the 64-bit restatement of a registration takes seconds
EXACT_LIMIT = 1.6e9

# ------------------------------------------------------------------------------ cases


def listed():
    return [
        # the smallest registration that is quoted: a 64^3 pair, the reference solver with
        # the values of params.ini; launches and latency count
        _register("ref_64cube", "reference", "64x64x64", iters=200, labels=4),
        # the drop-in throughput case: one brain-sized pair, 200 iterations
        _register("ref_182x218x182", "reference", "182x218x182", iters=200, labels=8),
        # the same pair with the sobolev solver
        _register("sob_182x218x182", "sobolev", "182x218x182", iters=200, labels=8),
        # a cohort of uneven pairs in one set of launches, as a study is registered
        _register("ref_cohort_uneven", "reference",
                  "96x112x96,192x224x192,128x160x96,160x112x128,96x224x192,192x160x128,"
                  "128x224x96,160x160x192,96x160x128,192x112x96,160x224x128,128x112x192", iters=200, labels=4),
        # an atlas cohort: equal sizes, sobolev solver
        _register("sob_cohort_160", "sobolev", ",".join(["160x192x160"] * 8), iters=200, labels=8),
        # a half-resolution pair of odd sizes with a wide smoothing kernel (a coarse level)
        _register("sob_wide_91x109x91", "sobolev", "91x109x91", iters=100, labels=8, width=11, sigma=2.5),
        # the differentiated registration at its quoted size: gradients w.r.t. the initial
        # velocity and the weight through 50 iterations, checkpoints every 10
        _loss_grad("loss_grad_128cube", "128x128x128", iters=50, every=10),
        # a hypergradient step on a small volume of odd sizes, where launches count
        _loss_grad("loss_grad_45x54x45", "45x54x45", iters=30, every=10),
        # an image and its labels resampled at params.ini's default size (odd in every axis)
        dict(name="warp_193x229x193", kind="warp", dims="193x229x193", labels=8, disp=6.0),
        # the smallest call: an image alone
        dict(name="warp_64cube", kind="warp", dims="64x64x64", labels=0, disp=3.0),
        # the gradient of a warped image w.r.t. positions and intensities
        dict(name="warp_adjoint_160x192x160", kind="warp_adjoint", dims="160x192x160", disp=5.0),
        # a vector field sampled at positions (composing deformations)
        dict(name="interp_182x218x182", kind="interp", dims="182x218x182", disp=6.0),
    ]


def _register(name, solver, dims, iters, labels, width=7, sigma=1.5, w_reg=0.2, reset=-1):
    case = dict(kind="register", solver=solver, dims=dims, iters=iters, labels=labels, width=width, sigma=sigma,
                w_reg=w_reg, reset=reset)
    return dict(case, name=name) if name else case


def _loss_grad(name, dims, iters, every, width=7, sigma=1.5, w_reg=0.2):
    case = dict(kind="loss_grad", dims=dims, iters=iters, every=every, width=width, sigma=sigma, w_reg=w_reg)
    return dict(case, name=name) if name else case


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def dims(lo, hi):
        return "x".join(str(log_int(lo, hi)) for _ in range(3))

    kind = rng.choice(["register"] * 4 + ["loss_grad"] * 2 + ["warp", "warp_adjoint", "interp"])
    if kind == "register":
        solver = rng.choice(["reference", "sobolev"])
        sizes = ",".join(dims(40, 200) for _ in range(rng.choice([1, 1, 1, 2, 5])))
        width = rng.choice([5, 7, 7, 9, 13]) if solver == "sobolev" else 7
        return _register(None, solver, sizes, iters=log_int(20, 200), labels=rng.choice([2, 4, 8, 32]), width=width,
                         sigma=round(width / 4.5, 2), w_reg=round(rng.uniform(0.05, 0.4), 3),
                         reset=rng.choice([-1, -1, 50]))
    if kind == "loss_grad":
        width = rng.choice([5, 7, 9])
        return _loss_grad(None, dims(32, 128), iters=log_int(5, 50), every=rng.choice([5, 8, 10]), width=width,
                          sigma=round(width / 4.5, 2), w_reg=round(rng.uniform(0.05, 0.4), 3))
    case = dict(kind=kind, dims=dims(40, 230), disp=round(rng.uniform(1.0, 6.0), 2))
    return dict(case, labels=rng.choice([0, 8])) if kind == "warp" else case


def _sizes(case):
    return [tuple(int(v) for v in d.split("x")) for d in case["dims"].split(",")]


def work(case):
    """Per voxel and iteration, at the FP32 layout.  Reference solver, 112 B: rho, v, psi_inv
    read and written, S, T and psi read once (76), then psi read and written and the new v
    read again by the update, which needs all of it (36).  Sobolev solver, 80 B: phi, S and T
    read for the gradient (20), the momentum read and written (24), then phi read and written
    and the new momentum read (36).  Differentiated: that, and for the reverse step phi, m, S
    and T read, both adjoint fields read and written, the smoothed one passed on (104).  The
    field operations: every array once."""
    n = sum(x * y * z for x, y, z in _sizes(case))
    kind = case["kind"]
    if kind == "register":
        ref = case["solver"] == "reference"
        taps = 0 if ref else 6 * 3 * case["width"]
        return dict(bytes=n * case["iters"] * (112 if ref else 80), flops=n * case["iters"] * (330 if ref else 170 + taps))
    if kind == "loss_grad":
        return dict(bytes=n * case["iters"] * 184, flops=n * case["iters"] * (500 + 12 * 3 * case["width"]))
    if kind == "warp":
        return dict(bytes=n * (20 + (4 if case["labels"] else 0)), flops=n * 30)
    if kind == "warp_adjoint":
        return dict(bytes=n * 36, flops=n * 60)
    return dict(bytes=n * 36, flops=n * 60)


# ------------------------------------------------------------------------------ inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _smooth_axis(v, axis, sigma):
    """Gaussian along one axis, replicate boundary, as a product with a banded matrix."""
    n = v.shape[axis]
    i = torch.arange(n, device=v.device, dtype=torch.float32)
    r = int(3 * sigma + 0.5)
    k = torch.arange(-r, r + 1, device=v.device)
    w = torch.exp(-k.float() ** 2 / (2 * sigma * sigma))
    w = w / w.sum()
    m = torch.zeros(n, n, device=v.device)
    for t in range(2 * r + 1):
        j = (i.long() + k[t]).clamp(0, n - 1)
        m[i.long(), j] += w[t]
    return torch.movedim(torch.movedim(v, axis, -1) @ m.T, -1, axis)


def _velocity(g, dims, sigma, peak):
    x, y, z = dims
    v = _randn(g, 3, z, y, x)
    for axis in (1, 2, 3):
        v = _smooth_axis(v, axis, sigma)
    return v * (peak / v.pow(2).sum(0).sqrt().max())


def _grid(dims, dtype=torch.float32):
    x, y, z = dims
    a = [torch.arange(n, device="cuda", dtype=dtype) for n in (z, y, x)]
    zz, yy, xx = torch.meshgrid(*a, indexing="ij")
    return torch.stack([xx, yy, zz])


def _sample32(field, disp, mode="bilinear"):
    """field (C, Z, Y, X) at x + disp, clamped to the volume."""
    c, z, y, x = field.shape
    scale = torch.tensor([2.0 / max(n - 1, 1) for n in (x, y, z)], device=field.device).view(3, 1, 1, 1)
    grid = ((_grid((x, y, z)) + disp) * scale - 1.0).permute(1, 2, 3, 0)[None]
    return F.grid_sample(field[None], grid, mode=mode, padding_mode="border", align_corners=True)[0]


def _displacement(g, dims, peak):
    u = _velocity(g, dims, 5.0, peak) / 64.0
    for _ in range(6):  # scaling and squaring
        u = u + _sample32(u, u)
    return u


def _target(g, dims):
    """A clipped sum of Gaussian blobs with a little noise."""
    n = max(40, dims[0] * dims[1] * dims[2] // 18000)
    r = torch.rand(n, 5, generator=g, device="cuda")
    s, a = 3.0 + 5.0 * r[:, 3:4], 0.2 + 0.8 * r[:, 4:5]
    gx, gy, gz = (torch.exp(-((torch.arange(d, device="cuda")[None] - r[:, k:k + 1] * (d - 1)) ** 2) / (2 * s * s))
                  for k, d in enumerate(dims))
    t = torch.einsum("nz,ny->zyn", a * gz, gy) @ gx
    return t.clamp(0.0, 1.0) + 0.01 * _randn(g, dims[2], dims[1], dims[0])


def _pair(g, dims, labels, peak=5.0):
    t = _target(g, dims)
    u = _displacement(g, dims, peak)
    s = _sample32(t[None], u)[0]
    thr = torch.arange(1, labels, device="cuda") / labels
    lab_t = torch.bucketize(t.clamp(0, 1), thr, right=True).to(torch.int16)
    lab_s = _sample32(lab_t[None].float(), u, "nearest")[0].to(torch.int16)
    return [v.contiguous() for v in (t, lab_t, s, lab_s)]


def _params(case, dims):
    return Params(volume_dims=dims, no_labels=case.get("labels", 4), max_iter=case["iters"],
                  solver=case.get("solver", "sobolev"), w_reg=case["w_reg"], smooth_sigma=case["sigma"],
                  smooth_width=case["width"], reset_iter=case.get("reset", -1))


def _field_inputs(case, seed):
    """Positions (identity plus a smooth displacement) and what is sampled there."""
    g, dims = _generator(seed), _sizes(case)[0]
    pos = (_grid(dims) + _displacement(g, dims, case["disp"])).contiguous()
    if case["kind"] == "interp":
        return dict(pos=pos, field=_velocity(g, dims, 4.0, 3.0).contiguous())
    img = _target(g, dims).contiguous()
    if case["kind"] == "warp_adjoint":
        return dict(pos=pos, img=img, wbar=0.1 * _randn(g, *img.shape))
    n = case["labels"]
    lab = None
    if n:
        thr = torch.arange(1, n, device="cuda") / n
        lab = torch.bucketize(img.clamp(0, 1), thr, right=True).to(torch.int16)
    return dict(pos=pos, img=img, lab=lab)


def prepare(case, seed):
    kind, sizes = case["kind"], _sizes(case)
    if kind == "register":
        g = _generator(seed)
        pairs = [_pair(g, d, case["labels"]) for d in sizes]
        # the solver's handle, and the buffers that a registration overwrites in place
        return dict(case=case, pairs=pairs, buffers=[[torch.empty_like(v) for v in p] for p in pairs],
                    handle=FastReg(_params(case, sizes[0])))
    if kind == "loss_grad":
        g = _generator(seed)
        t, _, s, _ = _pair(g, sizes[0], 4, peak=4.0)
        return dict(case=case, t=t, s=s, v0=_velocity(g, sizes[0], 4.0, 0.3).contiguous(), params=_params(case, sizes[0]))
    return dict(case=case, **_field_inputs(case, seed))


# ------------------------------------------------------------------------------ the calls


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "register":
        fr, bufs = state["handle"], state["buffers"]
        for pair, buf in zip(state["pairs"], bufs):  # the images arrive in the call's buffers
            for v, b in zip(pair, buf):
                b.copy_(v)
        if len(bufs) == 1:
            fr(*bufs[0])
        else:
            fr.register_batch([tuple(b) for b in bufs])
        out = [dict(zip(("T", "labT", "S", "labS"), b), psi=fr.get_deformation_field(k)) for k, b in enumerate(bufs)]
        if len(bufs) == 1:
            st = fr.stats()
            out[0].update(e_data=st.e_data, e_reg=st.e_reg, folds=st.folds)
        return out
    if kind == "loss_grad":
        loss, grad_w, grad_v0 = sobolev_loss_grad(state["t"], state["s"], state["params"], case["w_reg"],
                                                  case["iters"], case["every"], v0=state["v0"])
        return dict(loss=loss, grad_w=grad_w, grad_v0=grad_v0)
    if kind == "warp":
        out = warp(state["pos"], state["img"], state["lab"])
        return dict(zip(("img", "lab"), out)) if state["lab"] is not None else dict(img=out)
    if kind == "warp_adjoint":
        pos, img, wbar = state["pos"], state["img"], state["wbar"]
        pos_bar, img_bar = torch.empty_like(pos), torch.empty_like(img)
        lib = _native.load()
        _native.check(lib.fr_warp_adjoint(pos.data_ptr(), img.data_ptr(), wbar.data_ptr(),
                                          (ctypes.c_int * 3)(*_sizes(case)[0]), pos_bar.data_ptr(), img_bar.data_ptr(),
                                          None), None, "fr_warp_adjoint")
        return dict(pos_bar=pos_bar, img_bar=img_bar)
    return dict(out=interpolate_field(state["field"], state["pos"]))


# ------------------------------------------------------------------------------ 64 bits


def _cell(pos, dims):
    """Cell of a position clamped into the volume (both corners of every axis inside it):
    base indices, fractions, and which axes were not clamped."""
    p, g, f, inside = [], [], [], []
    for k, n in enumerate(dims):
        inside.append((pos[k] >= 0) & (pos[k] <= n - 1))
        p.append(pos[k].clamp(0, n - 1))
        g.append(p[k].detach().floor().long().clamp(max=n - 2))
        f.append(p[k] - g[k])
    return g[0] + dims[0] * (g[1] + dims[1] * g[2]), f, inside


def _corners(field, base, dims):
    flat, x, xy = field.reshape(-1), dims[0], dims[0] * dims[1]
    return {(i, j, k): flat[base + i + x * j + xy * k] for i in (0, 1) for j in (0, 1) for k in (0, 1)}


def _mix(v0, v1, t):
    return v0 + t * (v1 - v0)


def _along(c, f, axes):
    """Interpolates the corners along `axes`; the other axes are differentiated."""
    for axis in (2, 1, 0):
        low = {k: v for k, v in c.items() if k[axis] == 0}
        def high(k, axis=axis):
            return k[:axis] + (1,) + k[axis + 1:]
        c = {k: _mix(v, c[high(k)], f[axis]) if axis in axes else c[high(k)] - v for k, v in low.items()}
    return c[(0, 0, 0)]


def _sample(field, pos, dims):
    base, f, _ = _cell(pos, dims)
    return torch.stack([_along(_corners(v, base, dims), f, (0, 1, 2)) for v in field])


def _shift(f, axis, by):
    """f at the neighbour `by` along x, y or z (axis 0, 1, 2), edges repeated."""
    d = f.dim() - 1 - axis
    i = (torch.arange(f.shape[d], device=f.device) + by).clamp(0, f.shape[d] - 1)
    return f.index_select(d, i)


def _interior(dims, lo, hi):
    m = torch.ones(dims[2], dims[1], dims[0], dtype=torch.bool, device="cuda")
    for k, c in enumerate(_grid(dims, torch.long)):
        m &= (c >= lo[k]) & (c <= dims[k] - 1 - hi[k])
    return m


def _reference_iteration(dims, masks, T, S, grad_S, rho, v, q, psi, first, alpha, t, tau, w_reg):
    """One iteration of the reference's flow (p = 2, C = 1/4) in the fields rho, v, psi_inv
    (q) and psi, with its upwind differences, its determinant and its index slips as they are."""
    inner, inner2 = masks
    nb = [[(_shift(v[c], a, -1), _shift(v[c], a, 1)) for a in range(3)] for c in range(3)]
    div = 0.0
    for a in range(3):
        vm = nb[a][a][0]
        div = div + torch.where(v[a] > 0, -v[a] * rho, -v[a] * _shift(rho, a, 1))
        div = div + torch.where(vm > 0, vm * _shift(rho, a, -1), vm * rho)
    rho_n = torch.where(inner, rho + alpha * div, rho)
    M = [[(_shift(q[r], a, 1) - _shift(q[r], a, -1)) * 0.5 for a in range(3)] for r in range(3)]
    det = ((M[0][0] * M[1][1] * M[2][2] + M[1][0] * M[2][1] * M[0][2]) + M[2][0] * M[0][1] * M[1][2]) - (
        (M[0][2] * M[1][1] + M[2][0]) * (M[1][2] * M[2][1] * M[0][0]) + M[2][2] * M[0][1] * M[1][0])
    lap = torch.stack([torch.where(inner, 6 * p - sum(_shift(p, a, s) for a in range(3) for s in (-1, 1)),
                                   torch.zeros_like(p)) for p in psi])
    gathered = _sample(torch.cat([lap, T[None]]), q, dims)
    diff = S - (T if first else gathered[3])
    qd = (0.25 * 4.0) / (rho_n.abs() + 1e-5)
    v_n = []
    for c in range(3):
        adv = 0.0
        for a in range(3):
            lo, hi = nb[c][a]
            if a == c:
                sq = lambda w: w.clamp(min=0) ** 2 - w.clamp(max=0) ** 2  # noqa: E731
                adv = adv + 0.5 * (sq(v[c]) - sq(hi))
            else:
                adv = adv + torch.where(v[a] > 0, v[a] * (v[c] - lo), v[a] * (hi - v[c]))
        second = 0.0
        for a in range(3):
            lo, hi = nb[c][a]
            up = _shift(v[c], a, 2)
            if a == 1:  # at y = Y - 2 the y + 2 read is voxel (x, 0, z + 1)
                up = up.clone()
                up[:-1, -2] = v[c][1:, 0]
            fwd = (up - 2 * (hi if a == 0 else lo)) + v[c]
            second = second + torch.where(v[a] < 0, fwd, (v[c] - 2 * lo) + _shift(v[c], a, -2))
        dv = torch.where(inner2, -second, torch.zeros_like(second))
        gU = (diff * grad_S[c] + w_reg * gathered[c]) * det
        v_n.append(torch.where(inner, v[c] - alpha * (3.0 / t * v[c] + adv - tau * dv + qd * gU), v[c]))
    v_n = torch.stack(v_n)
    q_n = torch.stack([torch.where(inner, q[r] - alpha * sum(M[r][a] * v_n[a] for a in range(3)), q[r])
                       for r in range(3)])
    psi_n = psi + torch.where(inner, alpha * _sample(v_n, psi, dims), torch.zeros_like(psi))
    return rho_n, v_n, q_n, psi_n


def _reference_exact(case, pair, dims):
    p = _params(case, dims)
    T, S = pair[0].double(), pair[2].double()
    ident = _grid(dims, torch.float64)
    masks = _interior(dims, (1, 1, 1), (1, 1, 1)), _interior(dims, (2, 2, 2), (2, 1, 2))
    grad_S = [(_shift(S, a, 1) - _shift(S, a, -1)) * 0.5 for a in range(3)]
    rho, v, q, psi = torch.full_like(T, p.rho_0), torch.zeros_like(ident), ident, ident
    t = p.alpha
    for it in range(1, p.max_iter + 1):
        rho, v, q, psi = _reference_iteration(dims, masks, T, S, grad_S, rho, v, q, psi, it == 1, p.alpha, t, p.tau,
                                              p.w_reg)
        t = p.alpha if p.reset_iter > 0 and (it + 1) % p.reset_iter == 0 else t + p.alpha
    return dict(T=_sample(T[None], q, dims)[0], S=_sample(S[None], psi, dims)[0], psi=psi)


def _smooth64(v, width, sigma):
    """Separable normalised Gaussian, replicate boundary, along x, then y, then z."""
    r = width // 2
    w = torch.exp(-torch.arange(-r, r + 1, device=v.device, dtype=torch.float64) ** 2 / (2 * sigma * sigma))
    w = w / w.sum()
    for a in range(3):
        v = sum(w[k + r] * _shift(v, a, k) for k in range(-r, r + 1))
    return v


def _sobolev_step(phi, m, T, S, w_reg, ident, dims, p):
    base, f, inside = _cell(phi, dims)
    c = _corners(S, base, dims)
    r = _along(c, f, (0, 1, 2)) - T
    u = phi - ident
    lap = sum(u - _shift(u, a, s) for a in range(3) for s in (-1, 1))
    others = ((1, 2), (0, 2), (0, 1))
    grad = torch.stack([r * torch.where(inside[a], _along(c, f, others[a]), torch.zeros_like(r)) for a in range(3)])
    m = p.damping * m - p.step * _smooth64(grad + w_reg * lap, p.smooth_width, p.smooth_sigma)
    return phi + _sample(m, phi, dims), m


def _sobolev_exact(case, pair, dims):
    p = _params(case, dims)
    T, S = pair[0].double(), pair[2].double()
    ident = _grid(dims, torch.float64)
    phi, m = ident, torch.zeros_like(ident)
    for _ in range(p.max_iter):
        phi, m = _sobolev_step(phi, m, T, S, p.w_reg, ident, dims, p)
    return dict(T=pair[0].double(), S=_sample(S[None], phi, dims)[0], psi=phi)


def _energies(out, T, dims):
    """0.5 sum (T - S o psi)^2 and 0.5 sum |J|^2, J of psi - x with mirrored one-sided edges."""
    u = out["psi"] - _grid(dims, torch.float64)
    e = 0.0
    for a in range(3):
        d, n = 3 - a, dims[a]
        i = torch.arange(n, device=u.device)
        hi, lo = i + 1, i - 1
        hi[-1], lo[0] = n - 2, 1
        e += float((((u.index_select(d, hi) - u.index_select(d, lo)) * 0.5) ** 2).sum())
    return 0.5 * float(((T.double() - out["S"]) ** 2).sum()), 0.5 * e


def _exact_register(case, seed):
    sizes = _sizes(case)
    if sum(x * y * z for x, y, z in sizes) * case["iters"] > EXACT_LIMIT:
        return None
    g, outs = _generator(seed), []
    for pair, d in [(_pair(g, d, case["labels"]), d) for d in sizes]:
        out = (_reference_exact if case["solver"] == "reference" else _sobolev_exact)(case, pair, d)
        # labels follow positions near cell faces, so they have no 64-bit value of their own
        outs.append(dict(T=out["T"], labT=None, S=out["S"], labS=None, psi=out["psi"]))
        if len(sizes) == 1:
            e_data, e_reg = _energies(out, pair[0], d)
            # the reference flow's displacements are a few roundings of an FP32 position, so
            # the energy of their differences has no 64-bit value either
            outs[0].update(e_data=e_data, e_reg=None if case["solver"] == "reference" else e_reg, folds=None)
    return outs


def _exact_loss_grad(case, seed):
    s, dims = prepare(case, seed), _sizes(case)[0]
    p, T, S = s["params"], s["t"].double(), s["s"].double()
    ident = _grid(dims, torch.float64)
    v0 = s["v0"].double().requires_grad_()
    w = torch.tensor(case["w_reg"], device="cuda", dtype=torch.float64, requires_grad=True)
    phi, m = ident, v0
    for _ in range(case["iters"]):
        phi, m = checkpoint(_sobolev_step, phi, m, T, S, w, ident, dims, p, use_reentrant=False)
    loss = 0.5 * ((_sample(S[None], phi, dims)[0] - T) ** 2).sum() + 0.1 * (m ** 2).sum()
    loss.backward()
    return dict(loss=loss.item(), grad_w=w.grad.item(), grad_v0=v0.grad)


def exact(case, seed):
    kind = case["kind"]
    if kind == "loss_grad":
        return _exact_loss_grad(case, seed)
    with torch.no_grad():
        if kind == "register":
            return _exact_register(case, seed)
        s, dims = _field_inputs(case, seed), _sizes(case)[0]
        pos = s["pos"].double()
        if kind == "interp":
            return dict(out=_sample(s["field"].double(), pos, dims))
        img = s["img"].double()
        if kind == "warp":
            out = dict(img=_sample(img[None], pos, dims)[0])
            if s["lab"] is not None:  # the label of the position's floor voxel
                i = [s["pos"][k].clamp(0, n - 1).floor().long() for k, n in enumerate(dims)]
                out["lab"] = s["lab"].reshape(-1)[i[0] + dims[0] * (i[1] + dims[1] * i[2])]
            return out
        base, f, inside = _cell(pos, dims)
        c, wbar = _corners(img, base, dims), s["wbar"].double()
        others = ((1, 2), (0, 2), (0, 1))
        pos_bar = torch.stack([wbar * torch.where(inside[a], _along(c, f, others[a]), torch.zeros_like(wbar))
                               for a in range(3)])
        img_bar = torch.zeros_like(img).reshape(-1)
        for (i, j, k) in c:
            wt = (f[0] if i else 1 - f[0]) * (f[1] if j else 1 - f[1]) * (f[2] if k else 1 - f[2])
            img_bar.index_add_(0, (base + i + dims[0] * (j + dims[1] * k)).reshape(-1), (wt * wbar).reshape(-1))
        return dict(pos_bar=pos_bar, img_bar=img_bar.reshape(img.shape))
