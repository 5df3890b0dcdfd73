"""The work that a program has this library do, as cases that can be timed.

Every case goes through the public Python layer (`CudaCalcTholeDipoleForceKernel`,
`DeviceRigidWaterMD`, `ClusterBatch`, `thole_dipole`, `thole_dipole_clusters`), with device-resident
inputs and outputs wherever that layer takes them.  Systems are the library's own rigid-water boxes
and clusters at the density of its measured configurations (0.3107 nm per lattice site), solved to
the tolerances of its timed workloads (1e-7 in boxes, 1e-10 in clusters).

The mixed form carries FP32 pair arithmetic, so a program that picks it takes its results in single
precision (FP32 force buffers, FP32 parameters of a fit, FP32 trajectory frames); the plain form
gives FP64.

`exact` restates the physics in FP64 torch, without the library: the minimum-image or open all-pairs
sums with the quasi-internal-frame pair terms, and for the variational modes an energy function
(an Ewald sum with explicit reciprocal vectors) whose forces come from autograd.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tholedipoleplugin_b200 import _capi as A
from tholedipoleplugin_b200 import systems as S
from tholedipoleplugin_b200.autograd import ClusterGradients, thole_dipole, thole_dipole_clusters
from tholedipoleplugin_b200.batch import ClusterBatch
from tholedipoleplugin_b200.kernel import CudaCalcTholeDipoleForceKernel
from tholedipoleplugin_b200.md import D_HH, D_OH, DeviceRigidWaterMD, maxwell_boltzmann

SPACING = 0.3107          # nm per lattice site of the measured boxes (1.8643 / 6)
DT = 0.001                # ps
TEMPERATURE = 300.0
POLARIZATION = {"mutual": S.MUTUAL, "direct": S.DIRECT, "extrapolated": S.EXTRAPOLATED}


def listed():
    return [
        # One force evaluation of the smallest measured box (216 waters): an energy minimiser or a
        # Monte Carlo move on a small sample.  Launches and host reads dominate.
        _forces("forces_box648", 6, "mixed", "mutual"),
        # The same at 1,029 atoms with the FP64 form (7^3 waters, not a multiple of the 32-atom
        # tile): reference values for a check of another code.
        _forces("forces_box1029_fp64", 7, "double", "mutual"),
        # A droplet without periodic images (1,331 waters, 3,993 atoms), extrapolated polarization:
        # the fixed-order perturbation scheme that MD codes use in place of a solve.
        _forces("forces_drop3993_extrapolated", 11, "mixed", "extrapolated", method="nocutoff"),
        # The middle measured box (4,096 waters), one cold evaluation in each form: relaxed scans,
        # validation of force fields.
        _forces("forces_box12288", 16, "mixed", "mutual"),
        _forces("forces_box12288_fp64", 16, "double", "mutual"),
        # MD of the largest measured box (32,768 waters): the headline workload, one velocity
        # Verlet step with a warm-started solve.
        _md("md_box98304", 32, "mixed", ewald=False),
        # The same box with the true Ewald sum, the production setting for liquids.
        _md("md_ewald98304", 32, "mixed", ewald=True),
        # A small Ewald box (2,197 waters, odd size), where launches and the mesh matter.
        _md("md_ewald6591", 13, "mixed", ewald=True),
        # Many isolated clusters in one launch (4-64 waters): many-body expansion fragments,
        # training-set evaluation.
        _clusters("clusters1024", 1024, 4, 64, "mixed"),
        # One force-matching step over 256 clusters in FP64: forward, loss, backward.
        _fit_clusters("fit_clusters256_fp64", 256, 4, 64, "double"),
        # One force-matching step on the middle box in the mixed form.
        _fit_box("fit_box12288", 16, "mixed"),
        # Potential of the middle box on a 32^3 grid, a query with host arrays at both ends
        # (charge fitting, visualisation).
        _potential("potential_box12288", 16, 32, "double"),
    ]


def _forces(name, n_side, precision, polarization, method="pme", ewald=False, variational=False):
    return {"name": name, "kind": "forces", "n_side": n_side, "precision": precision, "polarization": polarization,
            "method": method, "ewald": ewald, "variational": variational}


def _md(name, n_side, precision, ewald):
    return {"name": name, "kind": "md", "n_side": n_side, "precision": precision, "ewald": ewald}


def _clusters(name, count, lo, hi, precision):
    return {"name": name, "kind": "clusters", "count": count, "lo": lo, "hi": hi, "precision": precision}


def _fit_clusters(name, count, lo, hi, precision):
    return {"name": name, "kind": "fit_clusters", "count": count, "lo": lo, "hi": hi, "precision": precision}


def _fit_box(name, n_side, precision):
    return {"name": name, "kind": "fit_box", "n_side": n_side, "precision": precision}


def _potential(name, n_side, grid, precision):
    return {"name": name, "kind": "potential", "n_side": n_side, "grid": grid, "precision": precision}


def draw(rng):
    """One more case: a kind by how often programs meet it, its size log-uniform over the kind's range."""

    def size(lo, hi):
        return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))

    kind = rng.choice(["forces", "forces", "forces", "variational", "md", "md_ewald", "md_ewald", "clusters",
                       "clusters", "fit_clusters", "fit_box", "potential"])
    precision = rng.choice(["mixed", "mixed", "double"])
    if kind == "forces":
        pol = rng.choice(["mutual", "mutual", "direct", "extrapolated"])
        method = rng.choice(["pme", "pme", "nocutoff"])
        # a box edge is at least twice the 0.8 nm cutoff: 6 sites
        c = _forces("", size(6 if method == "pme" else 3, 27 if precision == "mixed" else 20), precision, pol, method)
    elif kind == "variational":
        open_ = rng.random() < 0.5
        c = _forces("", size(3, 12) if open_ else size(6, 24), precision, rng.choice(["mutual", "mutual", "direct"]),
                    "nocutoff" if open_ else "pme", ewald=not open_, variational=open_)
    elif kind == "md":
        c = _md("", size(6, 31 if precision == "mixed" else 22), precision, False)
    elif kind == "md_ewald":
        c = _md("", size(6, 32 if precision == "mixed" else 26), precision, True)
    elif kind == "clusters":
        lo = rng.randint(2, 20)
        c = _clusters("", size(16, 2048), lo, lo + rng.randint(4, 44), precision)
    elif kind == "fit_clusters":
        lo = rng.randint(2, 12)
        c = _fit_clusters("", size(16, 512), lo, lo + rng.randint(4, 44), precision)
    elif kind == "fit_box":
        c = _fit_box("", size(6, 18 if precision == "mixed" else 15), precision)
    else:
        c = _potential("", size(6, 20), size(4, 40), precision)
    del c["name"]
    return c


# -- inputs --------------------------------------------------------------------------------------
def _box(case, seed):
    n = case["n_side"]
    pol = POLARIZATION[case.get("polarization", "mutual")]
    method = S.NO_CUTOFF if case.get("method") == "nocutoff" else S.PME
    return S.water_box(n, SPACING * n, seed=seed, cutoff=0.9 if n >= 7 else 0.8, polarization=pol,
                       target_eps=S.BOX_SOLVER_EPS, method=method)


def _cluster_list(case, seed):
    sizes = np.random.default_rng(3).integers(case["lo"], case["hi"] + 1, size=case["count"])  # the same for any seed
    rng = np.random.default_rng(seed)
    return [S.water_cluster(int(w), rng, target_eps=S.CLUSTER_SOLVER_EPS) for w in sizes]


def _parameters(system, dtype, seed):
    """Trial parameters of a fit (a few percent around the model's) as leaves that take gradients."""
    rng = np.random.default_rng(seed + 1)
    out = []
    for a in (system.charges, system.polarizabilities, system.tholes, system.dipoles):
        a = np.asarray(a) * rng.uniform(0.97, 1.03, np.asarray(a).shape)
        out.append(torch.tensor(a, dtype=dtype, device="cuda", requires_grad=True))
    return out


def _targets(n, dtype, seed):
    """Target forces of a fit, with the size of a water's forces in these units."""
    rng = np.random.default_rng(seed + 2)
    return torch.tensor(rng.normal(scale=5.0, size=(n, 3)), dtype=dtype, device="cuda")


def _grid(case, system, seed):
    m = case["grid"]
    shift = np.random.default_rng(seed + 3).uniform(0.0, 1.0, 3)
    g = [(np.arange(m) + s) * (L / m) for s, L in zip(shift, system.box)]
    return np.stack(np.meshgrid(*g, indexing="ij"), axis=-1).reshape(-1, 3)


def _result_dtype(case):
    return torch.float32 if case["precision"] == "mixed" else torch.float64


def prepare(case, seed):
    kind = case["kind"]
    dtype = _result_dtype(case)
    stream = torch.cuda.current_stream().cuda_stream
    st = {"case": case, "dtype": dtype}
    if kind == "forces":
        s = _box(case, seed)
        st["kernel"] = CudaCalcTholeDipoleForceKernel(s, precision=case["precision"], ewald=case["ewald"],
                                                      variational=case["variational"])
        st["kernel"].setStream(stream)
        st["pos"] = torch.tensor(s.positions, dtype=torch.float64, device="cuda")
        st["frc"] = torch.zeros((s.n, 3), dtype=dtype, device="cuda")
    elif kind == "md":
        st["md"] = DeviceRigidWaterMD(_box(case, seed), precision=case["precision"], dt=DT, temperature=TEMPERATURE,
                                      seed=seed, ewald=case["ewald"])
        st["turn"] = 20
    elif kind == "clusters":
        b = ClusterBatch(_cluster_list(case, seed), precision=case["precision"])
        b.setStream(stream)
        st["batch"] = b
        st["pos"] = torch.tensor(b.positions, dtype=torch.float64, device="cuda")
        st["frc"] = torch.empty_like(st["pos"])
        st["en"] = torch.empty(b.num_clusters, dtype=torch.float64, device="cuda")
        b.compute_device(st["pos"].data_ptr(), st["frc"].data_ptr(), st["en"].data_ptr())  # picks its tile once
    elif kind == "fit_clusters":
        cg = ClusterGradients(_cluster_list(case, seed), precision=case["precision"])
        st["batch"] = cg
        st["params"] = _parameters(cg.system, dtype, seed)
        st["target"] = _targets(cg.n, dtype, seed)
        run(st)
    elif kind == "fit_box":
        s = _box(case, seed)
        st["system"] = s
        st["kernel"] = CudaCalcTholeDipoleForceKernel(s, precision=case["precision"])
        st["pos"] = torch.tensor(s.positions, dtype=torch.float64, device="cuda")
        st["params"] = _parameters(s, dtype, seed)
        st["target"] = _targets(s.n, dtype, seed)
    else:
        s = _box(case, seed)
        st["kernel"] = CudaCalcTholeDipoleForceKernel(s, precision=case["precision"])
        st["kernel"].setStream(stream)
        st["grid"] = _grid(case, s, seed)
        st["positions"] = s.positions
    return st


def run(st):
    kind, dtype = st["case"]["kind"], st["dtype"]
    if kind == "forces":
        # forces are added to the caller's buffer, which starts from zero as a context's does
        st["frc"].zero_()
        e = st["kernel"].execute_device(st["pos"].data_ptr(), A.F64, st["frc"].data_ptr(),
                                        A.F32 if dtype == torch.float32 else A.F64)
        return {"energy": e, "forces": st["frc"]}
    if kind == "md":
        # The force has no repulsion: left alone, molecules run into one another within some hundred steps.  Velocities
        # turn round every 20 steps, which leads back along the same path, so a long run stays at the liquid's spacing.
        md = st["md"]
        if md.steps and md.steps % st["turn"] == 0:
            md.vel.neg_()
        e = md.step(1)
        # the frame that goes to a trajectory: single precision from the mixed form
        return {"energy": e, "forces": md.frc.to(dtype), "positions": md.pos.to(dtype), "velocities": md.vel.to(dtype)}
    if kind == "clusters":
        st["batch"].compute_device(st["pos"].data_ptr(), st["frc"].data_ptr(), st["en"].data_ptr())
        return {"energies": st["en"].to(dtype), "forces": st["frc"].to(dtype)}
    if kind in ("fit_clusters", "fit_box"):
        p = st["params"]
        for t in p:
            t.grad = None
        if kind == "fit_clusters":
            e, f = thole_dipole_clusters(*p, st["batch"])
        else:
            e, f = thole_dipole(*p, st["kernel"], st["system"], st["pos"])
        e, f = e.to(dtype), f.to(dtype)
        loss = ((f - st["target"]) ** 2).mean()
        loss.backward()
        return {"loss": loss.detach(), "energy": e.detach(), "forces": f.detach(), "grads": [t.grad for t in p]}
    v = st["kernel"].getElectrostaticPotential(st["grid"], st["positions"])
    return {"potential": v if dtype == torch.float64 else v.astype(np.float32)}


# -- work ----------------------------------------------------------------------------------------
# Operations per unordered pair: permanent field 75, mutual-field matvec 66, energy, force and torque
# 150 (a pair beyond the damping range), potential of one grid point and atom 20.  A cold solve to
# 1e-7 takes about 7 matvecs, one to 1e-10 about 10, a warm-started MD step 2; the extrapolated
# scheme takes 4; a reverse pass costs a second solve and about twice the energy pass.
F_FIXED, F_MATVEC, F_ENERGY, F_POINT = 75, 66, 150, 20


def _pairs(n_atoms, box_edge, cutoff):
    if cutoff is None:
        return 0.5 * n_atoms * (n_atoms - 1.0)
    return 0.5 * n_atoms * n_atoms * min(1.0, 4.0 / 3.0 * math.pi * cutoff ** 3 / box_edge ** 3)


def work(case):
    kind = case["kind"]
    if kind in ("clusters", "fit_clusters"):
        sizes = 3.0 * np.arange(case["lo"], case["hi"] + 1)
        n = case["count"] * float(sizes.mean())
        pairs = case["count"] * float((0.5 * sizes * (sizes - 1)).mean())
        its = 10
    else:
        n = 3.0 * case["n_side"] ** 3
        cut = (0.9 if case["n_side"] >= 7 else 0.8) if case.get("ewald") else None
        pairs = _pairs(n, SPACING * case["n_side"], cut)
        its = 2 if kind == "md" else {"direct": 0, "extrapolated": 4}.get(case.get("polarization"), 7)
    # positions, charges, dipoles, polarizabilities and Thole factors in (FP64); energy and forces out
    bytes_ = n * (24 + 8 + 24 + 8 + 8) + n * (12 if case["precision"] == "mixed" else 24)
    flops = pairs * (F_FIXED + its * F_MATVEC + F_ENERGY)
    if kind == "md":
        bytes_ += n * 48
    if kind in ("fit_clusters", "fit_box"):
        bytes_ += n * (24 + 48)
        flops += pairs * (F_FIXED + its * F_MATVEC + 2 * F_ENERGY)
    if kind == "potential":
        points = case["grid"] ** 3
        bytes_ += points * 32
        flops = pairs * (F_FIXED + its * F_MATVEC) + points * n * F_POINT
    return {"bytes": bytes_, "flops": flops}


# -- the same in 64 bits, without the library ------------------------------------------------------
def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / _dot(a, a).sqrt().unsqueeze(-1)


def _frames(pos):
    """Rows x, y, z of every water's z-then-x frame at its oxygen (z towards H1)."""
    o, h1, h2 = pos[0::3], pos[1::3], pos[2::3]
    z = _unit(h1 - o)
    x = h2 - o
    x = _unit(x - z * _dot(z, x).unsqueeze(-1))
    return torch.stack([x, torch.linalg.cross(z, x), z], dim=1)


def _lab(pos, mol):
    out = mol.clone()
    out[0::3] = torch.einsum("wr,wrc->wc", mol[0::3], _frames(pos))
    return out


def _torque_forces(pos, torque):
    """Forces on the frame atoms that do the work of the oxygens' torques (the gradient of the frame's rotation)."""
    keep = torch.is_grad_enabled()
    with torch.enable_grad():
        p = pos.detach().clone().requires_grad_(True)
        rows = _frames(p)
        turn = 0.5 * torch.linalg.cross(rows.detach(), rows).sum(1)
        return torch.autograd.grad(turn, p, torque[0::3], create_graph=keep)[0]


def _thole_x(r, ti, tj):
    x = torch.minimum(ti, tj) * (r / (ti * tj)) ** 3
    return torch.where(x < 50.0, x, torch.full_like(x, 1e3))


def _geometry(sys, lo, hi):
    """Displacements r_j - r_i of the rows lo:hi, distance (1 on the diagonal), the atoms' pairs and molecules."""
    pos = sys["pos"]
    d = pos.unsqueeze(0) - pos[lo:hi].unsqueeze(1)
    if sys["box"] is not None:
        d = d - sys["box"] * torch.floor(d / sys["box"] + 0.5)
    n = pos.shape[0]
    i = torch.arange(lo, hi, device=pos.device).unsqueeze(1)
    j = torch.arange(n, device=pos.device).unsqueeze(0)
    r2 = torch.where(i == j, 1.0, _dot(d, d))
    return d, r2.sqrt(), i, j


def _rows(n):
    step = max(1, 8_000_000 // max(1, n))
    return [(lo, min(n, lo + step)) for lo in range(0, n, step)]


def _field_kernels(sys, lo, hi):
    d, r, i, j = _geometry(sys, lo, hi)
    x = _thole_x(r, sys["t"][lo:hi].unsqueeze(1), sys["t"].unsqueeze(0))
    e = torch.exp(-x)
    r3 = (i != j) / r ** 3
    return d, r3 * (1 - e), 3.0 * r3 / r ** 2 * (1 - (1 + x) * e), i // 3 != j // 3


def _permanent_field(sys):
    out = []
    for lo, hi in _rows(sys["pos"].shape[0]):
        d, a3, a5, other = _field_kernels(sys, lo, hi)
        f = other * (a3 * sys["q"] - a5 * torch.einsum("ijc,jc->ij", d, sys["m"]))
        out.append(-torch.einsum("ij,ijc->ic", f, d) - (other * a3) @ sys["m"])
    return torch.cat(out)


def _mutual_field(sys, mu):
    out = []
    for lo, hi in _rows(sys["pos"].shape[0]):
        d, a3, a5, _ = _field_kernels(sys, lo, hi)
        out.append(torch.einsum("ij,ijc->ic", a5 * torch.einsum("ijc,jc->ij", d, mu), d) - a3 @ mu)
    return torch.cat(out)


def _solve(field, apply_t, alpha):
    """mu = alpha (E + T mu) by conjugate gradients on the symmetric form, to rounding."""
    s = alpha.sqrt().unsqueeze(-1)
    b = s * field
    y = b.clone()
    res = b - (y - s * apply_t(s * y))
    p = res.clone()
    rr = (res * res).sum()
    stop = 1e-26 * (b * b).sum()
    for _ in range(200):
        if rr <= stop:
            break
        q = p - s * apply_t(s * p)
        a = rr / (p * q).sum()
        y, res = y + a * p, res - a * q
        new = (res * res).sum()
        p, rr = res + new / rr * p, new
    return s * y


def _induced(sys, polarization):
    e = _permanent_field(sys)
    al = sys["alpha"].unsqueeze(-1)
    if polarization == "direct":
        return al * e
    if polarization == "extrapolated":
        mu = al * e
        acc = S.OPT4[0] * mu
        for c in S.OPT4[1:]:
            mu = al * (e + _mutual_field(sys, mu))
            acc = acc + c * mu
        return acc
    if sys["pos"].shape[0] <= 1024 and torch.is_grad_enabled():  # one dense solve, which autograd can go through
        n = sys["pos"].shape[0]
        d, a3, a5, _ = _field_kernels(sys, 0, n)
        t = (a5.unsqueeze(-1).unsqueeze(-1) * d.unsqueeze(-1) * d.unsqueeze(-2) -
             a3.unsqueeze(-1).unsqueeze(-1) * torch.eye(3, dtype=d.dtype, device=d.device))
        s = sys["alpha"].sqrt()
        t = t * (s.unsqueeze(1) * s.unsqueeze(0)).unsqueeze(-1).unsqueeze(-1)
        m = torch.eye(3 * n, dtype=d.dtype, device=d.device) - t.permute(0, 2, 1, 3).reshape(3 * n, 3 * n)
        s = s.unsqueeze(-1)
        return s * torch.linalg.solve(m, (s * e).reshape(-1)).reshape(n, 3)
    return _solve(e, lambda v: _mutual_field(sys, v), sys["alpha"])


def _pair_rows(sys, mu, mutual, lo, hi):
    """Energy, forces and torques of the pairs lo <= i < hi, j > i: the pair routine in its quasi-internal frame (rows
    X, Y, Z with Z along the pair, component 0 along X, and the permuted way back), 1/r^4 terms zero."""
    d, r, i, j = _geometry(sys, lo, hi)
    pos, m = sys["pos"], sys["m"]
    use = (j > i).to(d.dtype)
    ms = use * (i // 3 != j // 3)
    rinv = 1.0 / r
    z = torch.where((i == j).unsqueeze(-1), torch.tensor([0.0, 0.0, 1.0], dtype=d.dtype, device=d.device),
                    d * rinv.unsqueeze(-1))
    differ = (pos[lo:hi, None, 1] != pos[None, :, 1]) | (pos[lo:hi, None, 2] != pos[None, :, 2])
    x = z + torch.stack([differ, ~differ, torch.zeros_like(differ)], dim=-1)
    x = _unit(x - z * _dot(z, x).unsqueeze(-1))
    y = torch.linalg.cross(z, x)
    fr = (x, y, z)

    def turned(v, rows):
        w = v[lo:hi].unsqueeze(1) if rows else v.unsqueeze(0)
        return [_dot(a, w) for a in fr]

    ui, uj, pi, pj = turned(mu, True), turned(mu, False), turned(m, True), turned(m, False)
    qi, qj = sys["q"][lo:hi].unsqueeze(1), sys["q"].unsqueeze(0)
    au = _thole_x(r, sys["t"][lo:hi].unsqueeze(1), sys["t"].unsqueeze(0))
    ex = torch.exp(-au)
    tc = td1 = 1 - ex
    td0 = 1 - ex * (1 + 1.5 * au)
    r1, r2, r3 = rinv, rinv ** 2, rinv ** 3
    c1, c2, c3 = ms * r1, ms * r2, ms * r3
    u2, u3p, u3t = use * r2 * tc, use * r3 * td0, use * r3 * td1
    vij = [c1 * qj - c2 * pj[0] - u2 * uj[0], c2 * qj - 2 * c3 * pj[0] - 2 * u3p * uj[0],
           c3 * pj[1] + u3t * uj[1], c3 * pj[2] + u3t * uj[2]]
    vji = [c1 * qi + c2 * pi[0] + u2 * ui[0], -c2 * qi - 2 * c3 * pi[0] - 2 * u3p * ui[0],
           c3 * pi[1] + u3t * ui[1], c3 * pi[2] + u3t * ui[2]]
    dij = [u2 * qj - 2 * u3p * pj[0], u3t * pj[1], u3t * pj[2]]
    dji = [-u2 * qi - 2 * u3p * pi[0], u3t * pi[1], u3t * pi[2]]
    dc = use * r3 * td0  # the damping factor of the radial charge-dipole term
    rij0, rji0 = -0.5 * c2 * qj + c3 * pj[0] + 2 * dc * uj[0], -0.5 * c2 * qi - c3 * pi[0] - 2 * dc * ui[0]
    energy = 0.5 * (qi * vij[0] + qj * vji[0] + sum(pi[k] * vij[k + 1] + pj[k] * vji[k + 1] for k in range(3))).sum()
    radial = qi * rij0 + pi[0] * (-c3 * qj) + qj * rji0 + pj[0] * (c3 * qi)

    def across(a, v):  # the x, y, z parts of the torque of a on v
        return a[2] * v[0] - a[0] * v[2], a[0] * v[1] - a[1] * v[0], a[1] * v[2] - a[2] * v[1]

    ti, tj = across(pi, vij[1:]), across(pj, vji[1:])
    si, sj = across(ui, dij), across(uj, dji)
    ex_, ey_ = ti[0] + tj[0] + si[0] + sj[0], ti[1] + tj[1] + si[1] + sj[1]
    if mutual:
        ex_ = ex_ - 4 * u3p * (ui[2] * uj[0] + uj[2] * ui[0]) - 2 * u3t * (ui[0] * uj[2] + uj[0] * ui[2])
        ey_ = ey_ + 4 * u3p * (ui[1] * uj[0] + uj[1] * ui[0]) + 2 * u3t * (ui[0] * uj[1] + uj[0] * ui[1])

    def back(a0, a1, a2):
        return torch.stack([y[..., k] * a0 + z[..., k] * a1 + x[..., k] * a2 for k in (1, 2, 0)], dim=-1)

    f = back(rinv * ey_, -rinv * ex_, -radial)
    out_i, out_j = -f.sum(1), f.sum(0)
    return energy, out_i, out_j, back(-ti[0], -ti[1], -ti[2]).sum(1), back(-tj[0], -tj[1], -tj[2]).sum(0)


def _reference_forces(sys, polarization):
    """(energy, forces) of the default mode."""
    n = sys["pos"].shape[0]
    mu = _induced(sys, polarization)
    energy, frc, trq = 0.0, 0.0, 0.0
    for lo, hi in _rows(3 * n):
        lo, hi = min(lo, n), min(hi, n)
        if lo == hi:
            break
        e, fi, fj, ti, tj = _pair_rows(sys, mu, polarization == "mutual", lo, hi)
        pad = (0, 0, lo, n - hi)
        energy = energy + e
        frc = frc + fj + torch.nn.functional.pad(fi, pad)
        trq = trq + tj + torch.nn.functional.pad(ti, pad)
    return energy, frc + _torque_forces(sys["pos"], trq)


def _variational_energy(sys, pos, mu, parts):
    """The variational functional's electrostatic terms (no polarization energy) as a list of callables, one for each
    block of pairs and of reciprocal vectors; `parts`: (permanent dipoles or None, charges)."""
    q, t, box = parts[1], sys["t"], sys["box"]

    def m():
        return _lab(pos, sys["mol"]) if parts[0] else torch.zeros_like(pos)

    alpha = 0.0 if box is None else 10.0 / float(box.min())
    blocks = []

    def real(lo, hi):
        def energy():
            p = m()
            d, r, i, j = _geometry({"pos": pos, "box": box}, lo, hi)
            off = (i != j).to(r.dtype)
            x = _thole_x(r, t[lo:hi].unsqueeze(1), t.unsqueeze(0))
            ex = torch.exp(-x)
            l3, l5 = 1 - ex, 1 - (1 + x) * ex
            b1, b2 = 1 / r ** 3, 3 / r ** 5
            e2 = torch.exp(-(alpha * r) ** 2) * 2 * alpha / math.sqrt(math.pi)
            w0 = torch.erfc(alpha * r) / r
            w1 = (w0 + e2) / r ** 2
            w2 = (3 * w1 + 2 * alpha ** 2 * e2) / r ** 2
            other = (i // 3 != j // 3).to(r.dtype)
            qi, qj = q[lo:hi].unsqueeze(1), q.unsqueeze(0)

            def radial(v, w):
                vi, wj = torch.einsum("ic,ijc->ij", v[lo:hi], d), torch.einsum("jc,ijc->ij", w, d)
                return vi, wj, v[lo:hi] @ w.T

            pi, pj, pp = radial(p, p)
            ui, uj, uu = radial(mu, mu)
            pu, up = p[lo:hi] @ mu.T, mu[lo:hi] @ p.T
            perm = (qj * pi - qi * pj + pp, -pi * pj)
            mixed = (qj * ui - qi * uj + pu + up, -pi * uj - ui * pj)
            ind = (uu, -ui * uj)
            e = qi * qj * (w0 - (1 - other) / r)
            e = e + perm[0] * (w1 - (1 - other) * b1) + perm[1] * (w2 - (1 - other) * b2)
            e = e + mixed[0] * (w1 - (1 - other * l3) * b1) + mixed[1] * (w2 - (1 - other * l5) * b2)
            e = e + ind[0] * (w1 - (1 - l3) * b1) + ind[1] * (w2 - (1 - l5) * b2)
            return 0.5 * (off * e).sum()
        return energy

    n = pos.shape[0]
    for lo, hi in _rows(2 * n):
        if lo < n:
            blocks.append(real(lo, min(hi, n)))
    if box is None:
        return blocks
    top = 2.0 * alpha * 5.0
    c = [int(top * float(L) / (2 * math.pi)) for L in box]
    k = torch.cartesian_prod(*[torch.arange(-a, a + 1, dtype=pos.dtype, device=pos.device) for a in c])
    first = (k[:, 0] > 0) | ((k[:, 0] == 0) & ((k[:, 1] > 0) | ((k[:, 1] == 0) & (k[:, 2] > 0))))
    k = k[first] * (2 * math.pi / box)
    k = k[_dot(k, k) <= top ** 2]
    vol = float(box.prod())

    def recip(kk):
        def energy():
            d = m() + mu
            ph = kk @ pos.T
            co, si = torch.cos(ph), torch.sin(ph)
            kd = kk @ d.T
            re, im = (q * co - kd * si).sum(1), (q * si + kd * co).sum(1)
            k2 = _dot(kk, kk)
            return (4 * math.pi / vol * torch.exp(-k2 / (4 * alpha ** 2)) / k2 * (re ** 2 + im ** 2)).sum()
        return energy

    step = max(1, 16_000_000 // n)
    blocks += [recip(k[a:a + step]) for a in range(0, k.shape[0], step)]

    def own():
        d = m() + mu
        return (-alpha / math.sqrt(math.pi) * (q * q).sum() - 2 * alpha ** 3 / (3 * math.sqrt(math.pi)) * (d * d).sum() -
                math.pi * q.sum() ** 2 / (2 * vol * alpha ** 2))
    return blocks + [own]


def _gradient(sys, pos, mu, parts, of):
    """(energy, gradient) of the functional's electrostatic terms with respect to `of`, block by block."""
    e, g = 0.0, torch.zeros_like(of)
    with torch.enable_grad():
        for block in _variational_energy(sys, pos, mu, parts):
            v = block()
            e += float(v.detach())
            if v.requires_grad:
                g += torch.autograd.grad(v, of)[0]
    return e, g


def _variational_forces(sys, polarization):
    """(energy, forces) of the Ewald mode, or of the variational mode where there is no box."""
    pos, n = sys["pos"], sys["pos"].shape[0]
    none = (False, torch.zeros_like(sys["q"]))
    full = (True, sys["q"])
    zero = torch.zeros((n, 3), dtype=pos.dtype, device=pos.device, requires_grad=True)
    field = -_gradient(sys, pos, zero, full, zero)[1]

    def apply_t(v):
        v = v.clone().requires_grad_(True)
        return -_gradient(sys, pos, v, none, v)[1]

    al = sys["alpha"].unsqueeze(-1)
    mu = al * field if polarization == "direct" else _solve(field, apply_t, sys["alpha"])
    p = pos.clone().requires_grad_(True)
    e, g = _gradient(sys, p, mu, full, p)
    e += float(0.5 * (mu * mu / al).sum())
    if polarization == "direct":
        p = pos.clone().requires_grad_(True)
        e0, g0 = _gradient(sys, p, mu, none, p)
        e, g = e - e0, g - g0
    return e, -g


def _physics(s, case, params=None):
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def t(a):
        return torch.tensor(np.asarray(a), dtype=torch.float64, device=dev)

    q, alpha, thole, mol = params if params is not None else (t(s.charges), t(s.polarizabilities), t(s.tholes),
                                                              t(s.dipoles))
    pos = t(s.positions)
    box = t(s.box) if s.method == S.PME else None
    return {"pos": pos, "q": q, "alpha": alpha, "t": thole, "mol": mol, "m": _lab(pos, mol), "box": box}


def _energy_forces(sys, case):
    pol = case.get("polarization", "mutual")
    if case.get("ewald") or case.get("variational"):
        return _variational_forces(sys, pol)
    return _reference_forces(sys, pol)


def _md_exact(case, seed):
    """One velocity Verlet step of rigid waters (constraints to rounding)."""
    s = _box(case, seed)
    sys = _physics(s, case)
    x = sys["pos"]
    nw = x.shape[0] // 3
    mass = torch.tensor(np.asarray(s.masses), dtype=torch.float64, device=x.device).unsqueeze(-1)
    v = torch.tensor(maxwell_boltzmann(nw, TEMPERATURE, seed), dtype=torch.float64, device=x.device)
    a, b = [0, 0, 1], [1, 2, 2]
    goal = torch.tensor([D_OH, D_OH, D_HH], dtype=torch.float64, device=x.device) ** 2
    sign = torch.zeros((3, 3), dtype=torch.float64, device=x.device)  # of an atom in a constraint
    for k in range(3):
        sign[k, a[k]], sign[k, b[k]] = 1.0, -1.0
    winv = 1.0 / mass.reshape(nw, 3)[0]

    def bonds(p):
        p = p.reshape(nw, 3, 3)
        return p[:, a] - p[:, b]

    def coupled(left, right):
        """Change of the constraints' left . (relative displacement) by unit impulses along `right`."""
        g = torch.einsum("ka,la,a->kl", sign, sign, winv)
        return torch.einsum("wkc,wlc,kl->wkl", left, right, g)

    def push(lam, dirs):
        return torch.einsum("wk,ka,a,wkc->wac", lam, sign, winv, dirs).reshape(-1, 3)

    def rattle(p, vel):
        d = bonds(p)
        rate = (d * bonds(vel)).sum(-1)
        return vel - push(torch.linalg.solve(coupled(d, d), rate), d)

    def forces(p):
        return _energy_forces({**sys, "pos": p, "m": _lab(p, sys["mol"])}, case)

    v = rattle(x, v)
    f = forces(x)[1]
    v = v + 0.5 * DT * f / mass
    old, new = bonds(x), x + DT * v
    for _ in range(20):
        d = bonds(new)
        miss = (d * d).sum(-1) - goal
        shift = push(torch.linalg.solve(2 * coupled(d, old), miss), old)
        new, v = new - shift, v - shift / DT
    e, f = forces(new)
    v = rattle(new, v + 0.5 * DT * f / mass)
    return {"energy": float(e), "forces": f, "positions": new, "velocities": v}


def _fit_exact(parts, seed, system, single):
    """Loss, energies, forces and gradients of one fit step; `parts`: (system, slice of the atoms) of each evaluation."""
    leaves = [p.detach().double().requires_grad_(True) for p in _parameters(system, torch.float32 if single else
                                                                              torch.float64, seed)]
    target = _targets(system.n, torch.float32 if single else torch.float64, seed).double()
    loss, energies, forces = 0.0, [], []
    for s, sl in parts:
        sys = _physics(s, {}, [p[sl] for p in leaves])
        e, f = _reference_forces(sys, "mutual")
        part = ((f - target[sl]) ** 2).sum() / (3 * system.n)
        part.backward()
        loss += float(part.detach())
        energies.append(float(e.detach()))
        forces.append(f.detach())
    return {"loss": loss, "energy": np.array(energies), "forces": torch.cat(forces), "grads": [p.grad for p in leaves]}


def exact(case, seed):
    kind = case["kind"]
    n = 3 * case.get("n_side", 0) ** 3
    if kind == "forces":
        if n > (7000 if case["ewald"] or case["variational"] else 16000):
            return None
        s = _box(case, seed)
        with torch.no_grad():
            e, f = _energy_forces(_physics(s, case), case)
        return {"energy": float(e), "forces": f}
    if kind == "md":
        if n > (3200 if case["ewald"] else 12500):
            return None
        with torch.no_grad():
            return _md_exact(case, seed)
    if kind == "clusters":
        e, f = [], []
        with torch.no_grad():
            for s in _cluster_list(case, seed):
                ec, fc = _reference_forces(_physics(s, case), "mutual")
                e.append(float(ec))
                f.append(fc)
        return {"energies": np.array(e), "forces": torch.cat(f)}
    if kind == "fit_clusters":
        if case["count"] > 256:
            return None
        clusters = _cluster_list(case, seed)
        system, offs = S.concat_clusters(clusters)
        return _fit_exact([(c, slice(int(offs[k]), int(offs[k + 1]))) for k, c in enumerate(clusters)], seed, system,
                          case["precision"] == "mixed")
    if kind == "fit_box":
        if n > 1024:
            return None
        s = _box(case, seed)
        got = _fit_exact([(s, slice(0, s.n))], seed, s, case["precision"] == "mixed")
        return {**got, "energy": float(got["energy"][0])}
    if n > 16000:
        return None
    s = _box(case, seed)
    with torch.no_grad():
        sys = _physics(s, case)
        dip = sys["m"] + _induced(sys, "mutual")
        grid = torch.tensor(_grid(case, s, seed), dtype=torch.float64, device=dip.device)
        out = []
        for g in grid.split(max(1, 8_000_000 // sys["pos"].shape[0])):
            d = g.unsqueeze(1) - sys["pos"].unsqueeze(0)
            d = d - sys["box"] * torch.floor(d / sys["box"] + 0.5)
            rinv = _dot(d, d).rsqrt()
            out.append((rinv * sys["q"] + rinv ** 3 * torch.einsum("gac,ac->ga", d, dip)).sum(1))
        return {"potential": torch.cat(out)}
