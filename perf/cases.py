"""The measured workloads of the docking path, over its real range of sizes.

A case names one public call on a seeded synthetic complex:

* ``poses`` / ``poses_host``: energies of given rigid poses, with device
  pointers (a rescoring or sampling loop that keeps its poses on the GPU) or
  with host arrays (one call from a C or Python driver);
* ``remc``: one exchange interval (or a few) of a replica-exchange run that is
  already set up, and its state read back;
* ``batch``: the same for many ligands of uneven sizes against one protein;
* ``served``: requests submitted to a resident server and waited for;
* ``similarity`` / ``similarity_host``: the contact-map similarity matrix of
  trajectory conformations, left on the GPU or returned to the host.

Complexes follow gpudock_b200.synth: a protein of fixed point density packed
around an empty pocket, a random-tree ligand in it, the packaged force field.
The packing of a protein size is made once; the seed draws its coordinate
noise, point types, ligand, template, poses and random streams.
"""
import functools
import math

import numpy as np
import torch

from gpudock_b200 import abi, lib, synth

FLOP_PER_PAIR = 36  # + - x / sqrt exp of the always-executed pair terms


def listed():
    return [
        # one small host call: rescoring a handful of poses; latency decides
        dict(name="pose_call_33", kind="poses_host", n=33, lna=24, pnp=1500, box=3.0),
        # a few thousand poses of the plain complex, e.g. one round of a local search
        dict(name="poses_4k_1500x24", kind="poses", n=4096, lna=24, pnp=1500, box=4.0),
        # the energy sweep at its smallest protein: most points are near the ligand
        dict(name="poses_131k_2000x48", kind="poses", n=131072, lna=48, pnp=2000, box=8.0),
        # the sweep at the first protein size that does not fit shared memory, odd pose count
        dict(name="poses_30k_8000x48", kind="poses", n=30011, lna=48, pnp=8000, box=8.0),
        # the sweep at its largest protein
        dict(name="poses_65k_16000x48", kind="poses", n=65536, lna=48, pnp=16000, box=8.0),
        # a large ligand through host arrays
        dict(name="poses_host_12k_6000x96", kind="poses_host", n=12345, lna=96, pnp=6000,
             box=6.0),
        # the plain form: one complex, one ligand conformation, 8 temperatures
        dict(name="plain_run_1500x24", kind="remc", lna=24, pnp=1500, n_prt=1, n_lig=1, n_tmp=8,
             t_ceil=0.04, spe=10, steps=50),
        # the full replica ensemble: 11 x 50 conformations x 16 temperatures
        dict(name="ensemble_4000x40", kind="remc", lna=40, pnp=4000, n_prt=11, n_lig=50,
             n_tmp=16, t_ceil=0.08, spe=5, steps=5),
        # a screen of uneven ligands against one protein's conformations
        dict(name="batch_24_6000", kind="batch", n=24, lna=12, lna_max=96, pnp=6000, n_prt=4,
             n_lig=4, n_tmp=8, t_ceil=0.04, spe=10, steps=10),
        # a burst of small docking requests on a server with resident proteins
        dict(name="served_16_2000_4000", kind="served", n=16, lna=8, lna_max=80, pnp=2000,
             pnp_max=4000, n_lig=4, n_tmp=8, t_ceil=0.04, spe=10, steps=40),
        # clustering of a short trajectory, host arrays in and out
        dict(name="similarity_600", kind="similarity_host", n=600, lna=40, pnp=4000, n_prt=3,
             n_lig=6),
        # clustering of a long one, matrix left on the GPU
        dict(name="similarity_3001", kind="similarity", n=3001, lna=40, pnp=4000, n_prt=3,
             n_lig=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poses", "poses", "poses_host", "remc", "remc", "batch", "similarity",
                       "similarity_host"])
    lna = rng.randint(8, 96)
    pnp = _log_int(rng, 700, 16000)
    if kind.startswith("poses"):
        most = 5e10 if kind == "poses" else 7e9
        n = min(_log_int(rng, 1, 131072), int(most / (lna * pnp)))
        return dict(kind=kind, n=n, lna=lna, pnp=pnp, box=round(rng.uniform(2.0, 8.0), 2))
    if kind == "remc":
        n_tmp = rng.choice([4, 6, 8, 16])
        n_prt, n_lig = rng.randint(1, 4), _log_int(rng, 1, 20)
        spe = rng.choice([5, 10])
        return dict(kind=kind, lna=lna, pnp=min(pnp, 9000), n_prt=n_prt, n_lig=n_lig, n_tmp=n_tmp,
                    t_ceil=rng.choice([0.04, 0.08]), spe=spe, steps=spe)
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(2, 12), lna=rng.randint(8, 24),
                    lna_max=rng.randint(30, 96), pnp=min(pnp, 7000), n_prt=rng.randint(1, 4),
                    n_lig=rng.randint(1, 4), n_tmp=8, t_ceil=0.04, spe=10, steps=10)
    return dict(kind=kind, n=_log_int(rng, 40, 3001), lna=lna, pnp=min(pnp, 6000),
                n_prt=rng.randint(1, 3), n_lig=rng.randint(1, 6))


# --------------------------------------------------------------------------
# complexes
# --------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _packing(pnp, r_pocket, edge, min_dist):
    rng = np.random.Generator(np.random.PCG64(pnp))
    return synth.pack_points(rng, pnp, edge, min_dist, np.full(3, edge / 2.0), r_pocket)


def _protein(rng, pnp, n_prt, lna):
    """A protein around a pocket that holds a ligand of `lna` atoms."""
    r_pocket = 3.0 + round(2.2 * lna ** (1.0 / 3.0), 1)
    edge = (pnp / synth.DENSITY + 4.0 / 3.0 * math.pi * r_pocket ** 3) ** (1.0 / 3.0)
    base = _packing(pnp, r_pocket, edge, 2.8) + rng.normal(0.0, 0.05, size=(pnp, 3))
    confs = [base] + [base + rng.normal(0.0, 0.5, size=base.shape) for _ in range(n_prt - 1)]
    t, c, d, ele, hpp, hflag, seq3r = synth.protein_types(rng, pnp, synth.raw_ff()[0])
    return dict(xyz=np.stack(confs).astype(np.float32), t=t, c=c, d=d, ele=ele, hpp=hpp,
                hflag=hflag, seq3r=seq3r, center=np.full(3, edge / 2.0, np.float32), edge=edge)


def _complex(seed, lna, pnp, n_prt=1, n_lig=1, protein=None):
    rng = np.random.Generator(np.random.PCG64([seed, lna, pnp]))
    if protein is None:
        protein = _protein(rng, pnp, n_prt, lna)
    spec = synth.ComplexSpec(pnp=pnp, lna=lna, n_prt=len(protein["xyz"]), n_lig=n_lig)
    return synth.make_complex(spec, seed=int(rng.integers(1 << 31)), protein=protein)


def _sizes(case):
    """Atom counts of the ligands of a batch or a burst of requests."""
    return np.linspace(case["lna"], case["lna_max"], case["n"]).round().astype(int).tolist()


def _ladder(case):
    return lib.set_temperature(case["n_tmp"], 0.004, case["t_ceil"])[1]


def _poses(case, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 7]))
    return synth.random_poses(rng, case["n"], box=case["box"])


def _conformations(case, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 8]))
    n = case["n"]
    confs = np.zeros((n, 8), np.float32)
    confs[:, 0] = rng.integers(0, case["n_prt"], n)
    confs[:, 1] = rng.integers(0, case["n_lig"], n)
    confs[:, 2:5] = rng.normal(0.0, 1.5, (n, 3))
    confs[:, 5:8] = rng.normal(0.0, 0.3, (n, 3))
    return confs


def _own_complex(case, seed):
    return _complex(seed, case["lna"], case["pnp"], case.get("n_prt", 1), case.get("n_lig", 1))


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, kind = case, case["kind"]
    if kind == "served":
        s.mb = _ladder(case)
        s.server = lib.Server(steps_per_launch=20)
        s.jobs = []
        rng = np.random.Generator(np.random.PCG64([seed, 9]))
        proteins = []
        for pnp in (case["pnp"], case["pnp_max"]):
            p = _protein(rng, pnp, 1, case["lna_max"])
            first = _complex(seed, case["lna"], pnp, protein=p)
            proteins.append((p, pnp, s.server.add_protein(first)))
        for i, lna in enumerate(_sizes(case)):
            p, pnp, pid = proteins[i % 2]
            s.jobs.append((pid, _complex(seed + i, lna, pnp, n_lig=case["n_lig"], protein=p)))
        s.seed = seed
        return s
    s.stream = torch.cuda.Stream()
    s.ctx = lib.Context(0, s.stream.cuda_stream)
    if kind == "batch":
        rng = np.random.Generator(np.random.PCG64([seed, 9]))
        p = _protein(rng, case["pnp"], case["n_prt"], case["lna_max"])
        cxs = [_complex(seed + i, lna, case["pnp"], n_lig=case["n_lig"], protein=p)
               for i, lna in enumerate(_sizes(case))]
        base = lib.DeviceComplex(s.ctx, cxs[0])
        s.dcx = [base] + [lib.DeviceComplex(s.ctx, cx, share=base, prt_conf0=i % case["n_prt"],
                                            n_prt=1)
                          for i, cx in enumerate(cxs)]
        mb = _ladder(case)
        s.mc = lib.Batch(s.ctx, s.dcx[1:],
                         [abi.mc_params(100000, case["spe"], mb, seed=seed, stream_id=i)
                          for i in range(len(cxs))])
        s.mc.init()
        return s
    s.dcx = lib.DeviceComplex(s.ctx, _own_complex(case, seed))
    if kind == "remc":
        s.mc = lib.Remc(s.dcx, 100000, case["spe"], _ladder(case), seed=seed)
        s.mc.init()
    elif kind in ("poses", "poses_host"):
        s.poses = _poses(case, seed)
        if kind == "poses":
            s.poses = torch.from_numpy(s.poses).cuda()
            s.terms = torch.empty((case["n"], abi.NTERM), dtype=torch.float32, device="cuda")
    else:
        s.confs = _conformations(case, seed)
        if kind == "similarity":
            s.out = torch.empty((case["n"], case["n"]), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return s


def _log(b):
    return dict(energy=b.energy, move=b.movematrix, temperature=b.idx_tmp, accepted=b.acs_mc,
                exchanged=b.acs_temp_exchg)


def run(state):
    case = state.case
    kind = case["kind"]
    if kind == "poses":
        state.dcx.energy_poses_dev(case["n"], state.poses.data_ptr(), state.terms.data_ptr())
        return state.terms
    if kind == "poses_host":
        return state.dcx.energy_poses(state.poses, raw=False)[0]
    if kind == "remc":
        state.mc.run(case["steps"])
        return _log(state.mc.read())
    if kind == "batch":
        state.mc.run(case["steps"])
        logs = [_log(state.mc.read(i)) for i in range(case["n"])]
        return {k: np.concatenate([x[k] for x in logs]) for k in logs[0]}
    if kind == "served":
        ids = [state.server.submit(pid, cx, case["steps"], case["spe"], state.mb, 1,
                                   seed=state.seed, stream_id=i)
               for i, (pid, cx) in enumerate(state.jobs)]
        logs = [_log(state.server.wait(i)) for i in ids]
        return {k: np.concatenate([x[k] for x in logs]) for k in logs[0]}
    if kind == "similarity":
        state.dcx.similarity_matrix_dev(state.confs, state.out.data_ptr())
        return state.out
    return state.dcx.similarity_matrix(state.confs)


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _cell(lna, pnp):
    """Bytes of one protein conformation and one ligand conformation."""
    return 24 * pnp + 20 * lna


def work(case):
    kind = case["kind"]
    if kind in ("poses", "poses_host"):
        return dict(bytes=64 * case["n"] + _cell(case["lna"], case["pnp"]),
                    flops=FLOP_PER_PAIR * case["n"] * case["lna"] * case["pnp"])
    if kind.startswith("similarity"):
        n, lna, pnp = case["n"], case["lna"], case["pnp"]
        # the contact tests, and the product of the n maps (about 1 in 20 of
        # a map's pairs is a contact of some conformation)
        return dict(bytes=32 * n + 4 * n * n + case["n_prt"] * _cell(lna, pnp),
                    flops=9.0 * n * lna * pnp + 2.0 * n * n * (lna * pnp / 20.0))
    if kind == "remc":
        jobs = [(case["lna"], case["pnp"], case["n_prt"] * case["n_lig"] * case["n_tmp"],
                 case["n_prt"])]
    elif kind == "batch":
        jobs = [(a, case["pnp"], case["n_lig"] * case["n_tmp"], 1) for a in _sizes(case)]
    else:
        jobs = [(a, (case["pnp"], case["pnp_max"])[i % 2], case["n_lig"] * case["n_tmp"], 1)
                for i, a in enumerate(_sizes(case))]
    return dict(bytes=sum(2 * 84 * r + p * _cell(a, b) for a, b, r, p in jobs),
                flops=float(FLOP_PER_PAIR * case["steps"] * sum(a * b * r for a, b, r, _ in jobs)))


# --------------------------------------------------------------------------
# the same results in 64 bits
# --------------------------------------------------------------------------
def _rotation(m):
    s1, s2, s3 = (torch.sin(m[:, k]) for k in (3, 4, 5))
    c1, c2, c3 = (torch.cos(m[:, k]) for k in (3, 4, 5))
    return torch.stack([c1 * c2, c1 * s2 * s3 - c3 * s1, s1 * s3 + c1 * c3 * s2,
                        c2 * s1, c1 * c3 + s1 * s2 * s3, c3 * s1 * s2 - c1 * s3,
                        -s2, c2 * s3, c2 * c3], dim=1).reshape(-1, 3, 3)


def _exact_terms(cx, poses, dev):
    """The ten energy terms of each pose (protein and ligand conformation 0)."""
    def t(a):
        return torch.as_tensor(np.array(a, np.float64), device=dev)

    def i(a):
        return torch.as_tensor(np.array(a, np.int64), device=dev)

    f = abi.enepara_to_arrays(cx.ff)
    lt, pt = i(cx.lig_t), i(cx.prt_t)
    tab = {k: t(f[k].reshape(abi.NLT, abi.NPT))[lt][:, pt]
           for k in ("p1a", "p2a", "pmf0", "pmf1", "hdb0", "hdb1")}
    lj0, lj1, el0, el1, a1, b1 = (float(f[k]) for k in ("lj0", "lj1", "el0", "el1", "a1", "b1"))
    q = t(cx.lig_c)[:, None] * t(cx.prt_ele)[None]
    # no H-bond term below 0.1 (there 1 / width may be infinite)
    hb = tab["hdb1"] = torch.where(tab["hdb0"] > 0.1, tab["hdb1"], 0.0)
    flagged = (i(cx.prt_hpcflag) == 1).double() * t(cx.prt_hpp)
    psp = t(cx.psp)[lt][:, i(cx.prt_seq3r)] * (i(cx.prt_c) == 2).double()
    hpl = [t(f[k])[lt] for k in ("hpl0", "hpl1", "hpl2")]
    kde_same = (i(cx.kde_t)[None] == lt[:, None]).double()
    kde_n = kde_same.sum(1)
    mcs = t(cx.mcs_xyz)[:, i(cx.lig_n) + 1]
    mcs_ok = (mcs[..., 0] != float(abi.MCS_INVALID_COORD)).double()
    lig, prt = t(cx.lig_xyz[0]), t(cx.prt_xyz[0])
    center, pocket = t(cx.lig_center), t(cx.pocket_center)
    lna, s2pi = cx.lna, float(np.sqrt(np.float32(2.0) * np.float32(3.1415926535)))
    a, b, w = (t(f[k])[:9] for k in ("a_para", "b_para", "w"))
    out = torch.empty((len(poses), 10), dtype=torch.float64, device=dev)
    step = max(1, int(2.5e7 // (lna * cx.pnp)))
    for k in range(0, len(poses), step):
        m = t(poses[k:k + step])
        x = torch.einsum("bij,aj->bai", _rotation(m), lig) + (m[:, :3] + center)[:, None]
        d2 = ((x[:, :, None, 0] - prt[:, 0]) ** 2 + (x[:, :, None, 1] - prt[:, 1]) ** 2
              + (x[:, :, None, 2] - prt[:, 2]) ** 2)
        d = d2.sqrt()
        d6 = d2 ** 3
        p1 = tab["p1a"] / (d6 * d2 * d)
        raw = torch.empty((len(m), 9), dtype=torch.float64, device=dev)
        raw[:, 0] = ((p1 - tab["p2a"] / d6)
                     / (p1 * lj0 * (1.0 + lj1 * d2) + 1.0)).sum((1, 2)) / lna
        s1 = el1 * d
        raw[:, 1] = (q * torch.where(s1 < 1.0, el0 + s1 * s1 * (a1 + b1 * s1), 1.0 / s1)
                     ).sum((1, 2)) / lna
        dm = d - tab["pmf0"]
        raw[:, 2] = (tab["pmf1"] / (1.0 + torch.exp((6.0 - 0.5 * d) * dm))).sum((1, 2)) / lna
        raw[:, 3] = (psp * (dm <= 0.0)).sum((1, 2)) / lna
        h = (d - tab["hdb0"]) * tab["hdb1"]
        raw[:, 4] = -(hb * torch.exp(-0.5 * h * h)).sum((1, 2)) / lna / s2pi
        u = d2 / 81.0
        poly = 1.0 - u * (3.5 - u * (4.5 - u * (2.5 - 0.5 * u)))
        hs = ((flagged * poly * (d2 <= 81.0)).sum(2) - hpl[0]) / hpl[1]
        raw[:, 5] = (0.5 * hs * hs - hpl[2]).sum(1) / lna
        kd2 = ((x[:, :, None] - t(cx.kde_xyz)) ** 2).sum(3)
        kv = (torch.exp(float(f["kde2"]) * kd2) * kde_same).sum(2) / kde_n.clamp(min=1.0)
        raw[:, 6] = kv.sum(1) / float(f["kde3"]) / lna
        md2 = (((x[:, None] - mcs) ** 2).sum(3) * mcs_ok).sum(2) / mcs_ok.sum(1)
        raw[:, 7] = torch.log((t(cx.mcs_tcc) * md2.sqrt()).sum(1) / cx.pos)
        raw[:, 8] = (center + m[:, :3] - pocket).norm(dim=1)
        e = a * raw + b
        out[k:k + step, :9] = e
        out[k:k + step, 9] = (e * w).sum(1)
    return out


def _exact_similarity(cx, confs, dev):
    n = len(confs)
    c = torch.as_tensor(confs, dtype=torch.float64, device=dev)
    lig = torch.as_tensor(cx.lig_xyz, dtype=torch.float64, device=dev)
    prt = torch.as_tensor(cx.prt_xyz, dtype=torch.float64, device=dev)
    center = torch.as_tensor(np.array(cx.lig_center, np.float64), device=dev)
    pmf0 = np.array(cx.ff.pmf0, np.float64)[cx.lig_t][:, cx.prt_t]
    pmf0 = torch.as_tensor(pmf0, device=dev)
    m = c[:, 2:]
    x = torch.einsum("bij,baj->bai", _rotation(m), lig[c[:, 1].long()])
    x = x + (m[:, :3] + center)[:, None]
    near = []
    step = max(1, int(2e7 // (cx.lna * cx.pnp)))
    for k in range(0, n, step):
        p = prt[c[k:k + step, 0].long()]
        y = x[k:k + step]
        d2 = sum((y[:, :, None, j] - p[:, None, :, j]) ** 2 for j in range(3))
        near.append((d2.sqrt() <= pmf0).reshape(len(y), -1))
    near = torch.cat(near)
    maps = near[:, near.any(0)].double()
    tp = maps @ maps.T
    pop = near.sum(1).double()
    fn, fp = pop[:, None] - tp, pop[None] - tp
    tn = float(cx.lna * cx.pnp) - tp - fn - fp
    q = (tp + fp) * (tp + fn) * (tn + fp) * (tn + fn)
    return torch.where(q > 0, (tp * tn - fp * fn) / q.clamp(min=1.0).sqrt(),
                       torch.full_like(q, 10000.0))


def exact(case, seed):
    """Energies and similarities in 64 bits; Monte Carlo states have no such value."""
    kind = case["kind"]
    if kind.startswith("poses"):
        return _exact_terms(_own_complex(case, seed), _poses(case, seed), "cuda")
    if kind.startswith("similarity"):
        return _exact_similarity(_own_complex(case, seed), _conformations(case, seed), "cuda")
    return None
