"""The work that a user of qcdgpu_b200 has it do, as cases to be timed.

Each case is a run as the package's drivers and README make it, through the
public Python binding and the C-ABI it wraps:

  chain    sweeps of one lattice with the observables every few sweeps, then
           the configuration back on the host (the run a results file and a
           saved state come from);
  observe  the observables of a given configuration (a stored one that is
           analysed), without updates;
  store    a configuration in from the host, checked, reunitarised, measured
           and back out (resuming and saving a run);
  scan     many lattices of different sizes and couplings in one batch;
  learned  training steps of the learned proposal on heatbath configurations
           and Metropolis sweeps with it.

Extents are even (the checkerboard needs it across the periodic wrap) and,
in the drawn cases, mostly not powers of two.
"""
import ctypes
import math

import numpy as np
import torch

import qcdgpu_b200 as Q

DP = ctypes.POINTER(ctypes.c_double)


# ------------------------------------------------------------------- cases
def listed():
    return [
        # one heatbath sweep and its plaquette on the smallest lattice the tests use, with the reference's own
        # settings (FP64 links, RANLUX): launches and latency
        {"name": "chain_su3_4x4_step", "kind": "chain", "group": 3, "n1": 4, "n2": 4, "n3": 4, "n4": 4, "fp64": True,
         "ranlux": True, "beta": 6.0, "n_or": 0, "sweeps": 1, "every": 1, "tune": False, "loops": 0},
        # the SU(2) 8^4 run: FP64, 1 heatbath + 2 overrelaxation, plaquette and Polyakov loop every sweep
        {"name": "chain_su2_8x4_fp64", "kind": "chain", "group": 2, "n1": 8, "n2": 8, "n3": 8, "n4": 8, "fp64": True,
         "ranlux": False, "beta": 2.3, "n_or": 2, "sweeps": 10, "every": 1, "tune": False, "loops": 0},
        # the finite-temperature run: SU(3) 24^3 x 6, observables every sweep
        {"name": "chain_su3_24x24x24x6", "kind": "chain", "group": 3, "n1": 24, "n2": 24, "n3": 24, "n4": 6,
         "fp64": False, "ranlux": False, "beta": 5.9, "n_or": 4, "sweeps": 10, "every": 1, "tune": False, "loops": 0},
        # the headline run: SU(3) 32^4 beta = 6, FP32 links, 1 heatbath + 4 overrelaxation, tuned launch shapes
        {"name": "chain_su3_32x4", "kind": "chain", "group": 3, "n1": 32, "n2": 32, "n3": 32, "n4": 32, "fp64": False,
         "ranlux": False, "beta": 6.0, "n_or": 4, "sweeps": 20, "every": 5, "tune": True, "loops": 0},
        # the same lattice in the reference's arithmetic: FP64 links, RANLUX, heatbath only
        {"name": "chain_su3_32x4_fp64_ranlux", "kind": "chain", "group": 3, "n1": 32, "n2": 32, "n3": 32, "n4": 32,
         "fp64": True, "ranlux": True, "beta": 6.0, "n_or": 0, "sweeps": 10, "every": 2, "tune": True, "loops": 0},
        # SU(2) on a large lattice, FP32
        {"name": "chain_su2_32x4", "kind": "chain", "group": 2, "n1": 32, "n2": 32, "n3": 32, "n4": 32, "fp64": False,
         "ranlux": False, "beta": 2.4, "n_or": 4, "sweeps": 20, "every": 5, "tune": True, "loops": 0},
        # the large lattice: SU(3) 64^4, plaquette, Polyakov loop and all Wilson loops up to 8 x 8 every 10 sweeps
        {"name": "chain_su3_64x4_loops", "kind": "chain", "group": 3, "n1": 64, "n2": 64, "n3": 64, "n4": 64,
         "fp64": False, "ranlux": False, "beta": 6.2, "n_or": 4, "sweeps": 10, "every": 10, "tune": True, "loops": 8},
        # every observable of the reference's results file on a 32^4 FP64 configuration: plaquette, action and
        # Polyakov loop with their profiles, F_munu of both fields, the 7 x 2 Wilson loop
        {"name": "observe_su3_32x4_fp64", "kind": "observe", "group": 3, "n1": 32, "n2": 32, "n3": 32, "n4": 32,
         "fp64": True, "beta": 6.0, "set": "results", "r": 7, "t": 2},
        # the static-potential analysis of a ragged FP32 configuration: all loops, with FP64 products
        {"name": "observe_su3_ragged_loops", "kind": "observe", "group": 3, "n1": 20, "n2": 18, "n3": 22, "n4": 14,
         "fp64": False, "beta": 6.0, "set": "loops", "r": 6, "t": 6},
        # a stored configuration in, checked, reunitarised, measured, out
        {"name": "store_su3_32x4", "kind": "store", "group": 3, "n1": 32, "n2": 32, "n3": 32, "n4": 32, "fp64": False,
         "beta": 6.0},
        # the beta scan: 64 ensembles, N_s in {16,20,24,32}, N_t in {4,6,8}, observables every sweep
        {"name": "scan_64", "kind": "scan", "ensembles": 64, "n_or": 4, "sweeps": 10, "every": 1, "pick": 54},
        # the learned proposal on 16^4: heatbath sweep + 2 training steps a configuration, then Metropolis sweeps
        {"name": "learned_16x4", "kind": "learned", "n1": 16, "n2": 16, "n3": 16, "n4": 16, "beta": 5.7,
         "configs": 4, "steps": 2, "mh_sweeps": 4, "nhit": 4},
    ]


def draw(rng):
    def even(lo, hi):
        return 2 * max(1, round(0.5 * math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["chain", "chain", "chain", "observe", "observe", "store", "scan", "learned"])
    if kind == "scan":
        return {"kind": kind, "ensembles": even(4, 64) + rng.randint(0, 1), "n_or": rng.randint(0, 4),
                "sweeps": rng.randint(2, 10), "every": rng.choice([1, 2]), "pick": rng.randint(1, 10 ** 6)}
    side = even(4, 40)
    n = [max(4, side + 2 * rng.randint(-2, 2)) for _ in range(3)]
    n4 = rng.choice([4, 6, 8, max(4, side + 2 * rng.randint(-2, 2))])
    c = {"kind": kind, "n1": n[0], "n2": n[1], "n3": n[2], "n4": n4}
    if kind == "learned":
        c.update({"n1": min(n[0], 24), "n2": min(n[1], 24), "n3": min(n[2], 24), "n4": min(n4, 24), "beta": 5.7,
                  "configs": rng.randint(1, 4), "steps": rng.randint(1, 3), "mh_sweeps": rng.randint(1, 6),
                  "nhit": rng.randint(1, 8)})
        return c
    group = rng.choice([2, 3, 3])
    fp64 = rng.random() < 0.4
    beta = round(rng.uniform(2.2, 2.6) if group == 2 else rng.uniform(5.5, 6.4), 3)
    c.update({"group": group, "fp64": fp64, "beta": beta})
    if kind == "chain":
        every = rng.choice([1, 2, 5, 10])
        c.update({"ranlux": rng.random() < 0.3, "n_or": rng.randint(0, 5), "sweeps": every * rng.randint(1, 3),
                  "every": every, "tune": rng.random() < 0.5, "loops": 0})
        if not fp64 and rng.random() < 0.3:
            c["loops"] = rng.randint(2, min(8, min(n), n4))
    elif kind == "observe":
        c.update({"set": rng.choice(["results", "loops"]), "r": rng.randint(1, min(8, min(n))),
                  "t": rng.randint(1, min(8, n4))})
    return c


def size(c):
    return (c["n1"], c["n2"], c["n3"], c["n4"])


def ensembles(c):
    """(size, beta) of a scan's lattices, spread as the package's beta-scan driver spreads them"""
    r = np.random.default_rng(c["pick"])
    nt = r.choice([4, 6, 8], size=c["ensembles"])
    ns = r.choice([16, 20, 24, 32], size=c["ensembles"])
    betas = 5.5 + 0.7 * np.arange(c["ensembles"]) / max(c["ensembles"] - 1, 1)
    return [((int(s), int(s), int(s), int(t)), float(b)) for s, t, b in zip(ns, nt, betas)]


# ----------------------------------------------------------------- prepare
def host_table(L):
    """a page-locked buffer for the reference-layout link table, as a program that saves its runs keeps one"""
    return torch.zeros(L.info().ref_elems, dtype=torch.float64 if L.cfg.precision else torch.float32, pin_memory=True)


def links(c, seed):
    """a smooth random SU(N) field from the seed, complex128 [4][N1][N4][N3][N2][N][N] on the GPU (the reference's
    site order: y fastest, then z, t, x): Gaussian matrices near the unit matrix, orthonormalised -- average
    plaquettes as on an equilibrium configuration"""
    N = c["group"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = (4, c["n1"], c["n4"], c["n3"], c["n2"])
    if N == 2:
        q = 0.35 * torch.randn(shape + (4,), generator=g, device="cuda", dtype=torch.float64)
        q[..., 0] += 1.0
        q /= q.norm(dim=-1, keepdim=True)
        a, b = torch.complex(q[..., 0], q[..., 1]), torch.complex(q[..., 2], q[..., 3])
        return torch.stack([torch.stack([a, b], -1), torch.stack([-b.conj(), a.conj()], -1)], -2)
    z = 0.25 * torch.randn(shape + (2, 3, 2), generator=g, device="cuda", dtype=torch.float64)
    z[..., 0, 0, 0] += 1.0
    z[..., 1, 1, 0] += 1.0
    return su3_rows(torch.view_as_complex(z))


def su3_rows(m):
    """rows 1, 2 of m orthonormalised in that order, row 3 = conj(row 1 x row 2)"""
    u = m[..., 0, :] / m[..., 0, :].abs().square().sum(-1, keepdim=True).sqrt()
    v = m[..., 1, :] - (m[..., 1, :] * u.conj()).sum(-1, keepdim=True) * u
    v = v / v.abs().square().sum(-1, keepdim=True).sqrt()
    return torch.stack([u, v, torch.linalg.cross(u, v).conj()], -2)


def table(c, U, dtype):
    """the reference's link table of U: planes of 4-vectors, rows padded to 64 sites"""
    N, V = c["group"], U[0, ..., 0, 0].numel()
    W = U.reshape(4, V, N, N)
    if N == 2:
        planes = torch.stack([W[..., 0, 0].real, W[..., 0, 1].real, W[..., 0, 0].imag, W[..., 0, 1].imag], -1)[None]
    else:
        planes = torch.stack([
            torch.stack([W[..., 0, 0].real, W[..., 0, 1].real, W[..., 0, 2].real, W[..., 1, 2].real], -1),
            torch.stack([W[..., 0, 0].imag, W[..., 0, 1].imag, W[..., 0, 2].imag, W[..., 1, 2].imag], -1),
            torch.stack([W[..., 1, 0].real, W[..., 1, 1].real, W[..., 1, 0].imag, W[..., 1, 1].imag], -1)])
    rows = (V + 63) // 64 * 64
    t = torch.zeros((planes.shape[0] * 4, rows, 4), dtype=dtype, device=U.device)
    t[:, :V] = planes.reshape(-1, V, 4).to(dtype)
    return t


def stored(c, seed):
    """the configuration as a stored table (link precision) on the GPU; the links it stores, in 64 bits"""
    t = table(c, links(c, seed), torch.float64 if c["fp64"] else torch.float32)
    if c["kind"] == "store":
        # rows off SU(N) by rounding, as sweeps without reunitarisation leave them
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        t = t * (1 + 2e-6 * torch.randn(t.shape, generator=g, device="cuda", dtype=t.dtype))
    return t


def unpack(c, t):
    """the matrices a table stores, complex128 [4][N1][N4][N3][N2][N][N]"""
    V = c["n1"] * c["n2"] * c["n3"] * c["n4"]
    p = t[:, :V].double().reshape(-1, 4, V, 4)
    if c["group"] == 2:
        a, b = torch.complex(p[0, ..., 0], p[0, ..., 2]), torch.complex(p[0, ..., 1], p[0, ..., 3])
        m = torch.stack([torch.stack([a, b], -1), torch.stack([-b.conj(), a.conj()], -1)], -2)
    else:
        u = torch.complex(p[0, ..., :3], p[1, ..., :3])
        v = torch.stack([torch.complex(p[2, ..., 0], p[2, ..., 2]), torch.complex(p[2, ..., 1], p[2, ..., 3]),
                         torch.complex(p[0, ..., 3], p[1, ..., 3])], -1)
        m = torch.stack([u, v, torch.linalg.cross(u, v).conj()], -2)
    return m.reshape(4, c["n1"], c["n4"], c["n3"], c["n2"], c["group"], c["group"])


def series(seed):
    return 1 + seed % 2147483000


def prepare(c, seed):
    if c["kind"] == "scan":
        cfg = Q.default_config(group=3, precision=0, prng=Q.PRNG_PHILOX, n_or=c["n_or"], reunit_every=10,
                               reunit_fp64=1, nhit=10, row_align=64)
        ens = [(s, b, series(seed) + i) for i, (s, b) in enumerate(ensembles(c))]
        B = Q.Batch(cfg, ens, max_measurements=c["sweeps"] // c["every"])
        B.init(Q.START_COLD)
        B.tune()
        n = [12 * ((int(np.prod(s)) + 63) // 64 * 64) * 4 for s, _, _ in ens]
        out = torch.zeros(sum(n), dtype=torch.float32, pin_memory=True)
        return {"c": c, "B": B, "out": out, "at": np.concatenate([[0], np.cumsum(n)]).tolist()}
    learned = c["kind"] == "learned"
    ranlux = c.get("ranlux", False)
    cfg = Q.default_config(
        group=c.get("group", 3), size=size(c), precision=int(c.get("fp64", False)), start=Q.START_COLD,
        prng=Q.PRNG_RANLUX if ranlux else Q.PRNG_PHILOX, beta=c["beta"], randseries=series(seed),
        n_or=c.get("n_or", 0), reunit_every=1 if ranlux else 10, reunit_fp64=1)
    L = Q.Lattice(cfg)
    L.seed()
    if c["kind"] in ("observe", "store"):
        t = stored(c, seed)
        host = t.cpu().pin_memory()
        L.lib.qg_links_upload(L.ctx, host.data_ptr(), Q.LAYOUT_REFERENCE)
        return {"c": c, "L": L, "in": host, "out": host_table(L)}
    L.init()
    if c.get("tune"):
        L.tune()
    L.sweep(5)                                           # away from the cold start
    s = {"c": c, "L": L, "out": host_table(L)}
    if learned:
        r = 0.45 / 1.5
        L.net_set(Q.net_init(seed=7, out_bias=math.log(r / (1 - r))), 1.5)
    L.sync()
    return s


# --------------------------------------------------------------------- run
def configuration(L, out):
    L._ck(L.lib.qg_links_download(L.ctx, out.data_ptr(), Q.LAYOUT_REFERENCE), "qg_links_download")
    return out


def run(s):
    return {"chain": run_chain, "observe": run_observe, "store": run_store, "scan": run_scan,
            "learned": run_learned}[s["c"]["kind"]](s)


def run_chain(s):
    c, L = s["c"], s["L"]
    obs, loops = [], []
    for _ in range(c["sweeps"] // c["every"]):
        L.sweep(c["every"])
        obs.append(L.plaquette_sums() + L.polyakov_sums())
        if c["loops"]:
            loops.append(L.wilson_all(c["loops"], c["loops"], fp64_products=False))
    got = {"observables": np.array(obs), "links": configuration(L, s["out"])}
    if loops:
        got["loops"] = np.array(loops)
    return got


def run_observe(s):
    c, L = s["c"], s["L"]
    if c["set"] == "loops":
        return {"loops": L.wilson_all(c["r"], c["t"]), "plaquette": np.array(L.plaquette_sums()),
                "polyakov": np.array(L.polyakov_sums())}
    pl, pl_prof = L.measure_all()
    po, po_prof = L.measure_all(polyakov=True)
    return {"plaquette": np.array(pl), "action_profiles": np.concatenate(pl_prof), "polyakov": np.array(po),
            "polyakov_profiles": np.concatenate(po_prof), "fmunu": L.fmunu(Q.FMUNU_H), "f0mu": L.fmunu(Q.FMUNU_E),
            "wilson": np.array([L.wilson_sum(c["r"], c["t"])])}


def run_store(s):
    L = s["L"]
    L._ck(L.lib.qg_links_upload(L.ctx, s["in"].data_ptr(), Q.LAYOUT_REFERENCE), "qg_links_upload")
    bad = L.field_check()
    L.reunitarize(fp64=True)
    return {"bad": bad, "plaquette": np.array(L.plaquette_sums()), "links": configuration(L, s["out"])}


def run_scan(s):
    c, B = s["c"], s["B"]
    B.init(Q.START_COLD)
    B.run(c["sweeps"], measure_every=c["every"])
    ser = B.series()
    for e in range(B.n):
        at = s["out"].data_ptr() + 4 * s["at"][e]
        B._ck(B.lib.qg_batch_links_download(B.b, e, ctypes.c_void_p(at)), "qg_batch_links_download")
    return {"series": ser, "links": s["out"]}


def run_learned(s):
    c, L = s["c"], s["L"]
    stats = []
    for _ in range(c["configs"]):
        L.sweep(1)
        stats.append(L.net_train(c["steps"], 2e-3))
    L.mh_sweep(c["mh_sweeps"], nhit=c["nhit"])
    acc, jump, hits = L.mh_stats(reset=True)
    return {"training": np.array(stats), "metropolis": np.array([acc, jump]), "hits": hits,
            "weights": L.net_get()[0], "plaquette": np.array(L.plaquette_sums()),
            "links": configuration(L, s["out"])}


# -------------------------------------------------------------------- work
def work(c):
    """bytes: one update phase reads every link once and writes the V/2 it updates (4.5 V links of traffic: the
    phases follow from one another); an observable reads the links it is made of once; a configuration crosses
    once for each direction it is moved in.  flops: two for each multiply-add of the staple and the subgroup steps
    (update) and of the matrix products of each loop (observables)."""
    if c["kind"] == "scan":
        V = sum(int(np.prod(s)) for s, _ in ensembles(c))
        group, real, n_or = 3, 4, c["n_or"]
    else:
        V = int(np.prod(size(c)))
        group, real, n_or = c.get("group", 3), 8 if c.get("fp64") else 4, c.get("n_or", 0)
    link = (12 if group == 3 else 4) * real
    upd, plq = (3700, 2600) if group == 3 else (420, 500)       # flops a link update, a site's six plaquettes
    field = 4.0 * V * link
    if c["kind"] in ("chain", "scan"):
        meas = c["sweeps"] // c["every"]
        b = c["sweeps"] * (1 + n_or) * 8 * 4.5 * V * link + meas * (field + V * link) + field
        f = c["sweeps"] * (1 + n_or) * 4.0 * V * upd + meas * V * (plq + 216.0)
        if c.get("ranlux"):
            b += c["sweeps"] * 8 * 2 * 0.5 * V * 33 * 16.0
        if c.get("loops"):
            b += meas * field
            f += meas * 3.0 * V * c["loops"] * (216 + c["loops"] * 36)
    elif c["kind"] == "observe":
        mul = 216.0 if group == 3 else 32.0
        if c["set"] == "loops":
            b = 2 * field + V * link
            f = V * (plq + mul) + 3.0 * V * c["r"] * (mul + c["t"] * 36)
        else:
            b = 4 * field + V * link
            f = V * (plq + mul) + 6.0 * V * 3 * mul + 3.0 * V * (c["r"] + c["t"] + 2) * mul
    elif c["kind"] == "store":
        b = 7 * field
        f = V * (plq + 4 * 100.0)
    else:
        b = (c["configs"] * (8 + c["steps"]) + 8 * c["mh_sweeps"]) * 4.5 * V * link + field
        f = (c["configs"] * (8 + c["steps"]) * 0.5 + 4 * c["mh_sweeps"]) * V * 3700.0
        f += 4.0 * c["mh_sweeps"] * V * c["nhit"] * 600.0
    return {"bytes": b, "flops": f}


# --------------------------------------------------------------- tolerance
def tolerance(c):
    """An update chain is a fixed sequence of IEEE operations (the sweeps are reproduced link by link from the seed),
    so what may differ is the order of sums and products of the observables: FP64 throughout for FP64 links; the
    Polyakov loop and the all-loops measurement are products in link precision on FP32 links (32 to 128 factors).
    The learned proposal's weights are BF16 on the device, and a step that moves with them moves the chain."""
    if c["kind"] == "learned":
        return {"rel": 1e-2}
    if c["kind"] == "scan" or not c["fp64"]:
        return {"rel": 1e-5}
    return {"rel": 1e-12}


# ------------------------------------------------------------------- exact
def dag(m):
    return m.conj().transpose(-1, -2)


AXIS = {0: 0, 1: 3, 2: 2, 3: 1}                # direction (x, y, z, t) -> axis of [N1][N4][N3][N2]


def ahead(m, d, n=1):
    return torch.roll(m, -n, AXIS[d]) if n else m


def tr(m):
    return m.diagonal(dim1=-2, dim2=-1).sum(-1)


def gen(P, N, a):
    """-i Tr(P T_a) of the reference's F_munu projections (real part only for SU(2))"""
    if N == 2:
        return torch.complex((P[..., 0, 1].imag, P[..., 0, 1].real, P[..., 0, 0].imag)[a - 1],
                             torch.zeros_like(P[..., 0, 0].real))
    if a == 3:
        return -0.5j * (P[..., 0, 0] - P[..., 1, 1])
    return -0.5j * (P[..., 0, 0] + P[..., 1, 1] - 2 * P[..., 2, 2]) / math.sqrt(3.0)


def exact(c, seed):
    if c["kind"] in ("chain", "scan", "learned"):
        return None                                 # a Monte Carlo chain: each accepted draw decides the next
    N = c["group"]
    U = unpack(c, stored(c, seed))
    if c["kind"] == "store":
        U = su3_rows(U[..., :2, :]) if N == 3 else U / U[..., 0, :].abs().square().sum(-1)[..., None, None].sqrt()
        out = table(c, U, torch.float64).cpu().reshape(-1)
        U = unpack(c, table(c, U, torch.float64 if c["fp64"] else torch.float32))
        return {"bad": None, "plaquette": plaquettes(c, U)[0][:2], "links": out}
    pl, prof = plaquettes(c, U)
    P = U[3].select(1, 0)
    for t in range(1, c["n4"]):
        P = P @ U[3].select(1, t)
    P = tr(P)                                       # [N1][N3][N2]
    q = P.abs().square()
    po = np.array([x.item() for x in (P.real.sum(), P.imag.sum(), q.sum(), (q * q).sum())])
    if c["set"] == "loops":
        return {"loops": all_loops(c, U, range(1, c["r"] + 1), range(1, c["t"] + 1)), "plaquette": pl[:2],
                "polyakov": po}
    pp = np.concatenate([np.stack([P.sum(o).real.cpu(), P.sum(o).imag.cpu()], -1) for o in ((1, 2), (0, 1), (0, 2))])
    return {"plaquette": pl, "action_profiles": prof, "polyakov": po, "polyakov_profiles": pp,
            "fmunu": fmunu(c, U, ((0, 1), (0, 2), (1, 2))), "f0mu": fmunu(c, U, ((0, 3), (1, 3), (2, 3))),
            "wilson": all_loops(c, U, [c["r"]], [c["t"]])[0]}


def plaquette(U, m, n):
    return U[m] @ ahead(U[n], m) @ dag(ahead(U[m], n)) @ dag(U[n])


def plaquettes(c, U):
    b = c["beta"] / c["group"] if c["fp64"] else float(np.float32(c["beta"] / c["group"]))
    sites = [sum(tr(plaquette(U, m, n)).real for m, n in ps)
             for ps in (((0, 1), (0, 2), (1, 2)), ((0, 3), (1, 3), (2, 3)))]
    act = [b * (3 * c["group"] - s) for s in sites]
    prof = []
    for d in (0, 1, 2):
        o = [a for a in range(4) if a != AXIS[d]]
        prof.append(np.stack([a.sum(o).cpu().numpy() for a in act], -1))
    return np.array([x.sum().item() for x in sites + act]), np.concatenate(prof)


def fmunu(c, U, planes):
    got = np.zeros((2, 3, 2))
    for p, (m, n) in enumerate(planes):
        P = plaquette(U, m, n)
        for k, a in enumerate((3, 8 if c["group"] == 3 else 2)):
            z = gen(P, c["group"], a).sum()
            got[k, p] = z.real.item(), z.imag.item()
    return got


def all_loops(c, U, Rs, Ts):
    """sum over sites and the three spatial directions of Re Tr of the R x T loops"""
    got = np.zeros((len(Rs), len(Ts)))
    for i in range(3):
        S = {}
        for r in range(1, max(Rs) + 1):
            S[r] = U[i] if r == 1 else S[r - 1] @ ahead(U[i], i, r - 1)
        for b, T in enumerate(Ts):
            L = U[3]
            for k in range(1, T):
                L = L @ ahead(U[3], 3, k)
            for a, R in enumerate(Rs):
                got[a, b] += tr(L @ ahead(S[R], 3, T) @ dag(ahead(L, i, R)) @ dag(S[R])).real.sum().item()
    return got
