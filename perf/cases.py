"""The work a user has this framework do, as cases that can be timed and compared.

A case is a plain dict; `prepare` makes from it what a host program holds before the call (the
engine context, the trajectory frames in host memory, a trainer, a data set) and `run` makes the
call as such a program does: for the engine one division, `engclear`, one `engconst` per frame,
`engstore`; for the proposal network one loss and gradient; for slvfe one free energy.

The listed cases follow the repository's own workloads (systems.make_workload and bench.py):

  soln_site_w1000      the smallest call: one LJ site in 1000 waters, mesh 32^3, a single frame
                       (solution runs call engconst once per trajectory frame, one target each)
  soln_chain_w4096     a 60-site solute in solution, 4096 waters, mesh 64^3, ten frames of an NPT
                       trajectory, whose cell is another one in every frame
  refs_ring_w512       small reference-solvent frames, 64 insertions, as a first look at a system
  refs_ring_w4096      the headline workload: 12-site ring, 4096 waters, 2000 insertions a frame
  refs_ring_npt        the same system at 500 insertions a frame from an NPT trajectory
  refs_chain_w32768    the largest system: 60-site chain, 32,768 waters, mesh 128^3
  refs_flex_mesh48     a flexible solute inserted as conformations from a file, mesh 48^3 (not a
                       power of two), order 6
  batch_w4096          eight solutes of 13 to 300 sites that share one solvent frame
  learned_200site      insertions of a 200-site solute drawn from the proposal network
  train_4096           the proposal network's loss and gradient on a batch of 4096 samples
  slvfe_1396           the free energy from one data set on the default energy mesh, unmerged
"""
import math

import numpy as np
import torch

from ermod_openacc_b200 import Batch, Engine
from ermod_openacc_b200 import _capi as A
from ermod_openacc_b200 import proposal as P
from ermod_openacc_b200 import slvfe as SF
from ermod_openacc_b200 import systems as S

SPACING = 3.1          # A per water along each box side, as the synthetic boxes have
CORES_HIST = dict(ecdmin=-80.0)   # the 60-site chain's mesh: its charges reach lower energies


def _frames(name, mode, nside, mesh, solute, sites, targets, frames, npt, order=4, mesh2=0, mesh3=0):
    return dict(name=name, kind="frames", mode=mode, nside=nside, mesh1=mesh, mesh2=mesh2 or mesh, mesh3=mesh3 or mesh,
                order=order, solute=solute, sites=sites, targets=targets, frames=frames, npt=npt)


def listed():
    return [
        _frames("soln_site_w1000", "soln", 10, 32, "site", 1, 1, 1, False),
        _frames("soln_chain_w4096", "soln", 16, 64, "chain", 60, 1, 10, True),
        _frames("refs_ring_w512", "refs", 8, 32, "ring", 12, 64, 4, False),
        _frames("refs_ring_w4096", "refs", 16, 64, "ring", 12, 2000, 10, False),
        _frames("refs_ring_npt", "refs", 16, 64, "ring", 12, 500, 8, True),
        _frames("refs_chain_w32768", "refs", 32, 128, "chain", 60, 2048, 2, False),
        _frames("refs_flex_mesh48", "flex", 12, 48, "ring", 12, 1000, 4, False, order=6),
        dict(name="batch_w4096", kind="batch", mode="refs", nside=16, mesh1=64, mesh2=64, mesh3=64, order=4,
             solute="recipe", least=13, most=300, members=8, targets=500, frames=2, npt=False),
        _frames("learned_200site", "learned", 16, 64, "recipe", 200, 4000, 1, False),
        dict(name="train_4096", kind="train", batch=4096),
        dict(name="slvfe_1396", kind="slvfe", samples=500, species=1, group=1),
    ]


def _between(rng, lo, hi):
    """A whole number spread evenly over the logarithm of lo..hi."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any of the kinds above at other sizes, odd and ragged ones among them."""
    kind = rng.choice(("soln", "refs", "refs", "refs", "flex", "batch", "learned", "train", "slvfe"))
    if kind == "train":
        return dict(kind="train", batch=_between(rng, 256, 4096))
    if kind == "slvfe":
        return dict(kind="slvfe", samples=rng.randint(200, 1000), species=rng.choice((1, 2)),
                    group=rng.choice((1, 2, 3, 5)))
    # meshes of about one point per Angstrom and finer, as the box asks for; powers of two and others
    nside = rng.randint(8, 18)
    box = SPACING * nside
    meshes = [k for k in (32, 36, 40, 48, 54, 64, 72) if 0.95 * box <= k <= 1.7 * box]
    if kind == "batch":
        case = dict(kind="batch", mode="refs", nside=nside, order=4, solute="recipe", least=rng.randint(8, 40),
                    most=rng.randint(60, 300), members=rng.randint(2, 8), targets=_between(rng, 32, 500),
                    frames=rng.randint(1, 2), npt=rng.random() < 0.3)
        case["mesh1"] = case["mesh2"] = case["mesh3"] = rng.choice(meshes)
        return case
    if kind == "soln":
        solute, sites = rng.choice((("site", 1), ("ring", 12), ("recipe", rng.randint(2, 64)), ("chain", rng.randint(8, 64))))
        targets, frames = 1, rng.randint(1, 10)
    elif kind == "refs":
        solute, sites = rng.choice((("ring", 12), ("ring", 12), ("recipe", _between(rng, 2, 150)), ("chain", rng.randint(8, 64))))
        targets, frames = _between(rng, 16, 2000), rng.randint(1, 6)
    elif kind == "flex":
        solute, sites = rng.choice((("ring", 12), ("recipe", rng.randint(3, 64))))
        targets, frames = _between(rng, 16, 1500), rng.randint(1, 4)
    else:
        solute, sites = "recipe", rng.randint(1, 200)
        targets, frames = _between(rng, 256, 4000), rng.randint(1, 2)
    case = dict(kind="frames", mode=kind, nside=nside, order=4 if rng.random() < 0.75 else 6, solute=solute, sites=sites,
                targets=targets, frames=frames, npt=rng.random() < 0.4)
    case["mesh1"] = rng.choice(meshes)
    for axis in ("mesh2", "mesh3"):
        case[axis] = case["mesh1"] if rng.random() < 0.7 else rng.choice(meshes)
    return case


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _solute(what, sites, seed):
    if what == "site":
        return S.lj_site()
    if what == "ring":
        return S.benzene_ring()
    if what == "chain":
        return S.random_chain(sites, seed)
    return S.ring_recipe_solute(sites, seed)


def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], axis=1).reshape(n, 3, 3)


def _waters(nside, box, rng, sites=None):
    """(3 nside^3, 3) coordinates of waters on a jittered lattice with random orientations; those
    within 3 A of a solute site are moved radially out of the solute's bounding sphere."""
    w = S.water()
    body = (w.coords - ((w.coords * w.mass).sum(axis=1) / w.mass.sum())[:, None]).T
    g = (np.arange(nside) + 0.5) * (box / nside)
    com = np.stack(np.meshgrid(g, g, g, indexing="ij"), axis=-1).reshape(-1, 3) + rng.normal(0.0, 0.3, (nside ** 3, 3))
    x = np.einsum("nij,kj->nki", _rotations(rng, nside ** 3), body) + com[:, None, :]
    if sites is not None:
        centre = sites.mean(axis=0)
        radius = np.linalg.norm(sites - centre, axis=1).max() + 3.2
        d = x[:, :, None, :] - sites
        d -= box * np.round(d / box)
        near = np.sqrt((d * d).sum(axis=-1)).min(axis=(1, 2)) < 3.0
        out = com[near] - centre
        r = np.linalg.norm(out, axis=1, keepdims=True)
        x[near] += (out / np.maximum(r, 1e-6) * np.maximum(radius + 1.2 - r, 0.0))[:, None, :]
    return x.reshape(-1, 3)


def _trajectory(case, rng, solute=None):
    """[(sitepos, cell)] of the case's frames in host memory, as a trajectory reader hands them over."""
    frames = []
    for _ in range(case["frames"]):
        box = SPACING * case["nside"] * (1.0 + (rng.normal(0.0, 0.002) if case["npt"] else 0.0))
        if solute is None:
            pos = _waters(case["nside"], box, rng)
        else:
            sites = (_rotations(rng, 1)[0] @ np.asarray(solute.coords)).T + box / 2
            pos = np.concatenate([sites, _waters(case["nside"], box, rng, sites)])
        frames.append((pos.astype(np.float32).ravel(), np.diag([box] * 3).astype(np.float32).ravel()))
    return frames


def _system(case, solute, iseed):
    """(parameters, topology, energy mesh settings) of one context."""
    mode, nw = case["mode"], case["nside"] ** 3
    prm = dict(ms1max=case["mesh1"], ms2max=case["mesh2"], ms3max=case["mesh3"], splodr=case["order"], iseed=iseed)
    if mode == "soln":
        topo = S.Topology([solute, S.water()], [1, nw], [A.PT_SOLUTE, A.PT_SOLVENT])
        prm.update(slttype=A.SLT_SOLN, maxins=1, corrcal=0, wgtslf=0)
    elif mode == "flex":
        topo = S.Topology([S.water(), solute], [nw, 1], [A.PT_SOLVENT, A.PT_TEST_FLEX])
        prm.update(slttype=A.SLT_REFS_FLEX, maxins=case["targets"], insposition=A.INSPOS_NOCHANGE,
                   insorient=A.INSROT_NOCHANGE)
    else:
        topo = S.Topology([S.water(), solute], [nw, 1], [A.PT_SOLVENT, A.PT_TEST_RIGID])
        prm.update(maxins=case["targets"])
        if mode == "learned":
            prm.update(proposal=A.PROPOSAL_LEARNED)
    return S.default_params(**prm), topo, CORES_HIST if solute.name.startswith("chain") else {}


def _conformations(case, solute, rng, cell):
    """[targets, sites, 3] conformations of a flexible solute placed over the cell."""
    m, s = case["targets"], solute.nsite
    x = np.asarray(solute.coords).T[None] + rng.normal(0.0, 0.05, (m, s, 3))
    x = np.einsum("nij,nkj->nki", _rotations(rng, m), x - x.mean(axis=1, keepdims=True))
    return (x + rng.uniform(0.0, float(cell[0]), (m, 1, 3))).astype(np.float32)


def _sizes(case, rng):
    """The solutes' site counts of a batch: the range's ends and values between."""
    return [case["least"], case["most"]] + [int(v) for v in rng.integers(case["least"], case["most"] + 1,
                                                                         case["members"] - 2)]


def _inputs(case, seed):
    """Everything prepare and exact start from."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "train":
        # standardised Poisson counts of the local density grid; a tenth of the samples are cavities
        x = (rng.poisson(0.8, (case["batch"], P.NIN)) - 0.8) / math.sqrt(0.8)
        y = (x.mean(axis=1) < np.quantile(x.mean(axis=1), 0.1))
        return dict(x=x.astype(np.float32), y=y.astype(np.float32), params=P.init_params(seed))
    if case["kind"] == "slvfe":
        return _distributions(case, rng)
    if case["kind"] == "batch":
        solutes = [_solute("recipe", n, seed + 17 * j) for j, n in enumerate(_sizes(case, rng))]
        return dict(systems=[_system(case, u, 1000 + seed % 100000 + j) for j, u in enumerate(solutes)],
                    frames=_trajectory(case, rng))
    solute = _solute(case["solute"], case["sites"], seed)
    system = _system(case, solute, 1000 + seed % 100000)
    frames = _trajectory(case, rng, solute if case["mode"] == "soln" else None)
    conf = [_conformations(case, solute, rng, c) for _, c in frames] if case["mode"] == "flex" else [None] * len(frames)
    return dict(systems=[system], frames=frames, conf=conf)


def _mesh(hist):
    """Left edges of the default energy mesh's bins (engproc.F90:171-226)."""
    h = dict(S.DEFAULT_HIST, **hist)
    gap = h["finfac"] * h["ecfbin"]
    lo, fine, mid = h["ecdmin"] - gap, h["ecfmns"] - gap, h["ecdcen"]
    marks = [lo, fine, mid - gap, mid + gap, 2 * mid - fine, h["eccore"] + 2 * mid - fine - mid, h["ecdmax"]]
    steps = [h["eclbin"], h["ecfbin"], h["ec0bin"], h["ecfbin"], h["eclbin"]]
    parts = []
    for r, step in enumerate(steps):
        n = int(math.floor((marks[r + 1] - marks[r]) / step + 0.5))
        parts.append(marks[r] + (marks[r + 1] - marks[r]) / n * np.arange(n))
    n = h["pecore"]        # the core's last edge is ecdmax itself
    parts.append(marks[5] * np.exp(math.log(marks[6] / marks[5]) / (n - 1) * np.arange(n)))
    parts[-1][-1] = marks[6]
    return np.concatenate(parts)


def _distributions(case, rng):
    """rho in solution, rho0 and chi0 in the reference solvent as engstore leaves them after a long run:
    the averages over insertions whose solvent molecules each fall into a bin with the insertion's own
    probabilities; the deepest bins and, in solution, the core stay empty."""
    crd, spec, edist, mean, cols = [], [], [], [], []
    for sp in range(case["species"]):
        n = 4096 if sp == 0 else 512
        c = _mesh({})
        mid = np.append(np.where(c[:-1] < 20.0, 0.5 * (c[1:] + c[:-1]), np.sqrt(np.abs(c[1:] * c[:-1]))), c[-1])
        width = np.append(np.diff(c), c[-1] - c[-2])
        p = width * (np.exp(-np.abs(mid) / 0.01) / 0.01 + 0.02 * np.exp(-np.abs(mid) / 1.5))
        p = np.where(mid > 20.0, 2e-4 / 200, np.where(mid < -8.0, 0.0, p * rng.uniform(0.8, 1.2, len(c))))
        shift = rng.normal(0.0, 0.4, (case["samples"], 1)) * np.tanh(mid / 0.5)
        q = p * np.exp(shift - shift * shift / 2)
        q *= n / q.sum(axis=1, keepdims=True)
        soln = np.where(mid > 12.0, 0.0, p * np.exp(-0.3 * np.tanh(mid / 2.0)))
        crd.append(mid)
        spec.append(np.full(len(c), sp + 1, dtype=np.int32))
        edist.append(soln * (n / soln.sum()))
        mean.append(q.mean(axis=0))
        cols.append(q)
    t = torch.from_numpy(np.concatenate(cols, axis=1))
    t = t.cuda() if torch.cuda.is_available() else t
    chi = (t.T @ t / case["samples"]).cpu().numpy()
    edens, spec = np.concatenate(mean), np.concatenate(spec)
    for sp, m in enumerate(mean):          # multinomial counts: n (n - 1) q q^T + n q
        at = np.nonzero(spec == sp + 1)[0]
        n = 4096 if sp == 0 else 512
        chi[np.ix_(at, at)] *= (n - 1) / n
        chi[at, at] += m
    return dict(edist=np.concatenate(edist), edens=edens, ecorr=chi, crd=np.concatenate(crd), spec=spec,
                aveuv=rng.normal(-5.0, 1.0, case["species"]))


# ---------------------------------------------------------------------------
# what a program holds before the call, and the call
# ---------------------------------------------------------------------------
VOXELS = 32            # voxels a side of the learned proposal, as the benchmark configures it


def prepare(case, seed):
    given = _inputs(case, seed)
    state = dict(given, kind=case["kind"])
    if case["kind"] == "train":
        state["trainer"] = P.Trainer(given["params"], max_batch=4096)
    elif case["kind"] == "slvfe":
        state["group"] = case["group"]
    else:
        state["engines"] = [Engine(*s) for s in given["systems"]]
        if case["mode"] == "learned":
            state["engines"][0].proposal_config(VOXELS, 0.2, P.init_params(seed), feature_cells=VOXELS)
        if case["kind"] == "batch":
            state["batch"] = Batch(state["engines"])
    return state


def _stored(engine):
    """One division's results, as the program writes them to engsln / engref, corref and the tables."""
    out, avediv = engine.engstore()
    kept = {k: out[k] for k in ("edens", "ecorr", "slnuv", "minuv", "maxuv", "engnorm")}
    if engine.params["wgtslf"]:      # without self-energy weights there is no offset
        kept["avediv"] = avediv
    return kept


def run(state):
    if state["kind"] == "train":
        grad, loss = state["trainer"].gradients(state["x"], state["y"])
        return dict(grad=grad, loss=loss)
    if state["kind"] == "slvfe":
        per, total = SF.delta_mu_gpu(state["edist"], state["edens"], state["ecorr"], state["crd"], state["spec"], 300.0,
                                     state["aveuv"], group=state["group"])
        return dict(per=per, total=total)
    engines = state["engines"]
    for e in engines:
        e.engclear()
    if state["kind"] == "batch":
        for i, (pos, cell) in enumerate(state["frames"]):
            state["batch"].engconst(i + 1, pos, cell)
        return [_stored(e) for e in engines]
    engine, energies = engines[0], []
    for i, ((pos, cell), conf) in enumerate(zip(state["frames"], state["conf"])):
        engine.engconst(i + 1, pos, cell, ins_conf=conf)
        if engine.params["slttype"] == A.SLT_SOLN:
            energies.append(engine.flceng)
    out = _stored(engine)
    if energies:
        out["flceng"] = np.stack(energies)
    return out


# ---------------------------------------------------------------------------
# the least a pass has to move and compute
# ---------------------------------------------------------------------------
def _bins(case):
    return len(_mesh(CORES_HIST if case.get("solute") == "chain" else {}))


def work(case):
    """Inputs read once, results written once; of the arithmetic: the site pairs inside the cutoff (40
    operations each), one mesh transform of a target's potential and its sums at the solvent atoms, and
    the correlation matrix's lower half."""
    if case["kind"] == "train":
        n, p = case["batch"], P.layout()["n"]
        return dict(bytes=4.0 * (n * (P.NIN + 1) + 2 * p), flops=6.0 * n * p)
    if case["kind"] == "slvfe":
        n = 1396 * case["species"]
        m = n / case["group"]
        return dict(bytes=8.0 * (n * n + 4 * n), flops=2.0 * n * n + m ** 3 / 3 + 8.0 * m * m)
    nw, frames, e = case["nside"] ** 3, case["frames"], _bins(case)
    mesh = case["mesh1"] * case["mesh2"] * case["mesh3"]
    nbytes = flops = 0.0
    sites = [case["sites"]] if case["kind"] == "frames" else [
        case["least"] + (case["most"] - case["least"]) * j / (case["members"] - 1) for j in range(case["members"])]
    for s in sites:
        m = case["targets"] * frames
        pairs = 3.0 * s * min(float(nw), 4.0 / 3.0 * math.pi * 12.0 ** 3 / SPACING ** 3)
        corr = 0.0 if case["mode"] == "soln" else 1.0
        flops += m * (40.0 * pairs + 2.5 * mesh * math.log2(mesh) + 6.0 * nw * case["order"] ** 3)
        flops += corr * m * e * e
        nbytes += 8.0 * e * (1 + corr * e) + (12.0 * s * m if case["mode"] == "flex" else 0.0)
    return dict(bytes=nbytes + 36.0 * nw * frames, flops=flops)


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _philox(c, key):
    """Philox4x32-10 on arrays of counters."""
    c = [np.asarray(v, dtype=np.uint64) for v in c]
    k0, k1, low = np.uint64(key[0]), np.uint64(key[1]), np.uint64(0xFFFFFFFF)
    for r in range(10):
        if r:
            k0, k1 = (k0 + np.uint64(0x9E3779B9)) & low, (k1 + np.uint64(0xBB67AE85)) & low
        a, b = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(b >> np.uint64(32)) ^ c[1] ^ k0, b & low, (a >> np.uint64(32)) ^ c[3] ^ k1, a & low]
    return np.stack([(v >> np.uint64(8)).astype(np.float64) / 16777216.0 for v in c], axis=-1)


def _insertions(prm, topo, cell, stnum):
    """[maxins, s, 3] rigid solutes at uniform positions and orientations (insertion.F90:116-161, 348-369)."""
    m = prm["maxins"]
    body = topo.bfcoord.reshape(-1, 3).astype(np.float64)
    mass = topo.sitemass[-len(body):].astype(np.float64)
    body = body - (mass[:, None] * body).sum(axis=0) / mass.sum()
    key, cnt = (prm["iseed"], 0x45524D44), np.arange(m)
    at = lambda attempt, tag: _philox([cnt, np.full(m, stnum), np.full(m, attempt), np.full(m, tag)], key)  # noqa: E731
    com = at(0, 0)[:, :3] @ cell.T
    q = np.zeros((m, 4))
    open_ = np.ones(m, dtype=bool)
    for attempt in range(1, 65):
        t = at(attempt, 1) * 2.0 - 1.0
        take = open_ & ((t * t).sum(axis=1) < 1.0)
        q[take] = t[take]
        open_ &= ~take
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    rot = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                    2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                    2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], axis=1).reshape(m, 3, 3)
    return np.einsum("nij,kj->nki", rot, body) + com[:, None, :]


def _spline(u, order):
    """M_n(u + c), c = 0 .. n-1, of offsets u in [0, 1)."""
    w = [torch.ones_like(u)] + [torch.zeros_like(u)] * (order - 1)
    for k in range(2, order + 1):
        new = []
        for c in range(order):
            x = u + c
            new.append((x * w[c] + (k - x) * (w[c - 1] if c else 0.0)) / (k - 1) if c < k else torch.zeros_like(u))
        w = new
    return torch.stack(w, dim=-1)


def _stencil(x, invcl, K, order):
    """Flat mesh indices [.., order^3] and weights of points x [.., 3]."""
    idx, wts = [], []
    for m in range(3):
        f = x @ invcl[m]
        f = (f - torch.floor(f)) * K[m]
        g = torch.floor(f)
        wts.append(_spline(f - g, order))
        idx.append((g.long()[..., None] - torch.arange(order, device=x.device)) % K[m])
    i = (idx[2][..., :, None, None] * K[1] + idx[1][..., None, :, None]) * K[0] + idx[0][..., None, None, :]
    w = wts[2][..., :, None, None] * wts[1][..., None, :, None] * wts[0][..., None, None, :]
    return i.flatten(-3), w.flatten(-3)


def _influence(prm, invcl, volume, K, dev):
    """The smooth-PME influence function on the whole mesh [K3, K2, K1]."""
    order, b = prm["splodr"], []
    node = _spline(torch.zeros(1, dtype=torch.float64, device=dev), order)[0]   # M_n(0 .. n-1)
    for k in K:
        r = torch.arange(k, dtype=torch.float64, device=dev)[:, None] * torch.arange(order - 1, dtype=torch.float64, device=dev)
        a = 2.0 * math.pi * r / k
        b.append((node[1:] * torch.cos(a)).sum(-1) ** 2 + (node[1:] * torch.sin(a)).sum(-1) ** 2)
    n = [torch.where(torch.arange(k, device=dev) <= k // 2, torch.arange(k, device=dev), torch.arange(k, device=dev) - k).double() for k in K]
    v = n[0][None, None, :, None] * invcl[0] + n[1][None, :, None, None] * invcl[1] + n[2][:, None, None, None] * invcl[2]
    r2 = (v * v).sum(-1)
    r2[0, 0, 0] = 1.0
    g = torch.exp(-math.pi ** 2 * r2 / prm["screen"] ** 2) / r2 / math.pi / volume
    g = g / (b[0][None, None, :] * b[1][None, :, None] * b[2][:, None, None])
    g[0, 0, 0] = 0.0
    return g


def _lennard_jones(prm, r2, eps, sg2):
    lw, up = prm["lwljcut"], prm["upljcut"]
    i6 = (sg2 / r2) ** 3
    e = 4.0 * eps * i6 * (i6 - 1.0)
    s = (2.0 * r2 + up ** 2 - 3.0 * lw ** 2) * (r2 - up ** 2) ** 2 / (up ** 2 - lw ** 2) ** 3
    e = torch.where(r2 > lw ** 2, s * e, e)
    return torch.where(r2 > up ** 2, torch.zeros_like(e), e)


def _energies(prm, topo, targets, solvent, molecules, cell, dev):
    """Pair energies [targets, molecules] and self energies [targets]; targets [m, s, 3], solvent [atoms, 3]
    in molecule order, `molecules` [atoms] the molecule of each atom."""
    K = (prm["ms1max"], prm["ms2max"], prm["ms3max"])
    s = targets.shape[1]
    soln = prm["slttype"] == A.SLT_SOLN
    f64 = lambda v: torch.as_tensor(np.array(v, dtype=np.float64), device=dev)  # noqa: E731
    lj = torch.as_tensor(np.asarray(topo.ljtype, dtype=np.int64) - 1, device=dev)
    q = f64(topo.charge)
    qs, ls, qv, lv = (q[:s], lj[:s], q[s:], lj[s:]) if soln else (q[-s:], lj[-s:], q[:-s], lj[:-s])
    nt = topo.ljtype_max
    ene, sg2 = f64(topo.ljene_mat).reshape(nt, nt), f64(topo.ljlensq_mat).reshape(nt, nt)
    box, x, atoms = f64(np.diag(cell)), f64(targets), f64(solvent)
    invcl, volume = torch.diag(1.0 / box), float(torch.prod(box))
    screen, nm = prm["screen"], int(molecules[-1]) + 1
    mol = torch.as_tensor(molecules, device=dev)
    G = _influence(prm, invcl, volume, K, dev)
    ai, aw = _stencil(atoms, invcl, K, prm["splodr"])
    aw = aw * qv[:, None]
    E = torch.zeros((len(x), nm), dtype=torch.float64, device=dev)
    rec = torch.zeros(len(x), dtype=torch.float64, device=dev)
    size, chunk = K[0] * K[1] * K[2], max(1, min(64, int(4e8 / (ai.numel() * 3 + 1)), int(6e8 / (8.0 * K[0] * K[1] * K[2]))))
    for b in range(0, len(x), chunk):
        part = x[b:b + chunk]
        ti, tw = _stencil(part, invcl, K, prm["splodr"])
        grid = torch.zeros((len(part), size), dtype=torch.float64, device=dev)
        grid.scatter_add_(1, ti.flatten(1), (tw * qs[:, None]).flatten(1))
        spec = torch.fft.fftn(grid.view(-1, K[2], K[1], K[0]), dim=(1, 2, 3))
        rec[b:b + chunk] = 0.5 * (G * (spec.real ** 2 + spec.imag ** 2)).sum(dim=(1, 2, 3))
        phi = (torch.fft.ifftn(spec * G, dim=(1, 2, 3)).real * size).reshape(len(part), -1)
        for j in range(len(part)):
            E[b + j].index_add_(0, mol, (phi[j][ai] * aw).sum(-1))
    first = atoms[torch.as_tensor(np.searchsorted(molecules, np.arange(nm)), device=dev)]
    per = len(atoms) // nm
    cut = max(prm["elecut"], prm["upljcut"])
    for t in range(len(x)):
        d = first - x[t, 0]
        d -= box * torch.round(d / box)
        e = x[t] - x[t, 0]
        e -= box * torch.round(e / box)
        reach = cut + float((e * e).sum(-1).max().sqrt()) + 1.1
        near = torch.nonzero((d * d).sum(-1) < reach * reach)[:, 0]
        if not len(near):
            continue
        at = (near[:, None] * per + torch.arange(per, device=dev)).flatten()
        r = atoms[at][:, None, :] - x[t]
        r -= box * torch.round(r / box)
        r2 = (r * r).sum(-1)
        pair = _lennard_jones(prm, r2, ene[lv[at][:, None], ls], sg2[lv[at][:, None], ls])
        rr = r2.sqrt()
        pair = pair + torch.where(rr < prm["elecut"], qv[at][:, None] * qs * torch.erfc(screen * rr) / rr, 0.0)
        E[t].index_add_(0, near, pair.sum(-1).view(-1, per).sum(-1))
    # the solute's own images and background in real space (realcal.F90:669-771)
    own = torch.full((len(x),), -float((qs * qs).sum()) * screen / math.sqrt(math.pi), dtype=torch.float64, device=dev)
    up = torch.triu_indices(s, s, 1, device=dev)
    for b in range(0, len(x), 64):
        d = x[b:b + 64, up[0]] - x[b:b + 64, up[1]]
        d -= box * torch.round(d / box)
        r = (d * d).sum(-1).sqrt()
        own[b:b + 64] -= (qs[up[0]] * qs[up[1]] * torch.erf(screen * r) / r).sum(-1)
    return E, rec, own


def _division(prm, topo, hist, frames, conf, dev):
    """engstore's results of one division in 64 bits."""
    soln = prm["slttype"] == A.SLT_SOLN
    edges = torch.as_tensor(_mesh(hist), device=dev)
    n = len(edges)
    edens = torch.zeros(n, dtype=torch.float64, device=dev)
    ecorr = None if soln else torch.zeros((n, n), dtype=torch.float64, device=dev)
    norm = avslf = smpl = slnuv = 0.0
    voffset, own0, flceng = None, None, []
    lo, hi, slo, shi = math.inf, -math.inf, math.inf, -math.inf
    for i, (pos, c) in enumerate(frames):
        cell = c.reshape(3, 3).astype(np.float64)
        x = pos.reshape(-1, 3).astype(np.float64)
        if soln:
            s = len(x) - 3 * (topo.nummol - 1)
            targets, solvent = x[None, :s], x[s:]
        else:
            solvent = x
            targets = conf[i].astype(np.float64) if conf is not None and conf[i] is not None else _insertions(prm, topo, cell, i + 1)
        E, rec, own = _energies(prm, topo, targets, solvent, np.arange(len(solvent)) // 3, cell, dev)
        if prm["slttype"] == A.SLT_REFS_RIGID:
            own0 = float(own[0]) if own0 is None else own0
            own = torch.full_like(own, own0)
        u0 = rec + own
        slo, shi = min(slo, float(u0.min())), max(shi, float(u0.max()))
        volume = float(np.linalg.det(cell))
        w = torch.full_like(u0, volume)
        avslf += float(w.sum())
        if prm["wgtslf"]:
            voffset = float(u0[0]) if voffset is None else voffset
            w = w * torch.exp(-(u0 - voffset) / prm["temp"])
        bins = torch.searchsorted(edges, E).clamp(max=n) - 1
        count = torch.zeros((len(E), n), dtype=torch.float64, device=dev)
        count.scatter_add_(1, bins, torch.ones_like(E))
        edens += w @ count
        if ecorr is not None:
            ecorr += (count * w[:, None]).T @ count
        norm, smpl = norm + float(w.sum()), smpl + len(E)
        if soln:
            flceng.append([float(E.sum())])
            slnuv += float(w[0] * E.sum())
        lo, hi = min(lo, float(E.min())), max(hi, float(E.max()))
    av = avslf / norm
    out = dict(edens=edens / norm, ecorr=None if ecorr is None else ecorr / norm, engnorm=norm,
               slnuv=np.array([slnuv / norm if soln else 0.0]), minuv=np.array([slo, lo]), maxuv=np.array([shi, hi]))
    if prm["wgtslf"]:
        out["avediv"] = np.array([norm / smpl, voffset + prm["temp"] * math.log(av)])
    if soln:
        out["flceng"] = np.array(flceng)[:, None, :]
    return out


def _gradient(given):
    """Loss and gradient of the proposal network with its weights rounded to BF16."""
    L = P.layout()
    p = torch.from_numpy(given["params"])
    take = lambda k: p[L[k][0]:L[k][0] + L[k][1]]  # noqa: E731
    keys = [("W1", (128, 64)), ("b1", (128,)), ("W2", (128, 128)), ("b2", (128,)), ("W3", (128, 128)), ("b3", (128,)),
            ("w4", (128,)), ("b4", (1,))]
    leaf = []
    for k, shape in keys:
        v = take(k)
        v = v.to(torch.bfloat16) if k[0] in "Ww" else v
        leaf.append(v.double().reshape(shape).requires_grad_(True))
    h = torch.from_numpy(given["x"]).double()
    for l in range(3):
        h = torch.relu(h @ leaf[2 * l].T + leaf[2 * l + 1])
    z = h @ leaf[6] + leaf[7]
    y = torch.from_numpy(given["y"]).double()
    loss = torch.nn.functional.softplus(z).sub(y * z).mean()
    loss.backward()
    return dict(grad=torch.cat([v.grad.flatten() for v in leaf]), loss=float(loss))


def _chmpot(given, group):
    """slvfe's free energy with its default options (slvfe.F90:744-803, 875-1232, 1467-1542)."""
    rd0, rr0, crd, spec = (np.asarray(given[k], dtype=np.float64) for k in ("edist", "edens", "crd", "spec"))
    chi, least = given["ecorr"], (rd0[rd0 > 0].min(), rr0[rr0 > 0].min())
    to, last = [], []
    for p in np.unique(spec):
        idx = np.nonzero(spec == p)[0]
        m = len(idx) // group
        base = (to[-1] + 1) if to else 0
        to += [base + min(j // group, m - 1) for j in range(len(idx))]
        last.append((base + m - 1, idx[-1]))
    M = np.zeros((to[-1] + 1, len(rd0)))
    M[to, np.arange(len(rd0))] = 1.0
    rd, rr, chi = M @ rd0, M @ rr0, M @ chi @ M.T
    mid, sp = (M @ crd) / M.sum(axis=1), (M @ spec) / M.sum(axis=1)
    for k, j in last:
        mid[k] = crd[j]
    kT = 300.0 * 8.314510e-3 / 4.184
    kinds = [np.rint(sp) == p for p in np.unique(spec)]
    number = [np.rint(rd[m].sum()) for m in kinds]
    rho, rho0 = rd.copy(), rr.copy()
    for m, k in zip(kinds, number):
        rho[m] *= k / rho[m].sum()
        rho0[m] *= k / rho0[m].sum()
    corr = np.ones(len(rho))
    for _ in range(100):
        for i in range(len(rho)):
            a = [corr[m] @ chi[m, i] for m in kinds]
            corr[i] = sum(k / v for k, v in zip(number, a) if v > 0) / len(kinds) * rho0[i]
        chi = chi * np.outer(corr, corr)
        if np.abs(corr - 1.0)[rho0 > 0].max() <= 1e-8:
            break
    both = (np.rint(np.minimum(rho / least[0], 10)) >= 1) & (np.rint(np.minimum(rho0 / least[1], 10)) >= 1)
    harm = np.where(rho + rho0 > 0, rho * rho0 / np.where(rho + rho0 > 0, rho + rho0, 1.0), 0.0)
    omega = np.zeros(len(rho))
    omega[both] = -kT * np.log(rho[both] / rho0[both]) - mid[both]
    for i in np.nonzero(~both & (rho > 0))[0]:
        same = both & (np.rint(sp) == np.rint(sp[i]))
        idx = np.nonzero(same)[0]
        below, above = idx[idx < i], idx[idx > i]
        m, k = (below[-1] if len(below) else 0), (above[0] if len(above) else len(rho) - 1)
        j = (m if i - m < k - i else k) if both[m] and both[k] else (m if both[m] else k)
        far = mid[idx] - mid[j]
        far = np.where(idx < i, -far - 2.0 * (mid[j] - mid[i]), far)
        w = np.exp(-far / kT) * harm[idx]
        w /= w.sum()
        x, y = mid[idx], omega[idx]
        mx, my = w @ x, w @ y
        slope = (w @ (x * y) - mx * my) / (w @ (x * x) - mx * mx)
        omega[i] = my + slope * (mid[i] - mx)
    pos = rho0 > 0
    a = np.where(np.outer(pos, pos), chi - np.outer(rho0, rho0), 0.0)
    a[np.diag_indices(len(a))] = np.where(pos, np.diag(a), 1.0)
    diff = -kT * (rho - rho0)
    for m in kinds:
        b = np.nonzero(m & pos)[0]
        a[np.ix_(b, b)] += np.trace(a[np.ix_(b, b)]) / len(b) ** 2
    x = np.linalg.solve(a, np.where(pos, diff, 0.0))
    omega0 = np.where(pos, diff / np.where(pos, rho0, 1.0) - x, 0.0)
    out = []
    for m, av in zip(kinds, given["aveuv"]):
        idx = np.nonzero(m)[0]
        j = [(u, v) for u, v in zip(idx[:-1], idx[1:]) if mid[u] <= 0.0 <= mid[v]][-1]
        low, high = abs(mid[j[0]]), mid[j[1]]
        k = j[0] if high > low + 1e-8 else j[1] if high < low - 1e-8 else (j[0] if rho0[j[0]] >= rho0[j[1]] else j[1])
        r, r0, om, om0 = rho[m], rho0[m], omega[m] / kT, (omega0[m] + x[k]) / kT
        with np.errstate(all="ignore"):
            ls = np.where(om < 0, om + om / np.expm1(-om) + 1.0, om / 2)
            lr = np.where(om0 < 0, np.log1p(-om0) * (1.0 / om0 - 1.0) + 1.0, om0 / 2)
        w = np.where(r >= r0, 1.0, 1.0 - ((r - r0) / np.where(r + r0 > 0, r + r0, 1.0)) ** 2)
        term = -kT * (r - r0) - (omega[m] + mid[m]) * r + kT * (w * ls + (1.0 - w) * lr) * (r - r0)
        out.append(term[(r > 0) | (r0 > 0)].sum() + av)
    return dict(per=np.array(out), total=float(np.sum(out)))


def exact(case, seed):
    given, dev = _inputs(case, seed), _device()
    if case["kind"] == "train":
        return _gradient(given)
    if case["kind"] == "slvfe":
        return _chmpot(given, case["group"])
    if case["kind"] == "frames" and case["mode"] == "learned":
        return None     # which voxel an insertion draws hangs on the network's own rounding
    conf = given.get("conf")
    found = [_division(*system, given["frames"], conf, dev) for system in given["systems"]]
    return found if case["kind"] == "batch" else found[0]
