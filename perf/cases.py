"""Performance cases of the docking path: GSO runs, pose scoring, the pyDock adjoint and the
final-pose stage, each through the package's public entry points (sparkledock_b200.Docking).

A case is a dict of plain values; `prepare` makes what a user's program holds before the call (a
context with the molecules and tables loaded, starting poses, random draws), `run` is one call of
that program and returns everything it computes.  Molecules are the seeded synthetic complexes of
the package with the atom and swarm counts of its benchmark configurations.
"""
import math

import numpy as np
import torch

import sparkledock_b200 as sd

PRECISION = {"fp64_ref": sd.SD_PREC_FP64_REF, "fp64": sd.SD_PREC_FP64, "mixed": sd.SD_PREC_MIXED}
SCORING = {"dfire": sd.SD_SCORING_DFIRE, "pydock": sd.SD_SCORING_PYDOCK}

# receptor atoms / ligand atoms / swarms of the eight-complex batch
BATCH = ("757/481/130 2039/1440/271 2516/1061/298 2030/1256/294 "
         "3052/1658/336 6058/1138/558 6032/1766/695 6143/633/620")


def listed():
    return [
        # A quick trial of a small peptide-sized pair: few glowworms, so each step is launch latency.
        dict(name="run_tiny", kind="run", complexes="200/100/4", glowworms=50, modes=10, steps=20,
             scoring="dfire", precision="mixed"),
        # The plain FP64 run of the small complex, whose trajectory equals the reference's.
        dict(name="run_small_fp64", kind="run", complexes="757/481/130", glowworms=200, modes=10, steps=5,
             scoring="dfire", precision="fp64"),
        # The ordinary production run: one complex of medium size at the default precision.
        dict(name="run_single", kind="run", complexes="3002/1274/402", glowworms=200, modes=10, steps=4,
             scoring="dfire", precision="mixed"),
        # A screening run: eight complexes of uneven size in one context.
        dict(name="run_batch", kind="run", complexes=BATCH, glowworms=200, modes=10, steps=2,
             scoring="dfire", precision="mixed"),
        # The largest receptor that the configurations dock, with its full swarm count.
        dict(name="run_large", kind="run", complexes="17307/1125/1245", glowworms=200, modes=10, steps=2,
             scoring="dfire", precision="mixed"),
        # A run with the electrostatics + Lennard-Jones scoring, odd swarm size and mode count.
        dict(name="run_pydock", kind="run", complexes="2039/1440/41", glowworms=157, modes=7, steps=4,
             scoring="pydock", precision="mixed"),
        # Scoring a handful of poses between other work (an interactive tool): latency counts.
        dict(name="score_few", kind="score", complexes="3002/1274/16", glowworms=1, modes=10,
             scoring="dfire", precision="mixed"),
        # Rescoring a ranked list at full precision, not a multiple of anything.
        dict(name="score_fp64", kind="score", complexes="2516/1061/4099", glowworms=1, modes=10,
             scoring="dfire", precision="fp64"),
        # Energies and gradients of a large set of poses (the adjoint's benchmark shape).
        dict(name="grad_many", kind="grad", complexes="3002/1274/4096", glowworms=1, modes=10,
             scoring="pydock", precision="mixed"),
        # A few FP64 gradients of a small pair, as an external minimiser asks for them.
        dict(name="grad_few_fp64", kind="grad", complexes="757/481/50", glowworms=1, modes=5,
             scoring="pydock", precision="fp64"),
        # Refinement of the best five poses of each of 402 swarms after a run.
        dict(name="refine", kind="refine", complexes="3002/1274/402", glowworms=5, modes=10, steps=10,
             scoring="pydock", precision="mixed"),
        # The end of a run: cluster the final poses and build the best three models of each swarm.
        dict(name="finish", kind="finish", complexes="757/481/130", glowworms=200, modes=10, steps=40,
             scoring="dfire", precision="fp64"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "score", "score", "grad", "grad", "refine", "finish"])
    nl = _log_int(rng, 100, 1766)
    modes = rng.choice([0, 5, 7, 10, 10, 10])
    if kind == "run":
        scoring = rng.choice(["dfire", "dfire", "dfire", "pydock"])
        precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        glowworms = rng.choice([200, 200, rng.randint(20, 300)])
        steps = rng.randint(1, 6)
        parts = []
        for _ in range(rng.choice([1, 1, 1, 2, 3])):
            nr = _log_int(rng, 200, 17307)
            nl = _log_int(rng, 100, 1766)
            most = max(2, int(150e9 / (min(nr, 4000) * nl * glowworms * steps)))
            parts.append("%d/%d/%d" % (nr, nl, _log_int(rng, 1, min(700, most))))
        return dict(kind=kind, complexes=" ".join(parts), glowworms=glowworms, modes=modes, steps=steps,
                    scoring=scoring, precision=precision)
    if kind == "finish":
        return dict(kind=kind, complexes="%d/%d/%d" % (_log_int(rng, 200, 3002), nl, _log_int(rng, 1, 150)),
                    glowworms=rng.randint(20, 256), modes=modes, steps=rng.randint(5, 20), scoring="dfire",
                    precision="fp64")
    nr = _log_int(rng, 200, 6143)
    if kind == "score":
        return dict(kind=kind, complexes="%d/%d/%d" % (nr, nl, _log_int(rng, 1, 6000)), glowworms=1, modes=modes,
                    scoring=rng.choice(["dfire", "dfire", "pydock"]),
                    precision=rng.choice(["mixed", "mixed", "fp64", "fp64_ref"]))
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "grad":
        return dict(kind=kind, complexes="%d/%d/%d" % (nr, nl, _log_int(rng, 1, 5000)), glowworms=1, modes=modes,
                    scoring="pydock", precision=precision)
    return dict(kind=kind, complexes="%d/%d/%d" % (nr, nl, _log_int(rng, 1, 402)), glowworms=5, modes=modes,
                steps=rng.randint(2, 10), scoring="pydock", precision=precision)


def _sizes(case):
    return [tuple(int(v) for v in part.split("/")) for part in case["complexes"].split()]


def _molecules(case, seed):
    return [sd.SyntheticComplex(nr, nl, ns, case["glowworms"], case["modes"], case["modes"], seed=64 * seed + i + 1)
            for i, (nr, nl, ns) in enumerate(_sizes(case))]


def _draws(case, seed):
    return [sd.gso_draws(seed + i + 1, ns, case["steps"], case["glowworms"])
            for i, (_, _, ns) in enumerate(_sizes(case))]


def prepare(case, seed):
    mols = _molecules(case, seed)
    dock = sd.Docking(mols, sd.synthetic_tables(seed + 2024), scoring=SCORING[case["scoring"]],
                      precision=PRECISION[case["precision"]])
    state = dict(case=case, dock=dock, poses=[m.poses for m in mols])
    if case["kind"] == "run":
        state["draws"] = _draws(case, seed)
    elif case["kind"] == "finish":
        # the swarms as a run leaves them; every eighth atom stands for the backbone (CA) atoms
        nr, nl, ns = _sizes(case)[0]
        state["backbone"] = [(np.arange(n) % 8 == 1).astype(np.int32) for n in (nr, nl)]
        dock.init_state(0, mols[0].poses)
        dock.set_draws(0, _draws(case, seed)[0])
        dock.step(case["steps"])
    else:
        state["poses"] = [mols[0].poses.reshape(-1, mols[0].pose_len)]
    return state


def run(state):
    case, dock, kind = state["case"], state["dock"], state["case"]["kind"]
    if kind == "run":
        for i, (poses, u) in enumerate(zip(state["poses"], state["draws"])):
            dock.init_state(i, poses)
            dock.set_draws(i, u)
        dock.step(case["steps"])
        out = [vars(dock.get_state(i)) for i in range(len(state["poses"]))]
        for o in out:
            del o["step"]  # the count of steps that the caller asked for
        return out
    poses = state["poses"][0]
    precision = PRECISION[case["precision"]]
    if kind == "score":
        score, energy = dock.score_poses(0, poses, precision)
        return dict(score=score, energy=energy)
    if kind == "grad":
        energy, gradient = dock.pydock_grad(0, poses, precision)
        return dict(energy=energy, gradient=gradient)
    if kind == "refine":
        refined, before, after = dock.refine(0, poses, case["steps"], precision=precision)
        return dict(poses=refined, before=before, after=after)
    clusters = dock.cluster(0, *state["backbone"])
    swarms, glowworms = clusters["rep"].shape
    best = [s * glowworms + g for s in range(swarms) for g in clusters["rep"][s, :min(3, clusters["n_clusters"][s])]]
    receptor, ligand = dock.materialise(0, best)
    used = np.arange(glowworms) < clusters["n_clusters"][:, None]  # the entries that sd_cluster defines
    return dict(n_clusters=clusters["n_clusters"], rep=np.where(used, clusters["rep"], -1),
                size=np.where(used, clusters["size"], -1), member=clusters["member"], receptor=receptor, ligand=ligand)


_pairs = {}


def pairs_in_cutoff(nr, nl):
    """Expected atom pairs within 15 A of a starting pose: uniform balls of the molecules' radii, the
    ligand's centre 10 A outside the receptor's surface (sampled once per size)."""
    if (nr, nl) not in _pairs:
        rng = np.random.default_rng(7)

        def ball(n, radius):
            v = rng.normal(size=(n, 3))
            return v / np.linalg.norm(v, axis=1, keepdims=True) * radius * rng.random((n, 1)) ** (1 / 3)

        rec, lig = 2.2 * nr ** (1 / 3), 2.2 * nl ** (1 / 3)
        a = ball(200000, rec)
        b = ball(200000, lig) + np.array([rec + 10.0, 0.0, 0.0])
        _pairs[nr, nl] = float(nr) * nl * float(np.mean(np.sum((a - b) ** 2, axis=1) <= 225.0))
    return _pairs[nr, nl]


def work(case):
    """Each input and output once; 8 operations for each pair's distance inside the cutoff, and those
    of the pair function (none for a table value but its sum; about 30 for the pyDock energy, 45 with
    its forces).  Of a run's poses, those of the first step and about 80 % in each later step."""
    nbytes, flops = 0.0, 0.0
    for nr, nl, ns in _sizes(case):
        n, m = ns * case["glowworms"], case["modes"]
        pose = 8 * (7 + 2 * m)
        nbytes += (nr + nl) * (24 + 24 * m + 8)
        if case["scoring"] == "dfire" and case["kind"] != "finish":
            nbytes += 168 * 168 * 20 * 8
        energy = 8 + (1 if case["scoring"] == "dfire" else 30)
        pairs = pairs_in_cutoff(nr, nl)
        if case["kind"] == "run":
            nbytes += n * (2 * pose + 3 * 8 + 4 * 4 + 24 + 8 * case["steps"])
            flops += n * (1 + 0.8 * (case["steps"] - 1)) * pairs * energy
        elif case["kind"] == "score":
            nbytes += n * (pose + 16)
            flops += n * pairs * energy
        elif case["kind"] == "grad":
            nbytes += n * (pose + 8 + 8 * (6 + 2 * m))
            flops += n * pairs * (8 + 45)
        elif case["kind"] == "refine":
            nbytes += n * (2 * pose + 16)
            flops += n * pairs * ((case["steps"] + 1) * energy + case["steps"] * (8 + 45))
        else:
            backbone = nr // 8 + nl // 8
            nbytes += n * (pose + 12) + 3 * ns * (nr + nl) * 24
            flops += n * (backbone * 60 + 10 * backbone * 8)  # poses, and about ten representatives each
    return dict(bytes=nbytes, flops=flops)


# ---- the same results in plain 64-bit torch ----

EXACT_PAIRS = 1.2e11  # atom pairs that plain torch gets through in some seconds


class _Plain:
    """One complex in 64 bits: brute-force energies of poses, without culling or tables by key."""

    def __init__(self, mol, tables, scoring):
        self.device = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.tensor(np.array(a), device=self.device)  # noqa: E731
        self.nr, self.nl, self.m = mol.n_rec, mol.n_lig, mol.n_modes_rec
        self.rec, self.lig = t(mol.rec_xyz), t(mol.lig_xyz)
        self.rec_modes = t(mol.rec_modes).reshape(self.m, self.nr, 3) * (t(mol.rec_mask) == 1)[None, :, None]
        self.lig_modes = t(mol.lig_modes).reshape(self.m, self.nl, 3) * (t(mol.lig_mask) == 1)[None, :, None]
        self.ref = t(mol.lig_ref)
        self.scoring = scoring
        if scoring == "dfire":
            self.table = torch.cat([t(tables[0]), torch.zeros(32, dtype=torch.float64, device=self.device)])
            self.row, self.col = t(mol.rec_type).long() * 3360, t(mol.lig_type).long() * 20
            # dist_to_bins - 1 of the potential by key = int(2 r - 1)
            self.bins = t([0, 0, 0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 13, 14, 14, 15, 15, 16, 16, 17, 17,
                           18, 18, 19, 19, 20])
        else:
            self.qr, self.ql = t(mol.rec_charge), t(mol.lig_charge)
            self.lr, self.ll = t(mol.rec_lj).long(), t(mol.lig_lj).long()
            eps, sig = t(tables[1]), t(tables[2])
            self.eps = torch.sqrt(eps[:, None] * eps[None, :])
            self.sig2 = (0.5 * (sig[:, None] + sig[None, :])) ** 2

    def rotation(self, poses):
        w, x, y, z = poses[:, 3], poses[:, 4], poses[:, 5], poses[:, 6]
        n2 = w * w + x * x + y * y + z * z
        r = torch.stack([w * w + x * x - y * y - z * z, 2 * (x * y - w * z), 2 * (x * z + w * y),
                         2 * (x * y + w * z), w * w - x * x + y * y - z * z, 2 * (y * z - w * x),
                         2 * (x * z - w * y), 2 * (y * z + w * x), w * w - x * x - y * y + z * z], dim=1)
        return (r / n2[:, None]).reshape(-1, 3, 3)

    def atoms(self, poses):
        rec = self.rec + torch.einsum("pm,mad->pad", poses[:, 7:7 + self.m], self.rec_modes)
        lig = self.lig + torch.einsum("pm,mad->pad", poses[:, 7 + self.m:], self.lig_modes)
        rot = self.rotation(poses)
        arm = torch.einsum("pij,paj->pai", rot, lig)
        return rec, arm + poses[:, None, :3], arm, rot

    def reference_points(self, poses):
        return torch.einsum("pij,j->pi", self.rotation(poses), self.ref) + poses[:, :3]

    def energies(self, poses, gradient=False):
        poses = torch.as_tensor(poses, device=self.device)
        step = max(1, int(6e7 // (self.nr * self.nl)))
        parts = [self._chunk(poses[k:k + step], gradient) for k in range(0, max(1, len(poses)), step)]
        energy = torch.cat([p[0] for p in parts])
        return (energy, torch.cat([p[1] for p in parts])) if gradient else energy

    def _chunk(self, poses, gradient):
        rec, lig, arm, rot = self.atoms(poses)
        d2 = torch.zeros(len(poses), self.nr, self.nl, dtype=torch.float64, device=self.device)
        for k in range(3):
            d2 += (rec[:, :, None, k] - lig[:, None, :, k]) ** 2
        p, i, j = torch.nonzero(d2 <= 225.0, as_tuple=True)
        x = d2[p, i, j]
        energy = torch.zeros(len(poses), dtype=torch.float64, device=self.device)
        if self.scoring == "dfire":
            key = (2.0 * torch.sqrt(x) - 1.0).long().clamp(min=0)
            return (energy.index_add_(0, p, self.table[self.row[i] + self.col[j] + self.bins[key]]),)

        def switch(on, off):
            a = off - x
            inside = (x > on) & (x < off)
            s = torch.where(inside, a * a * (off + 2 * x - 3 * on) / (off - on) ** 3, (x <= on).double())
            return s, torch.where(inside, 6 * a * (on - x) / (off - on) ** 3, torch.zeros_like(x))

        s, ds = switch(196.0, 225.0)
        el = 332.0636 / 4.0 * self.qr[i] * self.ql[j] / (x + 1.0)
        e, de = el * s, -el / (x + 1.0) * s + el * ds
        s, ds = switch(49.0, 64.0)
        eps, sig2 = self.eps[self.lr[i], self.ll[j]], self.sig2[self.lr[i], self.ll[j]]
        v = sig2 / (x + 0.5 * sig2)
        lj, dlj = 4 * eps * (v ** 6 - v ** 3), -4 * eps * (6 * v ** 5 - 3 * v ** 2) * v / (x + 0.5 * sig2)
        energy.index_add_(0, p, e + 0.1 * lj * s)
        if not gradient:
            return (energy,)
        de = de + 0.1 * (dlj * s + lj * ds)
        g = 2.0 * de[:, None] * (rec[p, i] - lig[p, j])  # dE/dr_i of each pair
        on_rec = torch.zeros_like(rec).reshape(-1, 3).index_add_(0, p * self.nr + i, g).reshape(rec.shape)
        on_lig = torch.zeros_like(lig).reshape(-1, 3).index_add_(0, p * self.nl + j, -g).reshape(lig.shape)
        back = torch.einsum("pij,pai->paj", rot, on_lig)
        return energy, torch.cat([on_lig.sum(1), torch.cross(arm, on_lig, dim=2).sum(1),
                                  torch.einsum("mad,pad->pm", self.rec_modes, on_rec),
                                  torch.einsum("mad,pad->pm", self.lig_modes, back)], dim=1)

    def scores(self, energy):
        return -(energy * 0.0157 - 4.7) if self.scoring == "dfire" else -energy


def _extents(cur, other, step):
    delta = other - cur
    n = torch.sqrt((delta * delta).sum(1, keepdim=True))
    return torch.where(n >= 1e-8, cur + delta * (step / n.clamp(min=1e-300)), cur)


def _slerp(cur, other, step):
    cur = cur / torch.sqrt((cur * cur).sum(1, keepdim=True))
    other = other / torch.sqrt((other * other).sum(1, keepdim=True))
    dot = (cur * other).sum(1, keepdim=True)
    cur = torch.where(dot < 0, -cur, cur)
    dot = dot.abs()
    near = cur + step * (other - cur)
    near = near / torch.sqrt((near * near).sum(1, keepdim=True))
    omega = torch.arccos(dot.clamp(max=1.0))
    so = torch.sin(omega).clamp(min=1e-300)
    far = torch.sin((1.0 - step) * omega) / so * cur + torch.sin(step * omega) / so * other
    return torch.where(dot > 0.9995, near, far)


def _swarms(plain, mol, u, steps, glowworms):
    """The GSO trajectory of one complex: every swarm steps on its own, all glowworms at once."""
    P, dev = sd.GsoParams(), plain.device
    S, G, m = mol.n_swarms, glowworms, plain.m
    pos = torch.tensor(np.array(mol.poses), device=dev).reshape(S * G, -1)
    u = torch.tensor(u, device=dev)
    luc = torch.full((S, G), P.initial_luciferin, dtype=torch.float64, device=dev)
    vision = torch.full((S, G), P.initial_vision_range, dtype=torch.float64, device=dev)
    score = torch.zeros(S * G, dtype=torch.float64, device=dev)
    moved = torch.ones(S, G, dtype=torch.bool, device=dev)
    own = torch.arange(G, device=dev).expand(S, G)
    for t in range(steps):
        k = torch.nonzero(moved.reshape(-1))[:, 0]
        score[k] = plain.scores(plain.energies(pos[k]))
        if t == 0:
            ref = plain.reference_points(pos)
        ref[k] = plain.reference_points(pos[k])
        luc = (1.0 - P.rho) * luc + P.gamma * score.reshape(S, G)
        r = ref.reshape(S, G, 3)
        d2 = ((r[:, :, None] - r[:, None]) ** 2).sum(3)
        gain = luc[:, None, :] - luc[:, :, None]
        nbr = (gain > 0) & (d2 < (vision * vision)[:, :, None])
        nnei = nbr.sum(2)
        share = torch.where(nbr, gain, torch.zeros_like(gain))
        reach = torch.cumsum(share / share.sum(2, keepdim=True).clamp(min=1e-300), dim=2)
        first = (nbr & ~(reach < u[:, t, :, None])).int().argmax(2)
        moved = nnei > 0
        select = torch.where(moved, first, own)
        other = pos.reshape(S, G, -1).gather(1, select[:, :, None].expand(S, G, pos.shape[1])).reshape(S * G, -1)
        delta = other[:, :3] - pos[:, :3]
        n = torch.sqrt((delta * delta).sum(1, keepdim=True))
        new = torch.cat([torch.where(n >= 1e-8, pos[:, :3] + delta * (P.translation_step / n.clamp(min=1e-300)),
                                     pos[:, :3]),
                         _slerp(pos[:, 3:7], other[:, 3:7], P.rotation_step),
                         _extents(pos[:, 7:7 + m], other[:, 7:7 + m], P.nmodes_step),
                         _extents(pos[:, 7 + m:], other[:, 7 + m:], P.nmodes_step)], dim=1)
        pos = torch.where(moved.reshape(-1, 1), new, pos)
        vision = (vision + P.beta * (P.max_neighbors - nnei).double()).clamp(0.0, P.max_vision_range)
    ints = lambda v: v.to(torch.int32).cpu().numpy()  # noqa: E731
    out = lambda v, *shape: v.reshape(*shape).cpu().numpy()  # noqa: E731
    return dict(pos=out(pos, S, G, -1), scoring=out(score, S, G), luciferin=out(luc, S, G),
                vision_range=out(vision, S, G), moved=ints(moved),
                nnei_len=ints(nnei), select=ints(select), ligand_reference_pose=out(ref, S, G, 3))


def exact(case, seed):
    sizes = _sizes(case)
    calls = case["steps"] if case["kind"] == "run" else 1
    if case["kind"] == "finish":
        return None  # clusters are whole numbers, and the models depend on a whole run before them
    if sum(nr * nl * ns for nr, nl, ns in sizes) * case["glowworms"] * calls > EXACT_PAIRS:
        return None
    mols, tables = _molecules(case, seed), sd.synthetic_tables(seed + 2024)
    plains = [_Plain(m, tables, case["scoring"]) for m in mols]
    if case["kind"] == "run":
        return [_swarms(p, m, u, case["steps"], case["glowworms"])
                for p, m, u in zip(plains, mols, _draws(case, seed))]
    poses = torch.tensor(mols[0].poses.reshape(-1, mols[0].pose_len))
    if case["kind"] == "grad":
        energy, gradient = plains[0].energies(poses, True)
        return dict(energy=energy.cpu().numpy(), gradient=gradient.cpu().numpy())
    energy = plains[0].energies(poses)
    if case["kind"] == "score":
        return dict(score=plains[0].scores(energy).cpu().numpy(), energy=energy.cpu().numpy())
    # which steps a refinement keeps hangs on the last bits of energies: only its start has a value
    return dict(poses=None, before=energy.cpu().numpy(), after=None)
