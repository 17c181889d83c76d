"""Timed cases: what a program that scores molecules with tmol_b200 asks of it.

A case is one call (or one energy + gradient step) through the public entry
points, on seeded synthetic proteins.  ``listed()`` names twelve, ``draw``
gives more from the same ranges, ``prepare`` builds what the caller holds
before the call, ``run`` makes the call, ``work`` counts the bytes and
operations it cannot do without, and ``exact`` evaluates the same outputs in
64 bits with plain torch and numpy, from the op arguments alone.

Tasks:

``gradient``     energies and gradient through a term's scoring module and
                 autograd: the minimiser's and the learned models' step
``scores``       energies alone, no gradient wanted: ranking decoys
``plan``         energies and gradient in one pass through plans the caller
                 holds: the inner loop of batched minimisation
``block_pairs``  energies of every block pair, and the gradient of their
                 weighted sum: per-residue breakdowns
``rotamers``     energies of every rotamer pair: the packer's tables
``bondsep``      a PoseStack's bond separations from its connectivity
"""

import math

import numpy
import torch

WEIGHTS = {
    "ljlk": (1.0, 0.55, 1.0),
    "elec": (1.0,),
    "lkball": (-0.38, 0.92, -0.33, -0.33),
}
ATOMS_PER_RESIDUE = 17
# the rotamer sets: the native placement first, then resampled chis, a
# quarter of them mutated
MUTATE_FRACTION = 0.25

# per residue of a synthetic pose, energies + gradient: operations on the atom
# pairs in reach (LJ 656 pairs x 64, LK 178 x 111; elec 505 x 61; LK-ball 128
# pairs x 255 and 45 bridged ones x 661)
FLOPS_PER_RESIDUE = {"ljlk": 61700.0, "elec": 30800.0, "lkball": 62300.0}
# per dispatched rotamer pair, energies alone
FLOPS_PER_ROTAMER_PAIR = {"ljlk": 1500.0, "elec": 700.0, "lkball": 1000.0}
# later neighbours of a block (itself included) in a packed pose
NEIGHBOURS = 21.0


def _case(name, task, term, poses, lo, hi, chi_sd=0.0, dtype="float32", max_rots=0):
    return {
        "name": name, "task": task, "term": term, "poses": poses, "residues_lo": lo, "residues_hi": hi,
        "chi_sd": chi_sd, "dtype": dtype, "max_rots": max_rots,
    }


def listed():
    return [
        # one small protein, one evaluation: a design script's or a notebook's call, all latency
        _case("ljlk_1x100", "gradient", "ljlk", 1, 100, 100),
        # the batch the package is tuned on: many copies of a domain-sized protein
        _case("ljlk_64x150", "gradient", "ljlk", 64, 150, 150),
        # a whole structure set of uneven length in one call, the largest batch
        _case("ljlk_uneven_256", "plan", "ljlk", 256, 20, 1000),
        # ranking peptides and fragments without a gradient, odd sizes
        _case("ljlk_scores_200x37", "scores", "ljlk", 200, 37, 37),
        # per-residue breakdown of a few proteins, and its gradient
        _case("ljlk_block_pairs_16x150", "block_pairs", "ljlk", 16, 150, 150),
        # the electrostatic term alone on the tuned batch
        _case("elec_64x150", "gradient", "elec", 64, 150, 150),
        # LK-ball with its waters on the tuned batch
        _case("lkball_64x150", "gradient", "lkball", 64, 150, 150),
        # all three terms, as a minimiser evaluates them on clashing starting structures
        _case("all_32x300_clashing", "plan", "all", 32, 300, 300, chi_sd=30.0),
        # double precision, as finite-difference checks of a new model use it
        _case("ljlk_8x101_float64", "gradient", "ljlk", 8, 101, 101, dtype="float64"),
        # the packer's pair tables: many rotamers on a few proteins
        _case("ljlk_rotamers_16x150", "rotamers", "ljlk", 16, 150, 150, max_rots=31),
        # the same for LK-ball, waters on every rotamer
        _case("lkball_rotamers_8x100", "rotamers", "lkball", 8, 100, 100, max_rots=31),
        # building a PoseStack: bond separations of a batch of uneven length
        _case("bondsep_uneven_128", "bondsep", "", 128, 20, 1000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges."""
    task = rng.choice(["gradient"] * 4 + ["plan"] * 2 + ["scores", "block_pairs", "rotamers", "rotamers", "bondsep"])
    term = rng.choice(["ljlk", "ljlk", "elec", "lkball"])
    dtype = "float32"
    chi_sd = rng.choice([0.0, 0.0, 30.0])
    max_rots = 0
    lo = hi = _log_uniform(rng, 20, 1000)
    total = _log_uniform(rng, 100, 30000)  # residues in the batch
    if task == "gradient" and rng.random() < 0.2:
        dtype, total = "float64", _log_uniform(rng, 100, 1500)
    elif task == "plan":
        if rng.random() < 0.5:
            lo, hi = _log_uniform(rng, 20, 100), _log_uniform(rng, 150, 1000)
        if rng.random() < 0.4:
            term, total = "all", _log_uniform(rng, 100, 9600)
    elif task == "block_pairs":
        lo = hi = _log_uniform(rng, 20, 300)
        total = _log_uniform(rng, 100, 3000)
    elif task == "rotamers":
        lo = hi = _log_uniform(rng, 20, 200)
        max_rots = rng.randint(3, 31)
        total = _log_uniform(rng, 40, 800)
    elif task == "bondsep":
        term, chi_sd = "", 0.0
        lo, hi = 20, _log_uniform(rng, 100, 1000)
        total = _log_uniform(rng, 500, 20000)
    mean = _mean_size(lo, hi)
    poses = max(1, min(256, int(round(total / mean))))
    name = "%s_%s_%dx%d_%d" % (task, term, poses, lo, hi)
    case = _case(name, task, term, poses, lo, hi, chi_sd, dtype, max_rots)
    del case["name"]
    return case


# ---------------------------------------------------------------------------
# inputs


def _mean_size(lo, hi):
    return lo if lo == hi else (hi - lo) / math.log(hi / lo)


def _sizes(case):
    """Residues per pose: the quantiles of the log-uniform distribution over
    [residues_lo, residues_hi], shuffled."""
    n, lo, hi = case["poses"], case["residues_lo"], case["residues_hi"]
    sizes = [int(round(lo * (hi / lo) ** ((k + 0.5) / n))) for k in range(n)]
    return [sizes[k] for k in numpy.random.default_rng(2).permutation(n)]


def _pose_stack(case, seed):
    """(PoseStack, a seed per pose).  The case fixes the sequences, and so the
    outputs' shapes.  The seed draws every dihedral; where the conformations
    shape the outputs too (the packer's dispatch), or do not count (bond
    separations), it turns the poses in space and moves them along the batch
    instead."""
    from tmol_b200.chem.restypes import ResidueTypeSet, default_packed_block_types
    from tmol_b200.pose.builder import build_chain_coords, build_pose_stack, topology_from_sequence
    from tmol_b200.pose.synthetic import random_dihedrals, random_sequence

    sizes = _sizes(case)
    P = len(sizes)
    fixed = case["task"] in ("rotamers", "bondsep")
    rts = ResidueTypeSet.get_default()
    topologies, dihedrals = [], []
    for k, n in enumerate(sizes):
        topologies.append(topology_from_sequence(random_sequence(numpy.random.default_rng([n, k]), n), rts))
        rng = numpy.random.default_rng([n, k] if fixed else [seed, n, k])
        dihedrals.append(random_dihedrals(rng, n, case["chi_sd"]))
    device = torch.device("cuda:0")
    coords = None
    if case["task"] != "bondsep":
        pbt = default_packed_block_types(torch.device("cpu"))
        coords = build_chain_coords(pbt, topologies, *(list(v) for v in zip(*dihedrals)))
        side = max(1, math.ceil(P ** (1.0 / 3.0)))
        for k, c in enumerate(coords):
            cell = 0.0 if fixed else 1000.0 * numpy.array([k % side, (k // side) % side, k // (side * side)])
            coords[k] = c - c.mean(axis=0) + cell
    order = numpy.arange(P)
    if fixed:
        order = numpy.roll(order, seed % P)
        topologies = [topologies[k] for k in order]
        coords = coords and [_turned(coords[k], seed) for k in order]
    return build_pose_stack(topologies, coords, device=device), [int(k) for k in order]


def _turned(x, seed):
    """x under one of the 24 rotations that map the axes onto themselves."""
    axes = [(0, 1, 2), (1, 2, 0), (2, 0, 1)][seed % 3]
    sign = [(1, 1, 1), (1, -1, -1), (-1, 1, -1), (-1, -1, 1)][(seed // 3) % 4]
    y = x[:, axes] * numpy.array(sign)
    return y if seed // 12 % 2 == 0 else numpy.stack([y[:, 1], y[:, 0], -y[:, 2]], axis=1)


def _term(name, device):
    from tmol_b200.score.elec_energy_term import ElecEnergyTerm
    from tmol_b200.score.ljlk_energy_term import LJLKEnergyTerm
    from tmol_b200.score.lkball_energy_term import LKBallEnergyTerm

    return {"ljlk": LJLKEnergyTerm, "elec": ElecEnergyTerm, "lkball": LKBallEnergyTerm}[name](device=device)


def _rotamer_set(case, ps, seeds):
    from tmol_b200.pose.rotamers import synthetic_rotamer_set

    return synthetic_rotamer_set(
        ps, max_rots=case["max_rots"], mutate_fraction=MUTATE_FRACTION, seed=9, pose_seeds=seeds
    )


def _terms_of(case):
    return ("ljlk", "elec", "lkball") if case["term"] == "all" else (case["term"],)


def _pair_weights(case, ps, seed):
    """dL/dE of the block-pair energies: a term weight times a per-pair one."""
    gen = torch.Generator(device=ps.device).manual_seed(seed)
    P, B = ps.n_poses, ps.max_n_blocks
    per_pair = 0.5 + torch.rand((P, B, B), generator=gen, device=ps.device)
    w = torch.tensor(WEIGHTS[case["term"]], device=ps.device)
    return (w[:, None, None, None] * per_pair).to(getattr(torch, case["dtype"]))


def prepare(case, seed):
    """What the calling program holds: coordinates on the GPU and the scoring
    module, the plans (with their work ordered, as a minimiser would before
    its loop), or the PoseStack."""
    ps, seeds = _pose_stack(case, seed)
    device, dtype = ps.device, getattr(torch, case["dtype"])
    state = {"task": case["task"]}
    if case["task"] == "bondsep":
        state["pose_stack"] = ps
        return state
    coords = ps.coords.to(dtype)
    if case["task"] == "rotamers":
        rs = _rotamer_set(case, ps, seeds)
        state["coords"] = rs.coords.to(dtype).contiguous()
        state["module"] = _term(case["term"], device).render_rotamer_scoring_module(ps, rs)
    elif case["task"] == "plan":
        state["coords"] = coords.flatten(0, 1).contiguous()
        state["plans"] = [_plan(name, ps, state["coords"]) for name in _terms_of(case)]
        state["weights"] = [
            torch.tensor(WEIGHTS[name], device=device, dtype=dtype)[:, None].expand(-1, ps.n_poses).contiguous()
            for name in _terms_of(case)
        ]
        for plan, w in zip(state["plans"], state["weights"]):
            plan.balance(lambda: plan.energy_and_gradient(state["coords"], w))
    elif case["task"] == "block_pairs":
        state["coords"] = coords.requires_grad_(True)
        state["module"] = _term(case["term"], device).render_block_pair_scoring_module(ps)
        state["weights"] = _pair_weights(case, ps, seed)
    else:
        state["coords"] = coords.requires_grad_(case["task"] == "gradient")
        state["module"] = _term(case["term"], device).render_whole_pose_scoring_module(ps)
        state["weights"] = torch.tensor(WEIGHTS[case["term"]], device=device, dtype=dtype)[:, None]
    return state


def _plan(name, ps, coords):
    if name == "ljlk":
        from tmol_b200.score.ljlk_energy_term import pose_score_args
        from tmol_b200.score.ljlk_op import LJLKPlan

        return LJLKPlan(coords, pose_score_args(ps, _term(name, ps.device))[:-1])
    if name == "elec":
        from tmol_b200.score.elec_energy_term import elec_pose_score_args
        from tmol_b200.score.elec_op import ElecPlan

        return ElecPlan(coords, elec_pose_score_args(ps, _term(name, ps.device))[:-1])
    from tmol_b200.score.lkball_energy_term import score_args, water_gen_args
    from tmol_b200.score.lkball_op import LKBallPlan

    term = _term("lkball", ps.device)
    return LKBallPlan(coords, water_gen_args(ps, term), score_args(ps, term, None)[:-2])


def run(state):
    """One pass through the public entry points."""
    task = state["task"]
    if task == "bondsep":
        from tmol_b200.pose.bondsep import pose_bondsep

        dense, smallest = pose_bondsep(state["pose_stack"])
        return {"dense": dense, "min": smallest}
    x = state["coords"]
    if task == "rotamers":
        with torch.no_grad():
            scores, indices = state["module"](x)
        return {"scores": scores, "indices": indices}
    if task == "scores":
        with torch.no_grad():
            return {"scores": state["module"](x)}
    if task == "plan":
        out, total = {}, None
        for k, (plan, w) in enumerate(zip(state["plans"], state["weights"])):
            out["scores%d" % k], g = plan.energy_and_gradient(x, w)
            total = g if total is None else total + g
        out["gradient"] = total
        return out
    E = state["module"](x)
    (g,) = torch.autograd.grad((state["weights"] * E).sum(), x)
    return {"scores": E.detach(), "gradient": g}


def work(case):
    """Bytes (inputs and outputs once) and operations of one pass."""
    n_res = case["poses"] * _mean_size(case["residues_lo"], case["residues_hi"])
    real = 8.0 if case["dtype"] == "float64" else 4.0
    P, B = case["poses"], case["residues_hi"]
    if case["task"] == "bondsep":
        return {"bytes": 20.0 * P * B * B + 16.0 * n_res, "flops": 0.0}
    if case["task"] == "rotamers":
        mean = (1 + case["max_rots"]) / 2.0
        pairs = NEIGHBOURS * mean * mean * n_res
        terms = len(WEIGHTS[case["term"]])
        return {
            "bytes": 3 * real * ATOMS_PER_RESIDUE * mean * n_res + pairs * (12.0 + real * terms),
            "flops": pairs * FLOPS_PER_ROTAMER_PAIR[case["term"]],
        }
    n_bytes = 3 * real * ATOMS_PER_RESIDUE * n_res * (1 if case["task"] == "scores" else 2)
    flops = sum(FLOPS_PER_RESIDUE[t] for t in _terms_of(case)) * n_res
    if case["task"] == "scores":
        flops *= 0.6  # energies without derivatives
    if case["task"] == "block_pairs":
        n_bytes += 2 * real * len(WEIGHTS[case["term"]]) * P * B * B
    return {"bytes": n_bytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits, from the op's arguments with plain torch


def exact(case, seed):
    """What ``run`` returns, in float64."""
    if case["task"] == "bondsep":
        return None  # integers only
    ps, seeds = _pose_stack(case, seed)
    if case["task"] == "rotamers":
        return _exact_rotamers(case, ps, seeds)
    coords = ps.coords.to(getattr(torch, case["dtype"])).double()
    total = torch.zeros_like(coords.flatten(0, 1))
    out = {}
    for k, name in enumerate(_terms_of(case)):
        args = _op_args(name, ps)
        x = coords.flatten(0, 1).clone().requires_grad_(case["task"] != "scores")
        weights = (
            _pair_weights(case, ps, seed).double()
            if case["task"] == "block_pairs"
            else torch.tensor(WEIGHTS[name], device=x.device, dtype=torch.float32).double()[:, None].expand(
                -1, ps.n_poses
            )
        )
        E = _exact_pose_term(name, args, x, weights, case["task"] == "block_pairs")
        out["scores%d" % k if case["task"] == "plan" else "scores"] = E
        if x.requires_grad:
            total += x.grad
    if case["task"] == "plan":
        out["gradient"] = total
    elif case["task"] != "scores":
        out["gradient"] = total.reshape(coords.shape)
    return out


def _op_args(name, ps, rotamer_set=None):
    """The op's argument list after the coordinates, by what it means."""
    term = _term(name, ps.device)
    if name == "lkball":
        from tmol_b200.score.lkball_energy_term import rotamer_score_args, score_args, water_gen_args

        a = score_args(ps, term, None) if rotamer_set is None else rotamer_score_args(ps, rotamer_set, term, None)
        w = water_gen_args(ps, term, rotamer_set)
        d = dict(zip(
            ("irc", "min_sep", "seps", "n_atoms", "n_conn", "conn_atom", "n_pol", "n_occ", "pol_occ", "params",
             "intra", "gp", "max_dis"), a[12:25]))
        d["inter"] = d["intra"]
        d["water"] = w[12:]
    else:
        if rotamer_set is None:
            from tmol_b200.score.ljlk_energy_term import pose_score_args as args_of

            a = args_of(ps, term)
        else:
            from tmol_b200.score.ljlk_energy_term import rotamer_score_args

            a = rotamer_score_args(ps, rotamer_set, term)
        keys = {
            "ljlk": ("min_sep", "seps", "n_atoms", "n_heavy", "heavy", "types", "n_conn", "conn_atom", "intra", "lig",
                     "params", "gp", "max_dis"),
            "elec": ("min_sep", "seps", "n_atoms", "charge", "n_conn", "conn_atom", "inter", "intra", "lig", "gp",
                     "max_dis"),
        }[name]
        d = dict(zip(keys, a[12:12 + len(keys)]))
        d.setdefault("inter", d["intra"])
    d.update(zip(
        ("rot_off", "pose_of_atom", "first_rot", "first_bt", "block", "pose", "bt"), a[:7]))
    d["n_rots_for_block"], d["rot_off_for_block"] = a[9], a[10]
    return d


def _rotamer_spheres(args, coords):
    """Each rotamer's bounding sphere in the float32 arithmetic the dispatch
    is defined by (atoms summed in order, no fused operations)."""
    f = numpy.float32
    x = coords.detach().cpu().numpy().astype(f)
    bt, off = args["bt"].cpu().numpy().astype(numpy.int64), args["rot_off"].cpu().numpy().astype(numpy.int64)
    n = numpy.where(bt >= 0, args["n_atoms"].cpu().numpy()[numpy.maximum(bt, 0)], 0)
    c = numpy.zeros((len(bt), 3), f)
    for k in range(int(n.max()) if len(n) else 0):
        has = n > k
        c[has] = c[has] + x[off[has] + k]
    c = c / numpy.maximum(n, 1).astype(f)[:, None]
    d2 = numpy.zeros(len(bt), f)
    for k in range(int(n.max()) if len(n) else 0):
        has = n > k
        d = x[off[has] + k] - c[has]
        d = d * d
        d2[has] = numpy.maximum(d2[has], (d[:, 0] + d[:, 1]) + d[:, 2])
    return c, numpy.sqrt(d2)


def _block_spheres(args, coords):
    """Block spheres around their rotamers' spheres, float32 in order."""
    f = numpy.float32
    c, r = _rotamer_spheres(args, coords)
    nr = args["n_rots_for_block"].cpu().numpy().astype(numpy.int64)
    r0 = args["rot_off_for_block"].cpu().numpy().astype(numpy.int64)
    bc = numpy.zeros(nr.shape + (3,), f)
    for k in range(int(nr.max())):
        has = nr > k
        bc[has] = bc[has] + c[r0[has] + k]
    bc = bc / numpy.maximum(nr, 1).astype(f)[..., None]
    br = numpy.zeros(nr.shape, f)
    for k in range(int(nr.max())):
        has = nr > k
        d = c[r0[has] + k] - bc[has]
        d = d * d
        br[has] = numpy.maximum(br[has], numpy.sqrt((d[:, 0] + d[:, 1]) + d[:, 2]) + r[r0[has] + k])
    return bc, br, nr, r0


def _block_pairs(bc, br, real, reach):
    """(pose, b1, b2 >= b1) of the block pairs whose spheres come within
    reach, in that order."""
    out = []
    f = numpy.float32
    for p in range(real.shape[0]):
        d = bc[p][:, None, :] - bc[p][None, :, :]
        d = d * d
        d2 = (d[..., 0] + d[..., 1]) + d[..., 2]
        thr = (br[p][:, None] + br[p][None, :]) + f(reach)
        hit = numpy.triu(d2 < thr * thr) & real[p][:, None] & real[p][None, :]
        b1, b2 = numpy.nonzero(hit)
        out.append(numpy.stack([numpy.full(len(b1), p), b1, b2]))
    return numpy.concatenate(out, axis=1)


def _rotamer_pairs(pairs, nr, r0):
    """Dispatched rotamer pairs of the block pairs: every rotamer of b1 with
    every one of b2, a block's rotamers with themselves only."""
    p, b1, b2 = pairs
    n1, n2 = nr[p, b1], numpy.where(b1 == b2, 1, nr[p, b2])
    count = n1 * n2
    at = numpy.repeat(numpy.arange(len(p)), count)
    q = numpy.arange(len(at)) - numpy.repeat(numpy.cumsum(count) - count, count)
    i, j = q // n2[at], q % n2[at]
    same = (b1 == b2)[at]
    rot1 = r0[p, b1][at] + i
    return rot1, numpy.where(same, rot1, r0[p, b2][at] + j)


def _atom_pairs(args, x, rot1, rot2, max_dis):
    """(atom row 1, atom row 2, index into rot1, in-block atoms, bond
    separation) of every atom pair nearer than max_dis; within one rotamer
    each pair once."""
    n_atoms, bt, off = args["n_atoms"].long(), args["bt"].long(), args["rot_off"].long()
    A = args["intra"].shape[1]
    t1, t2 = bt[rot1], bt[rot2]
    k = torch.arange(A, device=x.device)
    rows1, rows2 = off[rot1][:, None] + k, off[rot2][:, None] + k
    has1, has2 = k < n_atoms[t1][:, None], k < n_atoms[t2][:, None]
    x1 = x[rows1.clamp(max=x.shape[0] - 1)]
    x2 = x[rows2.clamp(max=x.shape[0] - 1)]
    d2 = sum((x1[:, :, None, c] - x2[:, None, :, c]) ** 2 for c in range(3))
    same = rot1 == rot2
    keep = (d2 < max_dis**2) & has1[:, :, None] & has2[:, None, :]
    keep &= ~same[:, None, None] | (k[:, None] < k[None, :])
    e, a1, a2 = torch.nonzero(keep, as_tuple=True)
    del d2, keep, x1, x2
    # bond separations: within the block type, else through the connections
    sep = args["intra"][t1[e], a1, a2].long()
    other = ~same[e]
    eo, o1, o2 = e[other], a1[other], a2[other]
    p, b1, b2 = args["pose"].long()[rot1[eo]], args["block"].long()[rot1[eo]], args["block"].long()[rot2[eo]]
    best = torch.full_like(eo, 6)
    C = args["conn_atom"].shape[1]
    near = args["min_sep"][p, b1, b2] <= 4
    for u in range(C):
        for v in range(C):
            ok = near & (u < args["n_conn"][t1[eo]]) & (v < args["n_conn"][t2[eo]])
            c1 = args["conn_atom"][t1[eo], u].long().clamp(min=0)
            c2 = args["conn_atom"][t2[eo], v].long().clamp(min=0)
            s = (
                args["inter"][t1[eo], c1, o1].long()
                + args["seps"][p, b1, b2, u, v].long()
                + args["inter"][t2[eo], c2, o2].long()
            )
            best = torch.where(ok & (s < best), s, best)
    sep[other] = best
    return rows1[e, a1], rows2[e, a2], e, (t1[e], a1, t2[e], a2), sep


def _count_pair_weight(sep):
    return torch.where(sep > 4, 1.0, torch.where(sep == 4, 0.2, 0.0)).double()


def _fade(d, x0, p0, m0, x1):
    """Cubic from (x0, p0) with slope m0 to zero value and slope at x1."""
    h = x1 - x0
    t = (d - x0) / h
    m = m0 * h
    return p0 + t * (m + t * (-2 * m - 3 * p0 + t * (m + 2 * p0)))


def _sigma(ri, rj, di, dj, hi, hj, pi, pj, ai, aj, hb, oh, hh):
    pair = (di & aj) | (dj & ai)
    s = torch.where((pi & aj) | (pj & ai), hh, ri + rj)
    return torch.where(pair, torch.where((di & hi) | (dj & hj), oh, hb), s)


def _desolvation(d, r, dg, lam, vol):
    x = d - r
    return -vol * dg / (2 * float(numpy.float32(5.56832799683)) * lam) / (d * d) * torch.exp(-x * x / (lam * lam))


def _desolvation_slope(d, r, dg, lam, vol):
    return _desolvation(d, r, dg, lam, vol) * (-2 / d - 2 * (d - r) / (lam * lam))


def _lk_direction(d, sigma, cc, max_dis, r, dg, lam, vol):
    dm = sigma * 0.89
    dm = torch.where(cc & (dm < 4.2), torch.full_like(dm, 4.2), dm)
    n = torch.floor(20 * dm * dm)
    lo = torch.sqrt((n - 29).clamp(min=0) / 20)
    hi = torch.sqrt((n + 21).clamp(max=405) / 20)
    far = max_dis - 1.5
    flat = _desolvation(dm, r, dg, lam, vol)
    h = hi - lo
    t = (d - lo) / h
    p1, m1 = _desolvation(hi, r, dg, lam, vol), _desolvation_slope(hi, r, dg, lam, vol) * h
    close = flat + t * t * (-m1 - 3 * flat + 3 * p1 + t * (m1 + 2 * flat - 2 * p1))
    dfar = torch.full_like(d, far)
    tail = _fade(d, far, _desolvation(dfar, r, dg, lam, vol), _desolvation_slope(dfar, r, dg, lam, vol), max_dis)
    v = torch.where(d < hi, close, torch.where(d < far, _desolvation(d, r, dg, lam, vol), tail))
    return torch.where(d < lo, flat, v)


def _ljlk_energies(args, x, i, j, atoms, sep):
    t1, a1, t2, a2 = atoms
    par = args["params"].double()
    gp = args["gp"].double().reshape(-1)
    max_dis, lin = gp[0], gp[1]
    q1, q2 = par[args["types"][t1, a1].long()], par[args["types"][t2, a2].long()]
    f1, f2 = q1[:, 5:] != 0, q2[:, 5:] != 0
    sigma = _sigma(q1[:, 0], q2[:, 0], f1[:, 0], f2[:, 0], f1[:, 1], f2[:, 1], f1[:, 2], f2[:, 2], f1[:, 3], f2[:, 3],
                   gp[2], gp[3], gp[4])
    eps = torch.sqrt(q1[:, 1] * q2[:, 1])
    d = (x[i] - x[j]).pow(2).sum(1).sqrt()

    def form(r):
        s6 = (sigma / r) ** 6
        return eps * (s6 * s6 - 2 * s6), eps * 12 * (s6 - s6 * s6) / r

    d_lin = sigma * lin
    dmin = torch.minimum(torch.maximum(max_dis - 1.5, sigma), max_dis - 0.1)
    vl, ml = form(d_lin)
    vm, mm = form(dmin)
    mid = form(torch.maximum(d, d_lin))[0]
    lj = torch.where(d < d_lin, vl + ml * (d - d_lin), torch.where(d < dmin, mid, _fade(d, dmin, vm, mm, max_dis)))
    inside = d < sigma
    atr = torch.where(inside, -eps, lj)
    rep = torch.where(inside, lj + eps, torch.zeros_like(lj))
    cc = f1[:, 4] & f2[:, 4]
    lk = _lk_direction(d, sigma, cc, max_dis, q1[:, 0], q1[:, 2], q1[:, 3], q2[:, 4]) + _lk_direction(
        d, sigma, cc, max_dis, q2[:, 0], q2[:, 2], q2[:, 3], q1[:, 4]
    )
    heavy = _heavy_atoms(args)
    lk = torch.where(heavy[t1, a1] & heavy[t2, a2], lk, torch.zeros_like(lk))
    return _count_pair_weight(sep) * torch.stack([atr, rep, lk])


def _heavy_atoms(args):
    n_heavy, heavy = args["n_heavy"].cpu().numpy(), args["heavy"].cpu().numpy()
    nbt, nt = n_heavy.shape
    heavy = heavy.reshape(nbt, nt, -1)
    out = numpy.zeros((nbt, nt * 32), bool)
    for b in range(nbt):
        for t in range(nt):
            out[b, t * 32 + heavy[b, t, : n_heavy[b, t]]] = True
    return torch.tensor(out, device=args["n_heavy"].device)


def _elec_energies(args, x, i, j, atoms, sep):
    t1, a1, t2, a2 = atoms
    # the dielectric's end points are formed in single precision
    f = numpy.float32
    D, D0, S, lo, hi = (f(v) for v in args["gp"].cpu().numpy().reshape(-1))
    DD0 = float(f(D - D0))
    D_, S_ = float(D), float(S)

    def eps(r):
        return D_ - 0.5 * DD0 * (2 + 2 * r * S_ + r * r * S_ * S_) * (
            torch.exp(-r * S_) if isinstance(r, torch.Tensor) else math.exp(-r * S_)
        )

    def eps_single(r):
        poly, fall = f(2) + f(2) * r * S + r * r * S * S, numpy.exp(-r * S)
        return f(D_ - 0.5 * DD0 * float(poly) * float(fall))

    C1 = 322.0637
    C2 = C1 / float(hi * eps_single(hi))
    flat = C1 / float(lo * eps_single(lo)) - C2

    def coulomb(r):
        e, de = eps(r), 0.5 * DD0 * r * r * S_**3 * math.exp(-r * S_)
        return C1 / (r * e) - C2, -C1 * (e + r * de) / (r * r * e * e)

    lo0, lo1, hi0, hi1 = float(lo) - 0.25, float(lo) + 0.25, float(hi) - 1.0, float(hi)
    d = (x[i] - x[j]).pow(2).sum(1).sqrt()
    v1, m1 = coulomb(lo1)
    t = (d - lo0) / (lo1 - lo0)
    m = m1 * (lo1 - lo0)
    near = flat + t * t * (-m - 3 * flat + 3 * v1 + t * (m + 2 * flat - 2 * v1))
    v0, m0 = coulomb(hi0)
    r = d.clamp(min=lo0)
    f_d = torch.where(d < lo1, near, torch.where(d < hi0, C1 / (r * eps(r)) - C2, _fade(d, hi0, v0, m0, hi1)))
    f_d = torch.where(d < lo0, torch.full_like(d, flat), f_d)
    f_d = torch.where(d < hi1, f_d, torch.zeros_like(d))
    q = args["charge"].double()
    return (_count_pair_weight(sep) * q[t1, a1] * q[t2, a2] * f_d)[None]


def _lkball_tables(args):
    """Per block-type atom: polar, occluder, parameters."""
    n_pol, n_occ = args["n_pol"].cpu().numpy(), args["n_occ"].cpu().numpy()
    inds, par = args["pol_occ"].cpu().numpy(), args["params"].cpu().numpy().astype(numpy.float64)
    nbt, nt = n_pol.shape
    polar, occ = numpy.zeros((nbt, nt * 32), bool), numpy.zeros((nbt, nt * 32), bool)
    p = numpy.zeros((nbt, nt * 32, 9))
    for b in range(nbt):
        for t in range(nt):
            at = t * 32 + inds[b, t, : n_occ[b, t]]
            polar[b, at[: n_pol[b, t]]] = True
            occ[b, at] = True
            p[b, at] = par[b, t, : n_occ[b, t]]
    dev = args["n_pol"].device
    return torch.tensor(polar, device=dev), torch.tensor(occ, device=dev), torch.tensor(p, device=dev)


def _water_sites(args):
    """Every water: (atom row, slot, kind, the rows that place it, torsion,
    angle); kind 1 donor, 2 sp2, 3 sp3, 4 ring."""
    (irc, n_atoms, n_conn, conn_atom, _, bonds, ranges, n_donH, n_acc, donH, donH_hvy, which, acc, hyb, n_H, is_h, gp,
     sp2, sp3, ring) = [t.cpu().numpy() if isinstance(t, torch.Tensor) else t for t in args["water"]]
    tors, angles = {1: sp2.reshape(-1), 2: sp3.reshape(-1), 3: ring.reshape(-1)}, gp.reshape(-1)[1:4]
    bt, pose, block, off = (args[k].cpu().numpy().astype(numpy.int64) for k in ("bt", "pose", "block", "rot_off"))
    first_bt, first_rot = args["first_bt"].cpu().numpy(), args["first_rot"].cpu().numpy()

    def bonded(x, across):
        """Bonded neighbours of x = (hop, block type, atom), hop the
        connections crossed from the water's own block."""
        hop, t, a = x
        if a < 0:
            return
        for e in bonds[t, max(0, ranges[t, a, 0]):min(bonds.shape[1], ranges[t, a, 1])]:
            if e[1] >= 0:
                yield (hop, t, int(e[1]))
            else:
                o = across(hop, int(e[2]))
                if o is not None:
                    yield o

    def bases(x, h, across):
        hydrogen = lambda o: bool(is_h[o[1], o[2]])  # noqa: E731
        near = list(bonded(x, across))
        b = next((o for o in near if not hydrogen(o)), None)
        if h == 1:
            if b is None:
                return None
            b0 = next((o for o in bonded(b, across) if o != x and not (b[0] != x[0] and o[0] == x[0])), None)
        elif h == 2:
            b0 = next((o for o in near if o != b and hydrogen(o)), None)
            b0 = b0 or next((o for o in near if o != b), None) or b
        else:
            b0 = next((o for o in near if o != b and not hydrogen(o)), None)
        return None if b is None or b0 is None or b0 == b else (b, b0)

    found, cache = [], {}
    for r in range(len(bt)):
        t, p, k = int(bt[r]), int(pose[r]), int(block[r])
        if t < 0:
            continue

        def across(hop, c, p=p, k=k):
            at = k if hop is None else hop
            o = irc[p, at, c] if 0 <= c < irc.shape[2] else (-1, -1)
            if o[0] < 0 or o[1] < 0 or first_bt[p, o[0]] < 0:
                return None
            ob = int(first_bt[p, o[0]])
            return (None if o[0] == k else int(o[0]), ob, int(conn_atom[ob, o[1]]))

        around = tuple(
            (int(irc[p, k, c, 0]) - k, int(irc[p, k, c, 1]), int(first_bt[p, irc[p, k, c, 0]]))
            if irc[p, k, c, 0] >= 0 else None for c in range(irc.shape[2])
        )
        key = (t, around)
        if key not in cache:
            sites = []
            for tt in range(n_donH.shape[1]):
                for q in range(n_donH[t, tt]):
                    d, h = int(donH_hvy[t, tt, q]), tt * 32 + int(donH[t, tt, q])
                    sites.append((d, int(which[t, tt, q]), 1, (0, d), (0, h), (0, d), 0.0, 0.0))
                for q in range(n_acc[t, tt]):
                    a, h = tt * 32 + int(acc[t, tt, q]), int(hyb[t, tt, q])
                    got = bases((None, t, a), h, across) if 1 <= h <= 3 else None
                    if got is None:
                        continue
                    rel = [((0 if o[0] is None else o[0] - k), o[2]) for o in got]
                    for w in range(len(tors[h])):
                        slot = w + int(n_H[t, tt, q])
                        if slot < 4:
                            sites.append((a, slot, 1 + h, (0, a), rel[0], rel[1], float(tors[h][w]),
                                          float(angles[h - 1])))
            cache[key] = sites
        for a, slot, kind, xa, xb, xc, tor, ang in cache[key]:
            rows = [
                int(off[r]) + at if hop == 0 else int(off[first_rot[p, k + hop]]) + at for hop, at in (xa, xb, xc)
            ]
            found.append((int(off[r]) + a, slot, kind, rows[0], rows[1], rows[2], tor, ang))
    return numpy.array(found, dtype=numpy.float64).reshape(-1, 8), float(gp.reshape(-1)[0])


def _waters(args, x):
    """Waters [n_atoms, 4, 3] (zeros where there is none) and which exist."""
    sites, dist = _water_sites(args)
    s = torch.tensor(sites, device=x.device)
    row, slot, kind = s[:, 0].long(), s[:, 1].long(), s[:, 2].long()
    A, B, C = x[s[:, 3].long()], x[s[:, 4].long()], x[s[:, 5].long()]
    donor, ringed = kind == 1, kind == 4
    B = torch.where(ringed[:, None], (B + C) / 2, B)
    e0 = torch.nn.functional.normalize(A - B, dim=1)
    u = torch.linalg.cross(e0, torch.where(donor[:, None], e0.detach().roll(1, 1), C - B))
    e2 = torch.nn.functional.normalize(u, dim=1)
    e1 = torch.linalg.cross(e2, e0)
    bend, tor = math.pi - s[:, 7:8], s[:, 6:7]
    lone = A + dist * (torch.cos(bend) * e0 + torch.sin(bend) * (torch.cos(tor) * e1 + torch.sin(tor) * e2))
    W = torch.where(donor[:, None], A - dist * e0, lone)
    out = torch.zeros((x.shape[0] * 4, 3), dtype=x.dtype, device=x.device)
    has = torch.zeros(x.shape[0] * 4, dtype=torch.bool, device=x.device)
    has[row * 4 + slot] = True
    return out.index_put((row * 4 + slot,), W).reshape(-1, 4, 3), has.reshape(-1, 4)


def _lkball_energies(args, x, waters, has, i, j, atoms, sep):
    t1, a1, t2, a2 = atoms
    polar, occ, par = args["tables"]
    # both orders: either atom may be the polar one
    I, J = torch.cat([i, j]), torch.cat([j, i])
    tI, aI = torch.cat([t1, t2]), torch.cat([a1, a2])
    tJ, aJ = torch.cat([t2, t1]), torch.cat([a2, a1])
    sep2 = torch.cat([sep, sep])
    keep = polar[tI, aI] & occ[tJ, aJ] & (sep2 > 3) & has[I, 0]
    src = torch.cat([torch.arange(len(i), device=x.device)] * 2)[keep]
    I, J, sep2 = I[keep], J[keep], sep2[keep]
    q1, q2 = par[tI[keep], aI[keep]], par[tJ[keep], aJ[keep]]
    gp = args["gp"].double().reshape(-1)
    f1, f2 = q1[:, 4:] != 0, q2[:, 4:] != 0
    sigma = _sigma(q1[:, 0], q2[:, 0], f1[:, 0], f2[:, 0], f1[:, 1], f2[:, 1], f1[:, 2], f2[:, 2], f1[:, 3], f2[:, 3],
                   gp[0], gp[1], gp[2])
    d2 = (x[I] - x[J]).pow(2).sum(1)
    iso = _count_pair_weight(sep2) * _lk_direction(
        d2.sqrt(), sigma, f1[:, 4] & f2[:, 4], gp[4], q1[:, 0], q1[:, 1], q1[:, 2], q2[:, 3]
    )
    WI, WJ, hI, hJ = waters[I], waters[J], has[I], has[J]

    def overlap(s, width):
        """-log of the overlap, faded from 1 at 0 to 0 at width."""
        v = -torch.log(s.clamp(min=1e-300))
        return torch.where(v < 0, 1.0, torch.where(v < width, (1 - (v.clamp(max=width) / width) ** 2) ** 2, 0.0))

    low = ((1.4 + q2[:, 0]) ** 2 - 3.709).clamp(min=0)
    e = torch.exp(-((x[J][:, None] - WI).pow(2).sum(2) - low[:, None]))
    desolvated = overlap(torch.where(hI, e, torch.zeros_like(e)).sum(1), 3.709)
    b = torch.exp(-((WI[:, :, None] - WJ[:, None]).pow(2).sum(3) - 0.5))
    b = torch.where(hI[:, :, None] & hJ[:, None], b, torch.zeros_like(b)).sum((1, 2))
    base = d2 - 8.0 / 3.0 * gp[3] ** 2
    over = 2.8 * 2.6
    angle = torch.where(base.abs() > over, torch.zeros_like(base), (1 - (base / over) ** 2) ** 2)
    bridge = overlap(b, 2.6) * angle
    bridge = torch.where(f2[:, 0] | f2[:, 3], bridge, torch.zeros_like(bridge))
    return src, torch.stack([iso, iso * desolvated, iso * bridge, bridge / 2])


def _energies(name, args, x, waters, i, j, e, atoms, sep):
    """(output index, energies [terms, n]) of atom pairs."""
    if name == "lkball":
        src, E = _lkball_energies(args, x, *waters, i, j, atoms, sep)
        return e[src], E
    return e, (_ljlk_energies if name == "ljlk" else _elec_energies)(args, x, i, j, atoms, sep)


PAIRS_AT_ONCE = 60000  # rotamer pairs evaluated together


def _exact_pose_term(name, args, x, weights, block_pair):
    """Energies of one term; with x.requires_grad, the gradient of their
    weighted sum in x.grad."""
    P, B = args["first_bt"].shape
    bc, br, nr, r0 = _block_spheres(args, x)
    real = args["first_bt"].cpu().numpy() >= 0
    # every block pair with atoms in reach, with room for rounding
    pairs = _block_pairs(bc, br, real, float(args["max_dis"]) + 0.05)
    p, b1, b2 = (torch.tensor(v, device=x.device) for v in pairs)
    rot1, rot2 = torch.tensor(r0, device=x.device)[p, b1], torch.tensor(r0, device=x.device)[p, b2]
    max_dis = float(args["max_dis"])
    waters = None
    if name == "lkball":
        args["tables"] = _lkball_tables(args)
    out = torch.zeros((len(WEIGHTS[name]), P * B * B if block_pair else P), dtype=torch.float64, device=x.device)
    flat = weights.reshape(weights.shape[0], -1)
    target = (p * B + b1) * B + b2 if block_pair else p
    for s in range(0, len(p), PAIRS_AT_ONCE):
        t = slice(s, s + PAIRS_AT_ONCE)
        with torch.no_grad():
            i, j, e, atoms, sep = _atom_pairs(args, x, rot1[t], rot2[t], max_dis)
        if name == "lkball":
            waters = _waters(args, x) if waters is None else waters
        for q in range(0, len(i), 1 << 21):
            u = slice(q, q + (1 << 21))
            at, E = _energies(name, args, x, waters, i[u], j[u], e[u], tuple(v[u] for v in atoms), sep[u])
            to = target[t][at]
            if x.requires_grad:
                (E * flat[:, to]).sum().backward(retain_graph=name == "lkball")
            out.index_add_(1, to, E.detach())
    return out.reshape((-1, P, B, B) if block_pair else (-1, P))


def _exact_rotamers(case, ps, seeds):
    rs = _rotamer_set(case, ps, seeds)
    name = case["term"]
    args = _op_args(name, ps, rs)
    x32 = rs.coords.to(getattr(torch, case["dtype"]))
    x = x32.double()
    bc, br, nr, r0 = _block_spheres(args, x32)
    pairs = _block_pairs(bc, br, nr > 0, float(args["max_dis"]))
    rot1, rot2 = (torch.tensor(v, device=x.device) for v in _rotamer_pairs(pairs, nr, r0))
    out = torch.zeros((len(WEIGHTS[name]), len(rot1)), dtype=torch.float64, device=x.device)
    waters = None
    with torch.no_grad():
        if name == "lkball":
            args["tables"] = _lkball_tables(args)
            waters = _waters(args, x)
        for s in range(0, len(rot1), PAIRS_AT_ONCE):
            t = slice(s, s + PAIRS_AT_ONCE)
            i, j, e, atoms, sep = _atom_pairs(args, x, rot1[t], rot2[t], float(args["max_dis"]))
            at, E = _energies(name, args, x, waters, i, j, e, atoms, sep)
            out.index_add_(1, s + at, E)
    return {"scores": out, "indices": None}
