"""The atom-pair engine at the sizes where its groups can go wrong: one-atom
rows to several groups per block, a group with more pairs than the queue
holds (a pose squeezed until nearly every pair is in reach), block pairs and
rotamer pairs of such poses, type parameters without a common fade interval
(no far class), and the LK-ball walk over such poses.

float64 energies and gradients against the oracle.  A gradient component is
a sum of at most a few thousand signed terms, each no larger than the largest
component's magnitude allows by a factor of ten or so, so its float64 sum is
good to 1e-12 of the largest component (2.2e-16 x a few thousand); energies
likewise to 1e-11 relative.  A float32 pair force is good to about 1e-6 of
itself (some sixteen roundings, steep in the distance), so a component, whose
terms sum to some tens of the largest component in magnitude, to 2e-5 of the
largest component."""

import json

import numpy
import pytest
import torch

from oracle import oracle as O
from tmol_b200.pose.rotamers import synthetic_rotamer_set
from tmol_b200.pose.synthetic import synthetic_pose_stack
from tmol_b200.score.elec_energy_term import ElecEnergyTerm, elec_pose_score_args
from tmol_b200.score.elec_op import elec_pose_scores
from tmol_b200.score.ljlk_energy_term import LJLKEnergyTerm, pose_score_args, rotamer_score_args
from tmol_b200.score.ljlk_op import clear_plan_cache, ljlk_pose_scores, ljlk_rotamer_scores
from tolerances import E_close

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def close(x, ref, rel):
    ref = numpy.asarray(ref)
    err = numpy.abs(x.detach().cpu().numpy() - ref)
    assert err.max() <= rel * numpy.abs(ref).max() + 1e-9, (err.max(), numpy.abs(ref).max())


def on_gpu(args, dtype):
    return [
        a.to(DEV, dtype if a.is_floating_point() else a.dtype) if isinstance(a, torch.Tensor) else a for a in args
    ]


@pytest.mark.parametrize("scale", [1.0, 0.5])
@pytest.mark.parametrize("name", ["ljlk", "elec"])
@pytest.mark.parametrize("block_pair", [False, True])
def test_pose_groups(name, block_pair, scale):
    ps = synthetic_pose_stack([30, 1, 2, 9, 75], [5, 6, 7, 8, 9], spacing=0.0)
    x = (ps.coords * scale).flatten(0, 1).double()
    op, args_of, term = {
        "ljlk": (ljlk_pose_scores, pose_score_args, LJLKEnergyTerm()),
        "elec": (elec_pose_scores, elec_pose_score_args, ElecEnergyTerm()),
    }[name]
    args = args_of(ps, term, block_pair)
    oc = O.OracleCall(x, args, f64=True, term=name)
    n = 3 if name == "ljlk" else 1
    c = x.to(DEV).requires_grad_(True)
    E, nbr = op(c, *on_gpu(args, torch.float64))
    Eo, dVo, nbro = oc.pose_scores(block_pair=block_pair, require_gradient=True)
    close(E, numpy.asarray(Eo)[:n].reshape(E.shape), 1e-11)
    assert numpy.array_equal(nbr.cpu().numpy(), nbro)
    E.sum().backward()
    _, dVo, _ = oc.pose_scores(require_gradient=True)
    close(c.grad, dVo[:n].sum(0), 1e-12)
    E32, _ = op(x.to(DEV, torch.float32), *on_gpu(args, torch.float32))
    E_close(E32.cpu().numpy(), numpy.asarray(Eo)[:n].reshape(E.shape), what=f"{name} float32, scale {scale}")
    clear_plan_cache()


@pytest.mark.parametrize("scale", [1.0, 0.5])
def test_rotamer_groups(scale):
    ps = synthetic_pose_stack([12, 3], [15, 16], spacing=0.0)
    rs = synthetic_rotamer_set(ps, max_rots=40, seed=3)
    args = rotamer_score_args(ps, rs, LJLKEnergyTerm())
    x = (rs.coords * scale).double()
    Eo, ind, _ = O.OracleCall(x, args, f64=True).rotamer_scores()
    E, indices = ljlk_rotamer_scores(x.to(DEV), *on_gpu(args, torch.float64))
    assert numpy.array_equal(indices.cpu().numpy(), ind)
    close(E, Eo, 1e-11)
    clear_plan_cache()


def one_atom_pose_stack():
    """Poses with blocks of a single atom, alone, among residues and as the
    last of more blocks than a group has words."""
    from tmol_b200.chem.restypes import ChemicalDatabase, PackedBlockTypes, ResidueType, ResidueTypeSet
    from tmol_b200.pose.builder import PoseTopology, build_pose_stack

    one = ResidueType(
        name="ONE", base_name="ONE", atoms=[["A0", "CH3"]], bonds=[], connections=[], icoors=[], chis=[], aliases=[],
        is_polymer=False, is_ligand_fragment=True,
    )
    pbt = PackedBlockTypes(
        ChemicalDatabase.get_default(), list(ResidueTypeSet.get_default().types.values()) + [one]
    )
    rng = numpy.random.default_rng(7)
    names = [["ONE"], ["GLY"] * 3 + ["ONE"] * 40, (["ONE", "ALA"] * 10) + ["ONE"]]
    coords = [
        rng.normal(scale=3.0, size=(sum(pbt.active_block_types[pbt.bt_index[n]].n_atoms for n in pose), 3))
        for pose in names
    ]
    return build_pose_stack([PoseTopology(n, []) for n in names], coords, pbt=pbt)


@pytest.mark.parametrize("name, poses", [("ljlk", 1.0), ("ljlk", 0.5), ("ljlk", "one atom"), ("elec", 1.0), ("elec", 0.5)])
@pytest.mark.parametrize("block_pair", [False, True])
def test_weighted_gradients(name, block_pair, poses):
    """Energies and gradients under weights of every pose or block pair's own,
    in both precisions, of squeezed poses (groups with more pairs than the
    queue holds) and of blocks of one atom."""
    from tmol_b200.score.elec_op import ElecPlan
    from tmol_b200.score.ljlk_op import LJLKPlan

    if poses == "one atom":  # a block type without charges
        ps, scale = one_atom_pose_stack(), 1.0
    else:
        ps, scale = synthetic_pose_stack([30, 1, 2, 9, 75], [5, 6, 7, 8, 9], spacing=0.0), poses
    x = (ps.coords * scale).flatten(0, 1).float()
    args_of, term, plan_of, n = {
        "ljlk": (pose_score_args, LJLKEnergyTerm(), LJLKPlan, 3),
        "elec": (elec_pose_score_args, ElecEnergyTerm(), ElecPlan, 1),
    }[name]
    args = args_of(ps, term, block_pair)
    oc = O.OracleCall(x.double(), args, f64=True, term=name)
    Eo, _, nbr = oc.pose_scores(block_pair=block_pair)
    w = numpy.zeros((3,) + Eo.shape[1:])
    w[:n] = numpy.random.default_rng(11).normal(size=(n,) + Eo.shape[1:]).astype(numpy.float32)
    go = oc.backward(nbr, w, per_pose_weights=not block_pair)
    for dtype, rel in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
        c = x.to(DEV, dtype).contiguous()
        plan = plan_of(c, on_gpu(args, dtype)[:-1])
        E, _ = plan.forward(c, block_pair=block_pair)
        if dtype == torch.float64:
            close(E, Eo[:n].reshape(E.shape), 1e-11)
        else:
            E_close(E.cpu().numpy(), Eo[:n].reshape(E.shape))
        close(plan.backward(c, torch.tensor(w[:n], device=DEV), block_pair=block_pair), go, rel)


@pytest.mark.parametrize("scale", [1.0, 0.5])
def test_weighted_rotamer_gradients(scale):
    from tmol_b200.score.ljlk_op import LJLKPlan

    ps = synthetic_pose_stack([12, 3], [15, 16], spacing=0.0)
    rs = synthetic_rotamer_set(ps, max_rots=40, seed=3)
    args = rotamer_score_args(ps, rs, LJLKEnergyTerm())
    x = (rs.coords * scale).float()
    oc = O.OracleCall(x.double(), args, f64=True)
    Eo, ind, nbr = oc.rotamer_scores()
    w = numpy.random.default_rng(12).normal(size=Eo.shape).astype(numpy.float32).astype(numpy.float64)
    go = oc.rotamer_backward(nbr, w)
    for dtype, rel in ((torch.float64, 1e-12), (torch.float32, 2e-5)):
        c = x.to(DEV, dtype).contiguous()
        plan = LJLKPlan(c, on_gpu(args, dtype)[:-1], rotamers=True)
        indices, items = plan.rotamer_dispatch(c)
        assert numpy.array_equal(indices.cpu().numpy(), ind)
        close(plan.rotamer_backward(c, items, torch.tensor(w, device=DEV)), go, rel)


def pair_plan(name, rotamers, dtype, scale):
    """A plan over squeezed poses (or their rotamers) and its coordinates."""
    from tmol_b200.score.elec_energy_term import elec_rotamer_score_args
    from tmol_b200.score.elec_op import ElecPlan
    from tmol_b200.score.ljlk_op import LJLKPlan

    ps = synthetic_pose_stack([30, 1, 2, 9, 75], [5, 6, 7, 8, 9], spacing=0.0)
    term = {"ljlk": LJLKEnergyTerm, "elec": ElecEnergyTerm}[name]()
    if rotamers:
        ps = synthetic_pose_stack([12, 3], [15, 16], spacing=0.0)
        rs = synthetic_rotamer_set(ps, max_rots=40, seed=3)
        args = {"ljlk": rotamer_score_args, "elec": elec_rotamer_score_args}[name](ps, rs, term)
        x = rs.coords
    else:
        args = {"ljlk": pose_score_args, "elec": elec_pose_score_args}[name](ps, term, True)
        x = ps.coords.flatten(0, 1)
    x = (x * scale).to(DEV, dtype).contiguous()
    plan = {"ljlk": LJLKPlan, "elec": ElecPlan}[name](x, on_gpu(args, dtype)[:-1], rotamers=rotamers)
    return plan, x


@pytest.mark.parametrize("scale", [1.0, 0.5])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("rotamers", [False, True])
@pytest.mark.parametrize("name", ["ljlk", "elec"])
def test_pair_energies_repeat(name, rotamers, dtype, scale):
    """A pair's energy is the same bits in every call, whichever other pairs
    its warp scores beside it: across repeated calls, work items split anew
    by their measured costs or cut to other lengths, and groups of one and of
    nine pairs."""
    plan, x = pair_plan(name, rotamers, dtype, scale)
    if rotamers:
        indices, items = plan.rotamer_dispatch(x)
        run = lambda: plan.rotamer_forward(x, items, indices.shape[1])
    else:
        run = lambda: plan.forward(x, block_pair=True)[0]
    first = run()
    for _ in range(4):
        assert torch.equal(run(), first)
    for launch in (dict(slots_per_group=1), dict(slots_per_group=3, candidates_per_item=4), dict(warps_per_cta=2)):
        plan.set_launch(**launch)
        assert torch.equal(run(), first), launch
    if not rotamers:
        plan.balance(run)
        assert torch.equal(run(), first)


@pytest.mark.parametrize("scale", [1e-8, 1e-4, 0.3, 1.0, 1e4, 1e8])
@pytest.mark.parametrize("name", ["ljlk", "lkball"])
def test_gradient_spread(name, scale):
    """Two calls' float32 gradients differ in the order of their sums alone,
    and in the small part only: clashes' forces are summed exactly.  What is
    left adds some 300 terms of less than one under unit weights, each sum
    rounded by at most 2^-25: sqrt(300) x 3e-8 = 5e-7 a component, three times
    that between the extremes of ten calls, and as much again where the last
    addition rounds the other way: below 4e-6 of the weights' size as a root
    mean square (one plain sum: 1.5e-5).  The scale of the loss does not
    matter."""
    from tmol_b200.score.lkball_energy_term import LKBallEnergyTerm, score_args, water_gen_args
    from tmol_b200.score.lkball_op import LKBallPlan
    from tmol_b200.score.ljlk_op import LJLKPlan

    ps = synthetic_pose_stack([150] * 4, [0, 1, 2, 3], device=DEV, extra_chi_sd=30.0)
    x = ps.coords.flatten(0, 1).contiguous()
    if name == "ljlk":
        plan = LJLKPlan(x, pose_score_args(ps, LJLKEnergyTerm(device=DEV))[:-1])
        weights = torch.tensor([1.0, 0.55, 1.0], device=DEV)
    else:
        term = LKBallEnergyTerm(device=DEV)
        plan = LKBallPlan(x, water_gen_args(ps, term), score_args(ps, term, None)[:-2])
        weights = torch.tensor([-0.38, 0.92, -0.33, -0.33], device=DEV)
    weights = (weights[:, None] * scale).expand(-1, 4).contiguous()
    if name == "ljlk":
        run = lambda: plan.backward(x, weights)
    else:
        W = plan.waters(x)
        run = lambda: plan.backward(x, W, weights)[0]
    G = torch.stack([run().clone() for _ in range(10)])
    spread = (G.max(0)[0] - G.min(0)[0]).double()
    assert float(spread.pow(2).mean().sqrt()) < 4e-6 * scale


def test_infinite_force():
    """A force beyond float32's range is an infinite gradient, not a NaN: one
    atom pair of two residues brought to 1.2 A, the others farther apart."""
    from tmol_b200.score.ljlk_op import LJLKPlan

    ps = synthetic_pose_stack([4], [6], spacing=0.0)
    args = pose_score_args(ps, LJLKEnergyTerm())
    first = args[0].tolist() + [ps.coords.shape[1]]
    x = ps.coords.flatten(0, 1).double()
    u = torch.tensor([0.5, 0.8, 0.7], dtype=torch.float64)
    a = int((x[: first[1]] @ u).argmax())
    b = first[3] + int((x[first[3] :] @ u).argmin())
    x[first[1] : first[3]] += torch.tensor([500.0, -500.0, 0.0], dtype=torch.float64)
    x[first[3] :] += x[a] - x[b] + 1.2 * u / u.norm()
    apart = x.clone()
    apart[first[3] :] += 100.0
    rep = torch.tensor([[0.0], [1.0], [0.0]], dtype=torch.float64, device=DEV)
    plan64 = LJLKPlan(x.to(DEV), on_gpu(args, torch.float64)[:-1])
    g, rest = plan64.backward(x.to(DEV), rep)[[a, b]], plan64.backward(apart.to(DEV), rep)[[a, b]]
    top = torch.finfo(torch.float32).max
    w = 1.5 * top / float(g.abs().min())
    assert float(rest.abs().max()) * w < top / 4 and w < top
    plan = LJLKPlan(x.float().to(DEV), on_gpu(args, torch.float32)[:-1])
    got = plan.backward(x.float().to(DEV), rep * w)[[a, b]]
    assert torch.equal(got, torch.sign(g).float() * float("inf"))


@pytest.mark.parametrize("name", ["ljlk", "elec"])
def test_default_launch_again(name, tmp_path):
    """set_launch with zeros is the launch shape a plan is made with."""
    from torch.profiler import ProfilerActivity, profile

    from tmol_b200.score.elec_op import ElecPlan
    from tmol_b200.score.ljlk_op import LJLKPlan

    many = synthetic_pose_stack([200] * 8, list(range(8)))
    args = {"ljlk": pose_score_args, "elec": elec_pose_score_args}[name](
        many, {"ljlk": LJLKEnergyTerm, "elec": ElecEnergyTerm}[name]()
    )
    x = many.coords.flatten(0, 1).to(DEV).contiguous()
    plan = {"ljlk": LJLKPlan, "elec": ElecPlan}[name](x, on_gpu(args, torch.float32)[:-1])

    def blocks():
        plan.forward(x)
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            plan.forward(x)
            torch.cuda.synchronize()
        prof.export_chrome_trace(str(tmp_path / "trace.json"))
        events = json.loads((tmp_path / "trace.json").read_text())["traceEvents"]
        return [e["args"]["block"] for e in events if "score_kernel" in e.get("name", "")]

    made = blocks()
    if not made:
        pytest.skip("no kernel trace on this machine")
    plan.set_launch()
    assert blocks() == made


def test_plan_memory():
    """Plans of one size after another, some alive, map no device memory; a
    plan freed with its call still queued hands its memory on only after it;
    what plans gave back beyond 64 MB, and all of it after the last plan, goes
    back to the device (which the pool does in pieces of 32 MB)."""
    import gc

    from tmol_b200.score.ljlk_op import LJLKPlan

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info(DEV)[0]

    clear_plan_cache()
    gc.collect()
    ps = synthetic_pose_stack([100] * 8, list(range(8)), device=DEV)
    x = ps.coords.flatten(0, 1).contiguous()
    args = pose_score_args(ps, LJLKEnergyTerm(device=DEV))[:-1]
    weights = torch.ones(3, 8, device=DEV)
    warm = LJLKPlan(x, args)
    E, g = warm.energy_and_gradient(x, weights)
    del warm
    plans = [LJLKPlan(x, args) for _ in range(3)]
    held = free()
    for k in range(12):
        plans[k % 3] = None
        assert free() == held
        plans[k % 3] = LJLKPlan(x, args)
        assert free() == held
    out, dx = torch.empty_like(E), torch.empty_like(g)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        torch.cuda._sleep(20_000_000)
        plans[0].energy_and_gradient(x, weights, out, dx)
    assert not other.query()
    plans[0] = None
    assert other.query()
    plans[0] = LJLKPlan(x + 1.0, args)
    plans[0].energy_and_gradient(x + 1.0, weights * 0.5)
    torch.cuda.synchronize()
    assert torch.allclose(out, E, rtol=1e-5) and torch.allclose(dx, g, rtol=1e-4, atol=1e-4)
    held = free()  # some of it torch's for the second stream
    many = [LJLKPlan(x, args) for _ in range(100)]
    assert many[0].device_bytes() * 100 > 3 * (64 << 20)
    del many
    assert held - free() <= 64 << 20
    plans.clear()
    assert free() - held >= 32 << 20


def test_no_common_fade_interval():
    """A type whose LJ minimum lies inside the fade interval fades on an
    interval of its own: the general path serves every pair.  (Energies, from
    the oracle's energy-only form: for such a type the reference's form with
    derivatives divides attractive and repulsive parts otherwise.)"""
    ps = synthetic_pose_stack([40, 12], [25, 26], spacing=0.0)
    args = pose_score_args(ps, LJLKEnergyTerm())
    params = args[22].clone()
    params[int(args[17][0, 0]), 0] = 3.1  # the radius of the first block type's first atom's type
    args[22] = params
    x = ps.coords.flatten(0, 1).double()
    E, _ = ljlk_pose_scores(x.to(DEV), *on_gpu(args, torch.float64))
    Eo, _, _ = O.OracleCall(x, args, f64=True).pose_scores()
    close(E, Eo, 1e-11)
    clear_plan_cache()


@pytest.mark.parametrize("scale", [1.0, 0.6])
@pytest.mark.parametrize("block_pair", [False, True])
def test_lkball_lists(block_pair, scale):
    """The LK-ball walk over the neighbours' heavy atoms: lists of less than
    one and of many windows of 32 atoms, windows that begin inside a
    neighbour, and (poses drawn together) rows that meet every one of them.
    Energies and gradient as in the docstring above, with three more digits
    for the waters' frames and the ramps' quotients between."""
    from tests.test_gpu_lkball import gpu_run
    from tests.test_lkball_oracle import oracle_run
    from tmol_b200.score.lkball_energy_term import LKBallEnergyTerm

    ps = synthetic_pose_stack([30, 1, 2, 9, 75], [5, 6, 7, 8, 9], spacing=0.0)
    ps.coords = ps.coords * scale
    _, E, dx, nbr = gpu_run(ps, LKBallEnergyTerm(), torch.float64, block_pair)
    _, Eo, dxo, nbro = oracle_run(ps, True)
    if block_pair:
        E = E.sum((2, 3))
    close(E, numpy.asarray(Eo).reshape(E.shape), 1e-9)
    assert numpy.array_equal(nbr.cpu().numpy(), nbro)
    close(dx, dxo, 1e-9)


def wide_block_pose_stack():
    """Poses with a block of more than 32 heavy atoms, alone and bonded to
    small ones, and with lists of at most eight and sixteen."""
    from exotic_blocks import big_block_type
    from tmol_b200.chem.restypes import ChemicalDatabase, PackedBlockTypes, ResidueTypeSet
    from tmol_b200.pose.builder import PoseTopology, build_pose_stack

    wide = big_block_type("BIG70", 70, False, 5)
    pbt = PackedBlockTypes(
        ChemicalDatabase.get_default(), list(ResidueTypeSet.get_default().types.values()) + [wide]
    )
    rng = numpy.random.default_rng(3)
    topologies, coords = [], []
    for names in (["BIG70"], ["ALA:nterm", "BIG70", "GLY", "SER:cterm"], ["BIG70", "BIG70"], ["GLY"], ["ALA", "GLY"]):
        bonds = [(i, "up", i + 1, "down") for i in range(len(names) - 1)]
        n = sum(pbt.active_block_types[pbt.bt_index[x]].n_atoms for x in names)
        steps = rng.normal(size=(n, 3))
        walk = numpy.cumsum(1.5 * steps / numpy.linalg.norm(steps, axis=1, keepdims=True), axis=0)
        topologies.append(PoseTopology(names, bonds))
        coords.append(0.6 * walk + rng.normal(scale=0.3, size=walk.shape))
    return build_pose_stack(topologies, coords, pbt=pbt)


@pytest.mark.parametrize("block_pair", [False, True])
def test_lkball_wide_blocks(block_pair):
    """The walk where the rows take several tiles of 32 and where a list is
    short enough for two or four lanes an atom; tolerances as above."""
    from tests.test_gpu_lkball import gpu_run
    from tests.test_lkball_oracle import oracle_run
    from tmol_b200.score.lkball_energy_term import LKBallEnergyTerm

    ps = wide_block_pose_stack()
    _, E, dx, nbr = gpu_run(ps, LKBallEnergyTerm(), torch.float64, block_pair)
    _, Eo, dxo, nbro = oracle_run(ps, True)
    if block_pair:
        E = E.sum((2, 3))
    close(E, numpy.asarray(Eo).reshape(E.shape), 1e-9)
    assert numpy.array_equal(nbr.cpu().numpy(), nbro)
    close(dx, dxo, 1e-9)
