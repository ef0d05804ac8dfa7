"""The framework's work on one GPU, case by case: what a simulation code asks
of the gravity backend, through the public binding (galactic_tides_gb300.gtc).

Kinds of case:

* group    one force evaluation of the grouped solver on device arrays
           (Context.group_force_device): tree build, walk, list evaluation;
* host     the same through the drop-in call with host arrays
           (Context.group_force), as the C++ code calls it: the copies count;
* learned  one evaluation with the learned opening criterion (the committed
           model and its calibrated alpha), after a theta evaluation of the
           same bodies, as a run that switches it on has it;
* evolve   a galaxy encounter advanced by the CUDA-graph leapfrog, with the
           diagnostics a run logs;
* ensemble independent galaxies advanced together (Ensemble.leapfrog);
* direct   the tiled FP32 direct sum over all pairs;
* tree     the per-particle FP64 tree walk (the `gravity = tree` solver);
* sample   FP64 direct sums on a sample of targets: the accuracy judge that
           the benchmark and the evolve runs use.

Bodies are the benchmark galaxy model's (disk, bulge, halo). The grouped and
direct solvers compute accelerations and potentials in FP32 and store them
in the caller's FP64 arrays, a widening without rounding, so those results
are handed back as the FP32 values they are; an evolved state is handed back
in single precision as well, as GADGET-style snapshots keep it (its
velocities are sums of FP32 accelerations). The FP64 solvers' results are
FP64.
"""

import json
import math

import numpy as np
import torch

import __graft_entry__

gtc = __graft_entry__.load_package().gtc
_PKG = __graft_entry__.PKG_DIR

# the benchmark's solver settings; a case overrides what it varies
SOLVER = dict(G=1.0, theta=0.75, eps=0.025, quadrupole=True, group_size=32, leaf_size=8,
              pack=True)
_OPTIONS = ("theta", "eps", "quadrupole", "group_size", "leaf_size", "pack")


def listed():
    return [
        # latency: a small test particle set, where launches and host reads count
        dict(name="group_5k", kind="group", n=5003),
        # the small evolution run's galaxy
        dict(name="group_50k", kind="group", n=50_000),
        # the size of the published figures, through the drop-in host call
        dict(name="host_200k", kind="host", n=200_000),
        # the headline size
        dict(name="group_2m", kind="group", n=2_000_000),
        # monopole only, unsoftened, a tighter angle, an odd body count: the
        # other forms that the solver's parameters select
        dict(name="group_mono_100k", kind="group", n=100_003, theta=0.6, eps=0.0,
             quadrupole=False, group_size=24, leaf_size=12, pack=False),
        # the learned criterion
        dict(name="learned_200k", kind="learned", n=200_000),
        # an encounter of two galaxies between two log lines of a run
        dict(name="evolve_200k", kind="evolve", n=200_000, steps=20, dt=0.01),
        # a parameter study: many galaxies at once
        dict(name="ensemble_16", kind="ensemble", systems=16, n_min=10_000, n_max=200_000,
             steps=5, dt=0.01),
        # all-pairs solver: a small set with a ragged size, and the published size
        dict(name="direct_20k", kind="direct", n=20_011),
        dict(name="direct_200k", kind="direct", n=200_000),
        # the FP64 per-particle solver at the published size
        dict(name="tree_200k", kind="tree", n=200_000),
        # the accuracy sample of a run's check
        dict(name="sample_500k", kind="sample", n=500_000, m=4096),
    ]


def _log(rng, lo, hi):
    """A size between lo and hi, spread over its logarithm; odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["group", "group", "group", "host", "learned", "evolve", "ensemble",
                       "direct", "tree", "sample"])
    if kind in ("group", "host"):
        # one evaluation: from a few thousand bodies to the headline size
        case = dict(kind=kind, n=_log(rng, 3_000, 2_000_000 if kind == "group" else 1_000_000))
        if rng.random() < 0.5:
            case.update(theta=rng.choice([0.6, 0.7, 0.8, 1.0]), group_size=rng.choice([16, 24, 32]),
                        leaf_size=rng.choice([4, 8, 12, 16]), pack=rng.random() < 0.7,
                        quadrupole=rng.random() < 0.6, eps=rng.choice([0.0, 0.01, 0.05]))
        return case
    if kind == "learned":
        return dict(kind=kind, n=_log(rng, 50_000, 300_000))
    if kind == "evolve":
        return dict(kind=kind, n=2 * _log(rng, 5_000, 150_000), steps=rng.randint(5, 20),
                    dt=rng.choice([0.005, 0.01]))
    if kind == "ensemble":
        return dict(kind=kind, systems=rng.randint(3, 16), n_min=_log(rng, 3_000, 10_000),
                    n_max=_log(rng, 30_000, 200_000), steps=rng.randint(2, 5), dt=0.01)
    if kind == "direct":
        return dict(kind=kind, n=_log(rng, 3_000, 200_000), eps=rng.choice([0.025, 0.05]))
    if kind == "tree":
        return dict(kind=kind, n=_log(rng, 5_000, 200_000), theta=rng.choice([0.6, 0.75, 0.9]),
                    quadrupole=rng.random() < 0.8)
    return dict(kind=kind, n=_log(rng, 50_000, 500_000), m=rng.choice([1024, 2000, 4096]))


def _solver(case):
    return dict(SOLVER, **{k: case[k] for k in _OPTIONS if k in case})


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _ensemble_sizes(case):
    """Body counts of the study's galaxies (the seeds draw their bodies):
    log-uniform in [n_min, n_max], one per equal slice of the logarithm."""
    k = case["systems"]
    rng = np.random.default_rng(k)
    u = (np.arange(k) + rng.uniform(0.0, 1.0, k)) / k
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return [int(round(x)) for x in np.exp(lo + (hi - lo) * u)]


def _bodies(case, seed):
    if case["kind"] == "evolve":
        half = case["n"] // 2
        pos, vel, mass, _ = gtc.make_encounter(half, seed=2 * seed + 1, incl1=30.0, incl2=60.0,
                                               rp=2.0, r0=15.0)
        return pos, vel, mass
    pos, vel, mass, _ = gtc.make_galaxy(case["n"], seed=seed)
    return pos, vel, mass


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, kind=kind, kw=_solver(case))
    if kind == "ensemble":
        sizes = _ensemble_sizes(case)
        ens = gtc.Ensemble(len(sizes))
        systems = []
        for k, n in enumerate(sizes):
            pos, vel, mass, _ = gtc.make_galaxy(n, seed=1000 * seed + k)
            g = dict(pos0=_dev(pos), vel0=_dev(vel), mass=_dev(mass),
                     acc=torch.zeros((n, 3), dtype=torch.float64, device="cuda"),
                     pot=torch.zeros(n, dtype=torch.float64, device="cuda"))
            g.update(pos=g["pos0"].clone(), vel=g["vel0"].clone())
            ens.set_system(k, g["pos"].data_ptr(), g["vel"].data_ptr(), g["mass"].data_ptr(),
                           g["acc"].data_ptr(), g["pot"].data_ptr(), n, **st["kw"])
            systems.append(g)
        torch.cuda.synchronize()
        return dict(st, ens=ens, systems=systems)

    pos, vel, mass = _bodies(case, seed)
    n = len(mass)
    st.update(ctx=gtc.Context(0), n=n)
    if kind == "host":
        return dict(st, pos=pos, mass=mass)
    st.update(pos=_dev(pos), mass=_dev(mass),
              acc=torch.zeros((n, 3), dtype=torch.float64, device="cuda"),
              pot=torch.zeros(n, dtype=torch.float64, device="cuda"))
    if kind == "evolve":
        st.update(pos0=st["pos"].clone(), vel0=_dev(vel), vel=_dev(vel))
    elif kind == "sample":
        st["idx"] = _dev(gtc.sample_indices(n, case["m"], seed + 1).astype(np.int64))
        st["acc"] = torch.zeros((case["m"], 3), dtype=torch.float64, device="cuda")
        st["pot"] = torch.zeros(case["m"], dtype=torch.float64, device="cuda")
    elif kind == "tree":
        st.update(pos=pos, mass=mass)  # the binding has the host-array form
    torch.cuda.synchronize()
    if kind == "learned":
        info = json.loads((_PKG / "criterion_model.json").read_text())
        st["ctx"].learned_set_model(np.fromfile(_PKG / "criterion_model.f32", np.float32))
        # the criterion takes |a| from the previous evaluation of the bodies
        st["ctx"].group_force_device(st["pos"].data_ptr(), st["mass"].data_ptr(), n,
                                     st["acc"].data_ptr(), st["pot"].data_ptr(), **st["kw"])
        st["kw"].update(criterion=gtc.CRITERION_LEARNED, alpha=float(info["alpha"]))
    return st


def run(st):
    kind, kw = st["kind"], st["kw"]
    # the solver works on a stream of its own: what the caller queued for its
    # arrays (this program's earlier reads of them too) has to be done
    torch.cuda.current_stream().synchronize()
    if kind == "host":
        acc, pot = st["ctx"].group_force(st["pos"], st["mass"], **kw)
        return {"acc": acc.astype(np.float32), "pot": pot.astype(np.float32)}
    if kind == "tree":
        acc, pot = st["ctx"].tree_force(st["pos"], st["mass"], G=kw["G"], theta=kw["theta"],
                                        eps=kw["eps"], quadrupole=kw["quadrupole"],
                                        leaf_size=kw["leaf_size"])
        return {"acc": acc, "pot": pot}
    if kind == "ensemble":
        for g in st["systems"]:  # every pass runs from the initial conditions
            g["pos"].copy_(g["pos0"])
            g["vel"].copy_(g["vel0"])
        torch.cuda.current_stream().synchronize()
        st["ens"].leapfrog(st["case"]["dt"], st["case"]["steps"], prime=True, graph=True)
        return [{k: g[k].float() for k in ("pos", "vel", "acc", "pot")} for g in st["systems"]]

    ctx, n = st["ctx"], st["n"]
    pos, mass, acc, pot = (st[k].data_ptr() for k in ("pos", "mass", "acc", "pot"))
    if kind in ("group", "learned"):
        ctx.group_force_device(pos, mass, n, acc, pot, **kw)
    elif kind == "direct":
        ctx.direct_force_device(pos, mass, n, acc, pot, G=kw["G"], eps=kw["eps"])
    elif kind == "sample":
        ctx.direct_fp64_device(pos, mass, n, st["idx"].data_ptr(), len(st["pot"]), acc, pot,
                               G=kw["G"], eps=kw["eps"])
        return {"acc": st["acc"], "pot": st["pot"]}
    else:  # evolve, from the initial conditions
        st["pos"].copy_(st["pos0"])
        st["vel"].copy_(st["vel0"])
        torch.cuda.current_stream().synchronize()
        ctx.leapfrog_device(pos, st["vel"].data_ptr(), mass, acc, pot, n, st["case"]["dt"],
                            st["case"]["steps"], prime=True, graph=True, **kw)
        d = ctx.diagnostics_device(pos, st["vel"].data_ptr(), mass, pot, n)
        return {"pos": st["pos"].float(), "vel": st["vel"].float(), "acc": st["acc"].float(),
                "pot": st["pot"].float(), "energy": np.float32([d["kinetic"], d["potential"]])}
    return {"acc": st["acc"].float(), "pot": st["pot"].float()}


def _interactions(n, kw):
    """Cells and bodies a body of the galaxy model interacts with, about: a
    fit to the solver's own counters over this range of sizes."""
    grow = max(math.log2(n) - 8.0, 1.0)
    wide = (0.75 / kw["theta"]) ** 2
    return 80.0 * grow * wide, 490.0 * wide ** 0.5


def work(case):
    kind, kw = case["kind"], _solver(case)
    if kind == "ensemble":
        sizes = _ensemble_sizes(case)
        one = [work(dict(case, kind="group", n=n)) for n in sizes]
        evals = case["steps"] + 1
        return {k: evals * sum(w[k] for w in one) for k in ("bytes", "flops")}
    n = case["n"]
    # an interaction with a body: 20 operations; with a cell 64 with its
    # quadrupole, 21 without (a multiply-add is two)
    cell = 64.0 if kw["quadrupole"] else 21.0
    bytes_ = 32.0 * n + 32.0 * n  # positions and masses in, accelerations and potentials out
    if kind == "direct":
        return {"bytes": bytes_, "flops": 20.0 * n * n}
    if kind == "sample":
        return {"bytes": 32.0 * n + 40.0 * case["m"], "flops": 20.0 * n * case["m"]}
    cells, bodies = _interactions(n, kw)
    flops = n * (cell * cells + 20.0 * bodies)
    if kind == "tree":  # each body walks alone: about half the grouped lists
        flops *= 0.5
    elif kind == "learned":
        flops *= 0.4
    elif kind == "evolve":
        evals = case["steps"] + 1
        flops *= evals
        bytes_ = evals * (bytes_ + 4 * 24.0 * n)
    return {"bytes": bytes_, "flops": flops}


def _direct64(pos, mass, targets, eps):
    """Softened FP64 sums over all bodies but the target itself."""
    x, m = _dev(pos), _dev(mass)
    n = len(m)
    acc = torch.empty((len(targets), 3), dtype=torch.float64, device="cuda")
    pot = torch.empty(len(targets), dtype=torch.float64, device="cuda")
    chunk = max(1, (1 << 28) // n)
    for a in range(0, len(targets), chunk):
        t = targets[a:a + chunk]
        d = [x[t, k, None] - x[None, :, k] for k in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + eps * eps
        r2[torch.arange(len(t), device="cuda"), t] = math.inf
        inv = r2.rsqrt_()
        gm = inv * m
        pot[a:a + chunk] = -gm.sum(1)
        gm *= inv
        gm *= inv
        for k in range(3):
            acc[a:a + chunk, k] = -(gm * d[k]).sum(1)
    return acc, pot


def exact(case, seed):
    """The forces by direct summation in 64 bits, which every solver here
    computes or approximates; evolved states have no closed value."""
    if case["kind"] in ("evolve", "ensemble") or case["n"] > 200_000 and case["kind"] != "sample":
        return None
    pos, _, mass = _bodies(case, seed)
    n = len(mass)
    if case["kind"] == "sample":
        targets = _dev(gtc.sample_indices(n, case["m"], seed + 1).astype(np.int64))
    else:
        targets = torch.arange(n, device="cuda")
    acc, pot = _direct64(pos, mass, targets, _solver(case)["eps"])
    return {"acc": acc, "pot": pot}
