"""Performance cases of the Metropolis engine: what its users run, through the
public Python interface (mcx.Engine).

Most cases are one block of a run loop, the unit every run mode of the
simulator repeats: a temperature or field value is set, MCT sweeps thermalise,
the running sums are cleared, MCS measured sweeps follow, and the program reads
every replica's sums and directors (a po.dat row and a snapshot per replica).
The others are the training of the learned proposal and the measurement of a
loaded configuration with its per-site order parameter.

A case is a dict of plain values:

  kind      "block", "train" or "snapshot"
  model     "ll", "slab", "droplet", "ghrl" or "pear" (see _descs)
  nx ny nz  lattice; for "slabs" of mixed sizes, sides (0 = all nx^3)
  replicas  replicas in the engine
  mct, mcs  unmeasured and measured sweeps of a block
  tune      whether the program runs the engine's autotuner first, as long
            runs of the batched workloads do (the parameter-file driver, and
            short runs, keep the default shape)
  learned   whether the sweeps use the learned proposal
"""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.getcwd(), "mclics-backend_gb300"))

import mcx  # noqa: E402

# the four temperatures of the learned-proposal workload
TEMPS = (1.00, 1.10, 1.12, 1.15)
# FP32 operations of one site update: six bonds of the old and the new
# director, the rotation and its normalisation, the Metropolis test
FLOPS = {"ll": 110, "pear": 190, "ghrl": 290, "slab": 290, "droplet": 330}
L2_BYTES = 129e6
MLP_FLOPS = 2 * (19 * 64 + 64 * 64 + 64 * 4)


def _case(name, kind="block", model="ll", n=(16, 16, 16), replicas=1, mct=100, mcs=100, tune=False, learned=False,
          **more):
    return {"name": name, "kind": kind, "model": model, "nx": n[0], "ny": n[1], "nz": n[2], "replicas": replicas,
            "mct": mct, "mcs": mcs, "tune": tune, "learned": learned, **more}


def listed():
    return [
        # the reference's plain configuration: one 16^3 periodic LL lattice,
        # one temperature of its anneal (MCT = MCS = 100)
        _case("ll16"),
        # a few uneven LL lattices with one free axis of odd length, as a user
        # with a box of his own sizes runs them
        _case("ll_ragged", n=(46, 30, 27), replicas=4),
        # the headline anneal: one temperature of LL 128^3, MCT = MCS = 2000
        _case("ll128", n=(128, 128, 128), mct=2000, mcs=2000, tune=True),
        # the plain sampler of the learned-proposal workload: 96^3 lattices at
        # four temperatures (more than the caches hold)
        _case("ll96_batch", n=(96, 96, 96), replicas=16, mct=400, mcs=400, tune=True),
        # GHRL slabs with homeotropic faces, sides drawn from {16 .. 64}
        _case("slab_batch", model="slab", n=(0, 0, 0), replicas=48, mct=300, mcs=300, tune=True, sides=3),
        # chiral GHRL droplets with planar anchoring in a field: one field
        # value of the electric sweep
        _case("droplet_field", model="droplet", n=(96, 96, 96), replicas=8, mct=200, mcs=200, tune=True, radius=40.0,
              field=True),
        # the reference's sample droplet (25^3, homeotropic, an odd length),
        # sixteen seeds of one temperature
        _case("droplet25", model="droplet", n=(25, 25, 25), replicas=16, mct=150, mcs=100, radius=0.0, field=False),
        # the reference's chiral bulk sample (24^3 GHRL, p0 = 40)
        _case("ghrl24", model="ghrl", n=(24, 24, 24), replicas=1, mct=150, mcs=100),
        # the learned proposal on 96^3 LL lattices, every sweep measured as in
        # its autocorrelation protocol
        _case("learned_ll96", n=(96, 96, 96), replicas=4, mct=0, mcs=300, learned=True),
        # the learned proposal in chiral droplets with a field
        _case("learned_droplet", model="droplet", n=(64, 64, 64), replicas=6, mct=150, mcs=150, learned=True,
              radius=26.0, field=True),
        # training of the network on samples of the replicas' states
        _case("train", kind="train", n=(32, 32, 32), replicas=8, samples=200000, batch=8192, steps=200),
        # a configuration's energy, Q-tensor, S and per-site order parameter,
        # as the snapshot writer needs them
        _case("snapshot", kind="snapshot", n=(96, 96, 96)),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """A case of the listed ranges: any model, lattices of 8^3 to 112^3 sites
    with uneven sides (odd ones on free axes), one to many replicas."""
    what = rng.choice(["ll", "ll", "ll", "slab", "droplet", "ghrl", "pear", "learned", "learned", "train", "snapshot"])
    if what == "snapshot":
        n = [2 * _log(rng, 6, 56) for _ in range(3)]
        return {k: v for k, v in _case("", kind="snapshot", n=n).items() if k != "name"}
    if what == "train":
        return {k: v for k, v in _case("", kind="train", n=(2 * _log(rng, 6, 20),) * 3, replicas=_log(rng, 1, 12),
                                       samples=_log(rng, 20000, 300000), batch=_log(rng, 512, 16384),
                                       steps=_log(rng, 20, 200)).items() if k != "name"}
    learned = what == "learned"
    model = rng.choice(["ll", "droplet", "slab"]) if learned else what
    side = _log(rng, 8, 112)
    n = [max(4, int(side * (0.7 + 0.6 * rng.random()))) for _ in range(3)]
    more = {}
    if model == "droplet":
        n = [max(9, side + rng.choice([0, 0, 1]))] * 3
        more = {"radius": rng.choice([0.0, 0.42 * n[0]]), "field": rng.random() < 0.5}
        even = ()
    elif model == "slab" or (model == "ll" and rng.random() < 0.3):
        even = (0, 1)  # z is free
    else:
        even = (0, 1, 2)
    for q in even:
        n[q] += n[q] % 2
    sites = n[0] * n[1] * n[2]
    replicas = max(1, min(32, _log(rng, 1, 64), 4000000 // sites))
    # sweeps: about as many site updates as the listed blocks make
    sweeps = max(8, min(400, int(2.5e9 / (12.0 if learned else 1.0) / (sites * replicas))))
    mct = 0 if rng.random() < 0.2 else int(sweeps * (0.3 + 0.7 * rng.random()))
    c = _case("", model=model, n=n, replicas=replicas, mct=mct, mcs=sweeps, tune=rng.random() < 0.4, learned=learned,
              **more)
    del c["name"]
    return c


def _sides(case):
    """Replica lattices: the case's box, or cubes of mixed sides."""
    if case.get("sides"):
        r = np.random.default_rng(case["sides"])
        return [(int(s),) * 3 for s in r.choice([16, 24, 32, 48, 64], size=case["replicas"])]
    return [(case["nx"], case["ny"], case["nz"])] * case["replicas"]


def _descs(case, seed):
    out = []
    rng = np.random.default_rng(seed)
    for q, (nx, ny, nz) in enumerate(_sides(case)):
        key = dict(nx=nx, ny=ny, nz=nz, seed=int(rng.integers(1, 2**31)), stream=q)
        m = case["model"]
        if m == "ll":
            key.update(potential="ll", T=TEMPS[q % 4], zbound="free" if nz % 2 else "periodic")
        elif m == "pear":
            key.update(potential="pear", A=1.0, B1=0.04, C=0.3, T=0.7)
        elif m == "ghrl":
            key.update(potential="ghrl", k11=1.48, k22=1.0, k33=2.28, p0=40.0, T=0.9)
        elif m == "slab":
            hom = dict(anchoring="homeotropic", W=4.0)
            key.update(geometry="slab", potential="ghrl", k11=1.0, k22=0.8, k33=1.2, T=float(rng.uniform(0.8, 1.2)),
                       surfaces=[hom, hom])
        elif case["field"]:
            key.update(geometry="sphere", potential="ghrl", k11=1.0, k22=0.6, k33=1.4, p0=20.0, elecA=1.0, elecZ=1.0,
                       elecE=0.5, T=0.8, surfaces=[dict(anchoring="fg", W=1.0)], radius=case["radius"])
        else:
            key.update(geometry="sphere", potential="ghrl", k11=1.48, k22=1.0, k33=2.28, T=0.9,
                       surfaces=[dict(anchoring="homeotropic", W=4.0)], radius=case["radius"])
        out.append(mcx.replica(**key))
    return out


def _network(seed):
    """Weights of the learned proposal: a mean axis along the neighbours' sum
    and a constant concentration (what training finds first), passed through
    the hidden layers as gelu(x) - gelu(-x) = x, with small random weights
    everywhere else."""
    r = np.random.default_rng(seed)
    W1, W2, W3 = np.zeros((32, 64)), np.zeros((64, 64)), np.zeros((64, 8))
    W1[:19] = r.normal(0, 0.05, (19, 64))
    W2[:] = r.normal(0, 0.05, (64, 64))
    W3[:, :4] = r.normal(0, 0.05, (64, 4))
    for c in range(3):
        for d in range(6):
            W1[3 * d + c, 2 * c] += 1.0
            W1[3 * d + c, 2 * c + 1] -= 1.0
        for i in range(2):
            for o in range(2):
                W2[2 * c + i, 2 * c + o] += 1.0 if i == o else -1.0
            W3[2 * c + i, c] += 1.0 - 2.0 * i
    b3 = np.zeros(8)
    b3[3] = 1.3
    return np.concatenate([W1.ravel(), np.zeros(64), W2.ravel(), np.zeros(64), W3.ravel(), b3]).astype(np.float32)


def _start_weights(seed):
    r = np.random.default_rng(seed)
    W1, W3, b3 = np.zeros((32, 64)), np.zeros((64, 8)), np.zeros(8)
    W1[:19] = r.normal(0, 19 ** -0.5, (19, 64))
    W2 = r.normal(0, 0.125, (64, 64))
    W3[:, :4] = r.normal(0, 0.125, (64, 4))
    b3[3] = 1.0
    return np.concatenate([W1.ravel(), np.zeros(64), W2.ravel(), np.zeros(64), W3.ravel(), b3]).astype(np.float32)


def _field(case, seed):
    """An ordered director field with thermal noise (float32, natural order)."""
    r = np.random.default_rng(seed)
    v = r.normal(0, 0.6, (case["nx"] * case["ny"] * case["nz"], 3)) + r.normal(0, 1, 3)
    return (v / np.linalg.norm(v, axis=1, keepdims=True)).astype(np.float32)


def prepare(case, seed):
    eng = mcx.Engine(_descs(case, seed))
    if case["kind"] == "snapshot":
        eng.set_state(0, _field(case, seed))
        return {"eng": eng, "case": case, "pass": 0}
    for q in range(eng.n):
        if case["model"] == "ll":
            eng.init_homogeneous(q, 0.0, 0.0)
        else:
            eng.init_random(q, int(seed) % 2**31 + q)
    if case["tune"]:
        eng.autotune()
    eng.sweep(32)  # past the start: the step size has adapted, the states differ
    if case["kind"] == "train":
        eng.set_mlp(_start_weights(seed))
    elif case["learned"]:
        eng.set_mlp(_network(seed))
        eng.set_proposal("vmf_mlp")
    eng.sync()
    return {"eng": eng, "case": case, "pass": 0, "seed": int(seed) % 2**31}


def run(state):
    eng, case = state["eng"], state["case"]
    k = state["pass"]
    state["pass"] = k + 1
    if case["kind"] == "train":
        loss = eng.train_mlp(samples=case["samples"], batch=case["batch"], steps=case["steps"], lr=1e-3,
                             seed=state["seed"] + k, augment=mcx.AUG_FLIP | mcx.AUG_ROTATE)
        return {"loss": loss, "weights": eng.get_mlp()}
    if case["kind"] == "snapshot":
        m = eng.measure(0)
        return {"E": float(m["E"]), "Q": m["Q"], "S": float(m["S"]), "state": eng.get_state(0),
                "local": eng.local_order(0)}
    # the next value of the swept parameter, where the run sweeps one
    if case["model"] == "droplet" and case["field"]:
        eng.set_field(0.5 + 0.1 * (k % 8))
    elif eng.n == 1:
        eng.set_temperature(eng.descs[0].T - 0.01 * (k % 8))
    eng.sweep(case["mct"])
    eng.reset_stats()
    eng.sweep(case["mcs"], measure=True)
    return {"stats": np.stack([eng.stats(q) for q in range(eng.n)]), "state": [eng.get_state(q) for q in range(eng.n)]}


def work(case):
    n = [a * b * c for a, b, c in _sides(case)]
    sites = sum(n)
    if case["kind"] == "train":
        # forward, and backward to weights and activations
        return {"bytes": case["samples"] * 96 + case["steps"] * case["batch"] * 88,
                "flops": 3 * MLP_FLOPS * case["batch"] * case["steps"]}
    if case["kind"] == "snapshot":
        return {"bytes": sites * (12 + 12 + 4), "flops": sites * 400}
    # directors in and out once (and the point types of a mask); a state larger
    # than the L2 cache has to stream through it once per sweep, since every
    # sweep's step size needs the whole sweep before it
    sweeps = case["mct"] + case["mcs"]
    masked = 1 if case["model"] in ("slab", "droplet") else 0
    passes = sweeps if (12 + masked) * sites > L2_BYTES else 1
    active = 1.0
    if case["model"] == "droplet":
        active = min(1.0, 4.19 * (case["radius"] or case["nx"] / 2) ** 3 / sites * case["replicas"])
    fl = FLOPS[case["model"]] + (MLP_FLOPS if case["learned"] else 0)
    return {"bytes": passes * (24 + masked) * sites, "flops": sweeps * sites * active * fl}


def exact(case, seed):
    """A Markov chain and a training run have no 64-bit counterpart to compare
    with (a decision or a rounding early on changes all that follows); a
    measured configuration has."""
    if case["kind"] != "snapshot":
        return None
    v = _field(case, seed).astype(np.float64).reshape(case["nz"], case["ny"], case["nx"], 3)
    N = v.shape[0] * v.shape[1] * v.shape[2]
    E = 0.0
    loc = 3.0 * v[..., :, None] * v[..., None, :]
    near = loc.copy()
    for ax in range(3):
        E += 2 * float((-1.5 * (v * np.roll(v, -1, ax)).sum(-1) ** 2).sum())
        near += np.roll(loc, 1, ax) + np.roll(loc, -1, ax)
    Q = (loc.sum((0, 1, 2)) / N - np.eye(3)) / 2
    local = (np.linalg.eigvalsh(near.reshape(N, 3, 3))[:, -1] / 7 - 1) / 2
    return {"E": E / N, "Q": Q, "S": float(np.linalg.eigvalsh(Q)[-1]), "state": v.reshape(N, 3), "local": local}
