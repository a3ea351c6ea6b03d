"""Timing cases: the calls a user of the trial engine makes, over the sizes they are made at.

listed() names them, draw() gives more of the same ranges, prepare() makes what a program
holds before the call (an engine, a network resident on the device), run() makes one call
with the reads that follow it, work() states what it cannot do without, and exact() restates
the computed outputs in double precision with NumPy alone.

The kinds of case:

* ``test``     -- a batch of 500 ms test trials of a grown network (a synfire chain), with the
                  spike counts and first spike steps of every neuron of every trial read back;
* ``state``    -- a short probe of a grown network whose neuron states are read back, in
                  single or in double precision;
* ``growth``   -- consecutive growth trials of one network, then the weights, the synapse
                  lists, the maturation state (and the inhibition record, where it is on);
* ``group``    -- one round of a group of networks of uneven size, growing ones and test
                  batches side by side, with the same reads;
* ``topology`` -- the sampling of a new network (createNetworkForGrowth), arrays copied out.
"""
from __future__ import annotations

import math

import numpy as np

from unsupervised_growth_gb300.engine import Engine
from unsupervised_growth_gb300.network import synthetic_chain_network, synthetic_growth_network
from unsupervised_growth_gb300.workloads import DELAY_WIDTHS, chain_member, growth_member, log_uniform_sizes

STEPS_PER_MS = 50

# Growing synapses that reach both thresholds within a few trials: potentiation in steps of
# the reference's weight units, Nss 2, the training set's injections spread over 15 ms.
FAST_SYN = dict(A_P=20.0, A_D=20.0 / 1.05, ACTIVATION_THRESHOLD=10.0, SUPERSYNAPSE_THRESHOLD=40.0, WEIGHT_MAX=80.0,
                BETA=0.01, BETA_SUPERSYNAPSE=0.01, Nss=2)

TOPOLOGY = dict(A_RA2I=0.1, SIGMA_RA2I=120 / math.sqrt(2.0), B_I2RA=0.1, SIGMA_I2RA=120 / math.sqrt(2.0))


def _test(name, n_ra, n_i, groups, size, trials):
    return dict(name=name, kind="test", n_ra=n_ra, n_i=n_i, groups=groups, group_size=size, trials=trials, ms=500)


def _state(name, precision, n_ra, n_i, groups, size, trials, ms):
    return dict(name=name, kind="state", precision=precision, n_ra=n_ra, n_i=n_i, groups=groups, group_size=size,
                trials=trials, ms=ms)


def _growth(name, n_ra, n_i, trials, delays, fast=False, track_ms=0.0):
    return dict(name=name, kind="growth", n_ra=n_ra, n_i=n_i, trials=trials, delays=delays, fast=fast,
                track_ms=track_ms)


def _group(name, networks, lo, hi, tests):
    return dict(name=name, kind="group", networks=networks, lo=lo, hi=hi, tests=tests)


def _topology(name, n_ra, n_i, arrangement="sphere"):
    return dict(name=name, kind="topology", n_ra=n_ra, n_i=n_i, arrangement=arrangement)


def listed():
    return [
        # one trial of a small chain: chainTest of one trial, the smallest call there is
        _test("test_1x_300", 300, 75, 10, 15, 1),
        # one trial of the benchmark's 2000 / 550 chain
        _test("test_1x_2000", 2000, 550, 20, 100, 1),
        # a served test request: two dozen trials of a network of odd size
        _test("test_24x_777", 777, 194, 10, 38, 24),
        # the benchmark's batch: 1024 trials of the 2000 / 550 chain
        _test("test_1024x_2000", 2000, 550, 20, 100, 1024),
        # a short probe of several trials, every neuron's state read back
        _state("state_3x_333", 32, 333, 83, 8, 20, 3, 60),
        # the same in the double-precision build, the one results are checked with
        _state("state64_2x_301", 64, 301, 75, 8, 20, 2, 40),
        # growth trials of the small configuration: 300 / 100, delays 0-2 ms
        _growth("growth_2x_300", 300, 100, 2, "uniform"),
        # growth at scale: 2000 / 550, log-normal delays
        _growth("growth_3x_2000", 2000, 550, 3, "lognormal"),
        # growth with synapses that form and saturate, recording the inhibition onto every neuron
        _growth("growth_track_450", 450, 113, 1, "lognormal", fast=True, track_ms=1.0),
        # one round of a group: ten networks of uneven size, two of them test batches
        _group("group_10", 10, 200, 1600, 2),
        # createNetworkForGrowth at the reference's size, and a large network
        _topology("topology_2000", 2000, 550),
        _topology("topology_20000", 20000, 5000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges."""
    kind = rng.choice(["test", "test", "state", "state", "growth", "growth", "group", "topology"])
    if kind == "test":
        n_ra = _log_int(rng, 200, 2400)
        most = max(1, min(1024, 1024 * 2000 // n_ra))
        trials = _log_int(rng, 1, most)
        while trials > 64 and n_ra * trials > 1_000_000:   # keep a drawn batch below half the largest
            trials = trials // 2 + rng.randrange(2)
        groups = rng.randint(4, 20)
        return dict(kind="test", n_ra=n_ra, n_i=max(20, int(n_ra * rng.uniform(0.2, 0.3))), groups=groups,
                    group_size=max(2, n_ra // (groups + rng.randint(0, 8))), trials=trials, ms=500)
    if kind == "state":
        precision = rng.choice([32, 32, 64])
        n_ra = rng.randint(150, 600) if precision == 32 else rng.randint(80, 400)
        groups = rng.randint(4, 10)
        return dict(kind="state", precision=precision, n_ra=n_ra, n_i=max(10, n_ra // rng.randint(3, 5)), groups=groups,
                    group_size=max(2, n_ra // (groups + rng.randint(0, 8))), trials=rng.randint(1, 3),
                    ms=rng.randint(30, 60) if precision == 32 else rng.randint(20, 40))
    if kind == "growth":
        n_ra = _log_int(rng, 200, 2100)
        return dict(kind="growth", n_ra=n_ra, n_i=max(20, int(n_ra * rng.uniform(0.2, 0.34))), trials=rng.randint(1, 3),
                    delays=rng.choice(["uniform", "lognormal"]), fast=rng.random() < 0.5,
                    track_ms=rng.choice([0.0, 0.0, 0.0, 0.5]))
    if kind == "group":
        return dict(kind="group", networks=rng.randint(3, 12), lo=rng.randint(150, 400), hi=rng.randint(800, 1700),
                    tests=rng.randint(0, 2))
    n_ra = _log_int(rng, 200, 20000)
    return dict(kind="topology", n_ra=n_ra, n_i=max(50, int(n_ra * rng.uniform(0.2, 0.3))),
                arrangement=rng.choice(["sphere", "sphere", "square"]))


# ------------------------------------------------------------------------------ the calls


def _chain(case, seed):
    net = synthetic_chain_network(n_ra=case["n_ra"], n_i=case["n_i"], n_groups=case["groups"],
                                  group_size=min(case["group_size"], case["n_ra"] // case["groups"]), weight=500.0,
                                  seed=seed, num_steps=case["ms"] * STEPS_PER_MS)
    if case["kind"] == "state":
        # a probe shorter than the 100 ms before a trial's injections: their spread moves them to 8-10 ms
        net.training_spread = np.random.default_rng(seed).uniform(-92.0, -90.0, len(net.training))
    return net


def _growing(case, seed):
    delays = dict(delays="uniform", delay_width=2.0) if case["delays"] == "uniform" else dict(
        delays="lognormal", lognormal_mean=3.0, lognormal_sigma=1.5, delay_cap=10.0)
    net = synthetic_growth_network(n_ra=case["n_ra"], n_i=case["n_i"], n_tr=10, seed=seed, **delays,
                                   **(dict(syn=FAST_SYN) if case["fast"] else {}))
    if case["fast"]:
        net.training_spread = np.sort(np.random.default_rng(seed).uniform(0.0, 15.0, len(net.training)))
    return net


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case, seed=seed, trial=0, engine=Engine(precision=case.get("precision", 32)))
    if kind in ("test", "state"):
        state["net"] = state["engine"].load_network(_chain(case, seed))
    elif kind == "growth":
        state["net"] = state["engine"].load_network(_growing(case, seed))
        if case["track_ms"]:
            state["net"].set_inhibition_tracking(case["track_ms"])
    elif kind == "group":
        sizes = log_uniform_sizes(np.random.default_rng(case["networks"]), case["networks"], case["lo"], case["hi"])
        state["nets"] = []
        for k, n in enumerate(int(s) for s in sizes):
            if k < case["tests"]:
                state["nets"].append(("test", state["engine"].load_network(chain_member(n, seed * 100 + k, k))))
            else:
                width = DELAY_WIDTHS[k % len(DELAY_WIDTHS)]
                state["nets"].append(("growth", state["engine"].load_network(growth_member(n, seed * 100 + k, width, k))))
    return state


def _statistics(net):
    out = {}
    for which, word in enumerate(("soma", "dend", "inter")):
        out[word + "_count"], out[word + "_first"] = net.trial_stats(which)
    return out


def _grown(net):
    out = dict(weights=net.weights(), soma_count=net.trial_stats(0)[0])
    out["active"] = np.zeros((net.n_ra, net.n_ra), dtype=np.uint8)
    for i, targets in enumerate(net.synapse_list(0)):
        out["active"][i, targets] = 1
    out["supers"] = np.full((net.n_ra, 16), -1, dtype=np.int32)   # in their order, at most Nss of a row
    for i, targets in enumerate(net.synapse_list(1)):
        out["supers"][i, :len(targets)] = targets
    out["props"] = net.neuron_props()
    return out


def run(state):
    case, engine, first = state["case"], state["engine"], state["trial"]
    kind = case["kind"]
    if kind == "test":
        state["trial"] += case["trials"]
        state["net"].run_test_trials(first, case["trials"])
        return _statistics(state["net"])
    if kind == "state":
        state["trial"] += case["trials"]
        net = state["net"]
        net.run_test_trials(first, case["trials"])
        out = _statistics(net)
        for which, word in enumerate(("ra", "inter")):
            out[word + "_state"] = np.stack([net.neuron_state(b, which) for b in range(case["trials"])])
        return out
    if kind == "growth":
        state["trial"] += case["trials"]
        state["net"].run_growth_trials(first, case["trials"])
        out = _grown(state["net"])
        if case["track_ms"]:
            out["ginh"] = state["net"].inhibitory_conductance()[0]
        return out
    if kind == "group":
        state["trial"] += 3
        engine.run_group([(net, word, first, 3 if word == "test" else 1, True) for word, net in state["nets"]])
        return [_statistics(net) if word == "test" else dict(weights=net.weights(), soma_count=net.trial_stats(0)[0])
                for word, net in state["nets"]]
    state["trial"] += 1
    topology = engine.generate_topology(TOPOLOGY, case["n_ra"], case["n_i"], n_tr=10, seed=state["seed"] + first,
                                        arrangement=case["arrangement"])
    ra, inter = topology.coordinates()
    out = dict(ra=ra, inter=inter, clustered=topology.training(0), random=topology.training(1))
    for which, word in enumerate(("ra2i", "i2ra")):
        out[word + "_off"], targets, lengths = topology.connections(which)
        out[word + "_tgt"], out[word + "_len"] = _padded(targets, case), _padded(lengths, case)
    return out


def _padded(x, case):
    """A connection array at a length that is the same for every seed (about 3.1 per HVC(RA) neuron come)."""
    out = np.zeros(4 * case["n_ra"] + 64, dtype=x.dtype)
    out[:len(x)] = x
    return out


# ------------------------------------------------------------- what a call cannot do without

# Arithmetic of one neuron and one 0.02 ms step, an exponential or a division counted as one:
# the four right-hand sides of the Debrabant step (95 each) with their stage sums and noise,
# and the twelve of the Dormand-Prince step (72 each) with the tableau's sums.
RA_STEP = 4 * 95 + 190
I_STEP = 12 * 72 + 620
# RA->I (and I->RA) connections per HVC(RA) neuron of a sphere network: probability 0.1 within
# three interneuron spacings
EDGES = 3.1


def _trial_work(n_ra, n_i, steps, trials):
    flops = trials * steps * (n_ra * RA_STEP + n_i * I_STEP)
    inputs = 2 * EDGES * n_ra * 20 + n_ra * 16
    outputs = trials * 8 * (2 * n_ra + n_i)
    return flops, inputs + outputs


def _growth_work(n, n_i, trials):
    flops, bytes_ = _trial_work(n, n_i, 500 * STEPS_PER_MS, trials)
    # every trial decays every weight: read and written, with its two indicators
    return flops + trials * n * n * 3, bytes_ + trials * n * n * 18 + n * n * 8


def work(case):
    kind = case["kind"]
    n_ra, n_i = case.get("n_ra", 0), case.get("n_i", 0)
    if kind in ("test", "state"):
        size = min(case["group_size"], n_ra // case["groups"])
        flops, bytes_ = _trial_work(n_ra, n_i, case["ms"] * STEPS_PER_MS, case["trials"])
        bytes_ += (case["groups"] - 1) * size * size * 20
        if kind == "state":
            bytes_ += case["trials"] * 8 * (10 * n_ra + 7 * n_i)
    elif kind == "growth":
        flops, bytes_ = _growth_work(n_ra, n_i, case["trials"])
    elif kind == "group":
        flops = bytes_ = 0
        sizes = log_uniform_sizes(np.random.default_rng(case["networks"]), case["networks"], case["lo"], case["hi"])
        for k, n in enumerate(int(s) for s in sizes):
            f, b = _trial_work(n, n // 4, 25000, 3) if k < case["tests"] else _growth_work(n, n // 4, 1)
            flops, bytes_ = flops + f, bytes_ + b
    else:
        # each pair of either direction: a distance, a probability, a draw
        flops = 2 * n_ra * n_i * 15
        bytes_ = 24 * (n_ra + n_i) + 2 * EDGES * n_ra * 12
    return {"bytes": int(bytes_), "flops": int(flops)}


# ------------------------------------------------------------------- the same in 64 bits


def _philox(c0, c1, c2, c3, seed):
    """Philox4x32-10 over arrays of counters: four arrays of 32-bit words (as uint64)."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.asarray(x, dtype=np.uint64) for x in np.broadcast_arrays(c0, c1, c2, c3)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _unit(u):
    return np.asarray(u, dtype=np.float64) / 4294967295.0


POINTS = np.array([math.sqrt(6.0), -math.sqrt(6.0)] + [1.0] * 9 + [-1.0] * 9 + [0.0] * 10)


def _ra_rhs(y, Ge, Gi, EL, gca, mus, mud):
    vs, vd, n, h, l, r, c, ca = y
    m = 1 / (1 + np.exp(-(vs + 30) / 9.5))
    n4 = (n * n) ** 2
    kvs = (-0.1 * (vs - EL) - 60 * m ** 3 * h * (vs - 55) - 8 * n4 * (vs + 90) - 3.5 * l * (vs + 90) + 20 * mus
           + 100000 * (vd - vs) / (55 * 5000))
    kvd = (-0.1 * (vd - EL) - gca * r * r * (vd - 120) - 150 * (vd + 90) * c / (1 + 6 / ca) - Ge * vd - Gi * (vd + 80)
           + 10 * mud + 100000 * (vs - vd) / (55 * 10000))
    kn = (1 / (1 + np.exp(-(vs + 35) / 10)) - n) / (0.1 + 0.5 / (1 + np.exp((vs + 27) / 15)))
    kh = (1 / (1 + np.exp((vs + 45) / 7)) - h) / (0.1 + 0.75 / (1 + np.exp((vs + 40.5) / 6)))
    kl = (1 / (1 + np.exp(-(vs + 40) / 5)) - l) / 10
    kr = 1 / (1 + np.exp(-(vd + 5) / 10)) - r
    kc = (1 / (1 + np.exp(-(vd - 10) / 7)) - c) / 15
    kca = -0.1 * gca * r * r * (vd - 120) - 0.02 * ca
    return np.stack([kvs, kvd, kn, kh, kl, kr, kc, kca])


def _ra_step(y, Ge, Gi, EL, gca, noise, J):
    """One Debrabant step; y [8][B][N], J the four point values."""
    dt, e1, e2 = 0.02, math.exp(-0.02 / 5), math.exp(-0.01 / 5)
    par = (EL, gca, noise["white_noise_mean_soma"], noise["white_noise_mean_dend"])
    ns = math.sqrt(dt) * noise["white_noise_std_soma"] / 5000
    nd = math.sqrt(dt) * noise["white_noise_std_dend"] / 10000

    def at(x, a, b):
        x = x.copy()
        x[0] += ns * (a * J[0] + b * J[1])
        x[1] += nd * (a * J[2] + b * J[3])
        return x

    a1 = _ra_rhs(at(y, -0.01844540496323970, -0.1866426386543421), Ge, Gi, *par)
    a2 = _ra_rhs(at(y + dt * a1, 0.8017012756521233, -0.8575745885712401), Ge * e1, Gi * e1, *par)
    a3 = _ra_rhs(at(y + dt * (3 * a1 + a2) / 8, 0.5092227024816198, -0.4723392695015512), Ge * e2, Gi * e2, *par)
    a4 = _ra_rhs(at(y + dt * (-0.4526683126055039 * a1 - 0.4842227708685013 * a2 + 1.9368910834740051 * a3),
                    0.9758794209767762, 0.3060354860326548), Ge * e1, Gi * e1, *par)
    y = y + dt * (a1 / 6 - 0.005430430675258792 * a2 + 2 * a3 / 3 + 0.1720970973419255 * a4)
    return at(y, 100000.0, 0.0), Ge * e1, Gi * e1


# the 13-stage Dormand-Prince 8(7) tableau without its last stage
DP_C = [0, 1 / 18, 1 / 12, 1 / 8, 5 / 16, 3 / 8, 59 / 400, 93 / 200, 5490023248 / 9719169821, 13 / 20,
        1201146811 / 12990119798, 1]
DP_A = [[], [(0, 1 / 18)], [(0, 1 / 48), (1, 3 / 48)], [(0, 1 / 32), (2, 3 / 32)],
        [(0, 20 / 64), (2, -75 / 64), (3, 75 / 64)], [(0, 3 / 80), (3, 15 / 80), (4, 12 / 80)],
        [(0, 29443841 / 614563906), (3, 77736538 / 692538347), (4, -28693883 / 1125000000), (5, 23124283 / 1800000000)],
        [(0, 16016141 / 946692911), (3, 61564180 / 158732637), (4, 22789713 / 633445777), (5, 545815736 / 2771057229),
         (6, -180193667 / 1043307555)],
        [(0, 39632708 / 573591083), (3, -433636366 / 683701615), (4, -421739975 / 2616292301),
         (5, 100302831 / 723423059), (6, 790204164 / 839813087), (7, 800635310 / 3783071287)],
        [(0, 246121993 / 1340847787), (3, -37695042795 / 15268766246), (4, -309121744 / 1061227803),
         (5, -12992083 / 490766935), (6, 6005943493 / 2108947869), (7, 393006217 / 1396673457), (8, 123872331 / 1001029789)],
        [(0, -1028468189 / 846180014), (3, 8478235783 / 508512852), (4, 1311729495 / 1432422823),
         (5, -10304129995 / 1701304382), (6, -48777925059 / 3047939560), (7, 15336726248 / 1032824649),
         (8, -45442868181 / 3398467696), (9, 3065993473 / 597172653)],
        [(0, 185892177 / 718116043), (3, -3185094517 / 667107341), (4, -477755414 / 1098053517), (5, -703635378 / 230739211),
         (6, 5731566787 / 1027545527), (7, 5232866602 / 850066563), (8, -4093664535 / 808688257),
         (9, 3962137247 / 1805957418), (10, 65686358 / 487910083)]]
DP_B = [(0, 13451932 / 455176623), (5, -808719846 / 976000145), (6, 1757004468 / 5645159321), (7, 656045339 / 265891186),
        (8, -3867574721 / 1518517206), (9, 465885868 / 322736535), (10, 53011238 / 667516719), (11, 2 / 45)]


def _i_rhs(y, Ge, Gi):
    v, n, m, h, w = y
    kv = (-0.1 * (v + 65) - 100 * h * m ** 3 * (v - 55) - 20 * (n * n) ** 2 * (v + 80) - 500 * w * (v + 80) - Ge * v
          - Gi * (v + 75))
    kn = 0.15 * (v + 15) / (1 - np.exp(-(v + 15) / 10)) * (1 - n) - 0.2 * np.exp(-(v + 25) / 80) * n
    km = (v + 22) / (1 - np.exp(-(v + 22) / 10)) * (1 - m) - 40 * np.exp(-(v + 47) / 18) * m
    kh = 0.7 * np.exp(-(v + 34) / 20) * (1 - h) - 10 / (1 + np.exp(-(v + 4) / 10)) * h
    kw = 1 / (1 + np.exp(-v / 5)) - w
    return np.stack([kv, kn, km, kh, kw])


def _i_step(y, Ge, Gi):
    dt, k = 0.02, []
    for c, row in zip(DP_C, DP_A):
        x = y + dt * sum(a * k[s] for s, a in row) if row else y
        k.append(_i_rhs(x, Ge * math.exp(-c * dt / 2), Gi * math.exp(-c * dt / 5)))
    return y + dt * sum(b * k[s] for s, b in DP_B), Ge * math.exp(-dt / 2), Gi * math.exp(-dt / 5)


def _exact_states(case, seed):
    """The neuron states after a batch of test trials: the reference's trial with kicks at the
    0.25 ms synchronizations, over all instances at once."""
    net = _chain(case, seed)
    B, N, NI, S = case["trials"], net.n_ra, net.n_i, net.num_steps
    T = np.concatenate([[0.0], np.add.accumulate(np.full(S - 1, 0.02))])
    syncs, nt = [], 0.25
    for s in range(1, S):
        if T[s] > nt or s == S - 1:
            syncs.append(s)
            nt += 0.25
    rara = [(np.array(t, dtype=int), net.w_rara[i, t], net.d_rara[i, t]) for i, t in enumerate(net.lists("active"))]

    def csr(off, tgt, w, d):
        return [(tgt[off[i]:off[i + 1]], w[off[i]:off[i + 1]], d[off[i]:off[i + 1]]) for i in range(len(off) - 1)]

    ra2i = csr(net.ra2i_off, net.ra2i_tgt, net.ra2i_w, net.ra2i_d)
    i2ra = csr(net.i2ra_off, net.i2ra_tgt, net.i2ra_w, net.i2ra_d)
    Q = len(syncs)
    up = {k: np.zeros((Q, B, n)) for k, n in (("rr", N), ("ri", NI), ("ir", N))}

    def deliver(fired, lists, into, s):
        for b, i in zip(*np.nonzero(fired)):
            tgt, w, d = lists[i]
            at = np.searchsorted(T, T[s] + d)                  # first step whose time reaches the delivery
            q = np.searchsorted(syncs, at)
            ok = at < S
            np.add.at(into, (q[ok], b, tgt[ok]), w[ok])

    rest = [-79.97619025, -79.97268759, 0.01101284, 0.9932845, 0.0, 0.00055429, 0.00000261762353, 0.01689572]
    y = np.stack([np.full((B, N), v) for v in rest])
    Ge, Gi = np.zeros((B, N)), np.zeros((B, N))
    fs, fd = np.zeros((B, N), bool), np.zeros((B, N), bool)
    EL, gca = net.rest_potential[None], net.gca[None]
    kick = np.full(N, S + 1)
    kick[net.training] = np.searchsorted(T, net.training_spread + 100.0, side="right")
    z = np.stack([np.full((B, NI), v) for v in (-66.0, 0.125, 0.0, 0.99, 0.0)])
    Ie, Ii, fi = np.zeros((B, NI)), np.zeros((B, NI)), np.zeros((B, NI), bool)
    trial = np.arange(B)[:, None]
    words = np.stack(_philox(np.arange(2 + S // 100)[:, None, None], np.arange(NI)[None, None], trial[None],
                             (2 << 24) | net.net_id, net.seed), axis=1).reshape(-1, B, NI)
    word = np.zeros((B, NI), int)
    when = np.zeros((2, B, NI))
    for ch in range(2):
        for b in range(B):
            for i in range(NI):
                t = 0.0
                while t < 0.02:
                    t = 1000 * (-math.log(1 - words[word[b, i], b, i] / 4294967295.0) / 250.0)
                    word[b, i] += 1
                when[ch, b, i] = t
    q = 0
    for s in range(1, S):
        Ge[:, kick == s] += 3.0
        soma = fs & (y[0] < -35.0)
        fs = np.where(fs, ~soma, y[0] > -30.0)
        fd = np.where(fd, ~(y[1] < -35.0), y[1] >= -30.0)
        J = [POINTS[((w * np.uint64(30)) >> np.uint64(32)).astype(int)]
             for w in _philox(s - 1, np.arange(N)[None], trial, (1 << 24) | net.net_id, net.seed)]
        y, Ge, Gi = _ra_step(y, Ge, Gi, EL, gca, net.noise, J)
        if soma.any():
            deliver(soma, rara, up["rr"], s)
            deliver(soma, ra2i, up["ri"], s)
        inter = fi & (z[0] < -25.0)
        fi = np.where(fi, ~inter, z[0] > -20.0)
        for ch, G in ((0, Ie), (1, Ii)):
            for b, i in zip(*np.nonzero(T[s - 1] > when[ch])):
                def u():
                    word[b, i] += 1
                    return words[word[b, i] - 1, b, i] / 4294967295.0
                G[b, i] += 0.45 * u()
                gap = 1000 * (-math.log(1 - u()) / 250.0)
                while gap < 0.02:
                    gap = 1000 * (-math.log(1 - u()) / 250.0)
                    G[b, i] += 0.45 * u()
                when[ch, b, i] += gap
        z, Ie, Ii = _i_step(z, Ie, Ii)
        if inter.any():
            deliver(inter, i2ra, up["ir"], s)
        if s == syncs[q]:
            Ge = Ge + up["rr"][q] / 10000.0
            Gi = Gi + up["ir"][q]
            Ie = Ie + up["ri"][q]
            q += 1
    ra = np.stack(list(y) + [Ge, Gi], axis=-1)
    return dict(ra_state=ra, inter_state=np.stack(list(z) + [Ie, Ii], axis=-1))


def _exact_topology(case, seed):
    n_ra, n_i, sphere = case["n_ra"], case["n_i"], case["arrangement"] == "sphere"
    tag, root = 6 << 24, math.sqrt(n_i)
    if sphere:
        dphi, dz = math.pi * (3.0 - math.sqrt(5.0)), 2 / n_i
        zc = 1 - dz / 2
        a = (math.sqrt(1 - zc * zc), 0.0, zc)
        r2 = math.sqrt(1 - (zc - dz) ** 2)
        model = math.acos(a[0] * math.cos(dphi) * r2 + zc * (zc - dz))
    else:
        model = 1 / (root + 1)

    def dist(p, qs):
        if sphere:
            return np.arccos(np.minimum(qs @ p, 1.0))
        return np.sqrt(((qs - p) ** 2).sum(axis=-1))

    u = _philox(0, np.arange(n_i), 0, tag, seed)
    jit = [-0.15 * model + 2 * 0.15 * model * _unit(u[k]) for k in (0, 1)]
    inter = np.zeros((n_i, 3))
    if sphere:
        z0 = 1 - dz / 2 - np.concatenate([[0.0], np.add.accumulate(np.full(n_i - 1, dz))])
        phi = np.concatenate([[0.0], np.add.accumulate(np.full(n_i - 1, dphi))])
        theta = np.arccos(z0)
        ph, th = phi + jit[1] / np.sin(theta), theta + jit[0]
        inter = np.stack([np.cos(ph) * np.sin(th), np.sin(ph) * np.sin(th), np.cos(th)], axis=1)
    else:
        side = int(root)
        k = np.arange(side * side)
        inter[k, 0] = (k // side + 1) / (root + 1) + jit[0][k]
        inter[k, 1] = (k % side + 1) / (root + 1) + jit[1][k]
    close = model * 10.0 / 40.0
    kept, a = np.zeros((n_ra, 3)), 0
    count = 0
    while count < n_ra:
        u = _philox(0, np.arange(a, a + 4096), 1, tag, seed)
        if sphere:
            zz, ph = 2 * _unit(u[0]) - 1, 2 * math.pi * _unit(u[1])
            s = np.sin(np.arccos(zz))
            pts = np.stack([s * np.cos(ph), s * np.sin(ph), zz], axis=1)
        else:
            lo, width = 0.5 / (root + 1), 1 - 1 / (root + 1)
            pts = np.stack([lo + width * _unit(u[0]), lo + width * _unit(u[1]), np.zeros(4096)], axis=1)
        for p in pts:
            if count < n_ra and dist(p, inter).min() >= close and (count == 0 or dist(p, kept[:count]).min() >= close):
                kept[count] = p
                count += 1
        a += 4096
    out = dict(ra=kept, inter=inter)
    for part, word, src, dst in ((2, "ra2i", kept, inter), (3, "i2ra", inter, kept)):
        n = len(dst)
        u = np.stack(_philox(np.arange((n + 3) // 4)[None], np.arange(len(src))[:, None], part, tag, seed),
                     axis=-1).reshape(len(src), -1)[:, :n]
        d = np.stack([dist(p, dst) for p in src]) * 40.0 / model
        out[word + "_len"] = _padded(d[_unit(u) < 0.1 * np.exp(-d * d / (2 * TOPOLOGY["SIGMA_RA2I"] ** 2))], case)
    return out


def exact(case, seed):
    """The computed outputs of a new state's first run in 64 bits; None for the other outputs and
    for the cases it would take too long for (whole trials: 25 000 steps)."""
    if case["kind"] == "state":
        found = _exact_states(case, seed)
        keys = [w + c for w in ("soma", "dend", "inter") for c in ("_count", "_first")] + ["ra_state", "inter_state"]
    elif case["kind"] == "topology" and case["n_ra"] <= 3000:
        found = _exact_topology(case, seed)
        keys = ["ra", "inter", "clustered", "random"] + [w + c for w in ("ra2i", "i2ra") for c in ("_off", "_tgt", "_len")]
    else:
        return None
    return {k: found.get(k) for k in keys}
