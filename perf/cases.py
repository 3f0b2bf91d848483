"""The work whose speed this framework is judged by, one case per way of using it.

A case is one pass of a user's program through the public entry points, on a population that the
program already holds: generations drawn on the device, generations replayed from the reference's
own draws (the drop-in), the reference's stages one by one, many populations in one context, and the
analyses that a simulation logs.  Populations start from a pre-seeded load (carrier counts from the
neutral 1/i spectrum), so a pass meets rows as full as a run in progress has them.

listed() gives the cases, draw(rng) more of the same ranges, prepare/run/work/exact as their names say.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import clotho_gb300 as cg
from clotho_gb300 import serving
from clotho_gb300.tape import neutral_tape


def listed():
    return [
        # the shortest simulation step that is in use: a small neutral population, ten generations between
        # two looks at it; launches and latency are all of it
        _run("neutral_n1000", N=1000, A0=240, cap=1024, mu=0.01, rho=0.01, G=10, read="rows"),
        # the neutral Wright-Fisher configuration (N=1e4, mu=rho=0.01), fifty generations to the next log entry
        _run("neutral_wf_n10000", N=10_000, A0=2_700, cap=8_192, mu=0.01, rho=0.01, G=50, read="margins"),
        # a population that grows over a schedule and falls back to its founders (growth models, bottlenecks)
        {"name": "growth_n301_to_5003", "kind": "growth", "N": 5_003, "N0": 301, "A0": 900, "cap": 4_096, "mu": 0.02,
         "rho": 0.5, "T": 2, "fitness": "quadratic", "fit_param": 6.0, "p_neutral": 0.5, "G": 32, "kmax": 0, "q1": True},
        # QTL with selection (N=1e5, mu=0.1, rho=1, one trait, exp(-z^2/2)): rows above 65,536 slots
        _run("qtl_selection_n100000", N=100_000, A0=140_000, cap=1 << 19, mu=0.1, rho=1.0, T=1, fitness="gaussian_vs",
             fit_param=1.0, p_neutral=0.0, kmax=60, G=5, read="margins"),
        # wide allele spaces at a high crossover rate, ordinary population size
        _run("wide_rho5_n50000", N=50_000, A0=29_000, cap=131_072, mu=0.02, rho=5.0, T=2, fitness="gaussian",
             p_neutral=0.5, G=5, read="margins"),
        # the large population (N=1e6, four traits, rho=5, 65,536 slots), ten generations between samples
        _run("large_n1000000", N=1_000_000, A0=58_000, cap=65_536, mu=1e-3, rho=5.0, T=4, fitness="gaussian",
             p_neutral=0.0, G=10, read="margins"),
        # the drop-in, ordinary size: the host draws a generation, hands it over and takes the fitness
        # values that it draws the next one's parents from; four generations, then the log entry
        _tape("tape_n10007", N=10_007, A0=3_000, cap=8_192, mu=0.05, rho=1.0, T=1, fitness="gaussian_vs",
              fit_param=400.0, p_neutral=0.5),
        # the drop-in, large: a tape of millions of breakpoints
        _tape("tape_n200003", N=200_003, A0=20_000, cap=32_768, mu=0.005, rho=5.0, T=4, fitness="gaussian",
              p_neutral=0.0),
        # the reference's stages called one by one (its own Engine::simulate over the adapters), recombination
        # in both gametes
        dict(_tape("staged_n2001", N=2_001, A0=1_500, cap=4_096, mu=0.05, rho=2.0, T=2, fitness="gaussian",
                   p_neutral=0.25), kind="staged", q1=False),
        # the server's step: resident populations of mixed sizes advance by its chunk of eight generations and
        # the finished ones are read
        {"name": "batch_64_populations", "kind": "batch", "pops": 64, "N_lo": 1_000, "N_hi": 20_000, "G": 8,
         "burn": 60, "read_every": 16},
        # the analysis that is logged at each sampling point: allele frequencies, spectrum, means
        {"name": "frequencies_n100000", "kind": "sample", "N": 100_000, "A0": 58_000, "cap": 65_536, "T": 2,
         "sfs": 1_024},
        # pairwise differences over a sample of sequences
        {"name": "pairwise_4001_rows", "kind": "pairwise", "N": 10_000, "A0": 20_000, "cap": 20_480, "n": 4_001,
         "distances": False},
    ]


def _run(name, *, N, A0, cap, mu, rho, G, read, T=1, fitness="constant", fit_param=1.0, p_neutral=1.0, kmax=0, q1=True):
    return {"name": name, "kind": "run", "N": N, "A0": A0, "cap": cap, "mu": mu, "rho": rho, "G": G, "read": read,
            "T": T, "fitness": fitness, "fit_param": fit_param, "p_neutral": p_neutral, "kmax": kmax, "q1": q1}


def _tape(name, *, N, A0, cap, mu, rho, T, fitness, p_neutral, fit_param=1.0, q1=True):
    return {"name": name, "kind": "tape", "N": N, "A0": A0, "cap": cap, "mu": mu, "rho": rho, "T": T,
            "fitness": fitness, "fit_param": fit_param, "p_neutral": p_neutral, "kmax": 0, "q1": q1}


# ---------------------------------------------------------------------------------------------------------
def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _load(N, mu, limit=180_000):
    """(seeded alleles, capacity) of a population in progress: up to its neutral equilibrium."""
    eq = 4.0 * N * mu * (math.log(2.0 * N) + 0.58)
    return int(min(max(48, 0.7 * eq), limit)), int(min(max(512, 1.25 * eq + 20.0 * N * mu + 512), 2.8 * limit))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "growth", "tape", "tape", "staged", "batch", "sample", "pairwise"])
    if kind == "sample":
        return {"kind": kind, "N": int(_log_uniform(rng, 500, 150_000)), "A0": (A0 := int(_log_uniform(rng, 300, 60_000))),
                "cap": A0 + rng.randrange(1, 900), "T": rng.randint(1, 4), "sfs": rng.choice([64, 200, 1_024])}
    if kind == "pairwise":
        N = int(_log_uniform(rng, 1_000, 20_000))
        A0 = int(_log_uniform(rng, 500, 40_000))
        n = int(_log_uniform(rng, 20, min(2 * N, 6_000)))
        return {"kind": kind, "N": N, "A0": A0, "cap": A0 + rng.randrange(1, 600), "n": n, "distances": rng.random() < 0.3}
    if kind == "batch":
        return {"kind": kind, "pops": rng.randint(3, 96), "N_lo": 500, "N_hi": int(_log_uniform(rng, 2_000, 30_000)),
                "G": 8, "burn": 60, "read_every": 16}
    # one population; sizes and rates over the ranges of the configurations
    N = int(_log_uniform(rng, 400, {"staged": 8_000, "growth": 20_000}.get(kind, 120_000)))
    mu = _log_uniform(rng, 1e-3, 0.1)
    rho = _log_uniform(rng, 0.01, 6.0)
    A0, cap = _load(N, mu)
    T = rng.randint(1, 4)
    p_neutral = rng.choice([0.0, 0.5, 1.0])
    fitness = rng.choice(["constant", "gaussian", "gaussian_vs", "quadratic"])
    c = {"kind": kind, "N": N, "A0": A0, "cap": cap, "mu": mu, "rho": rho, "T": T, "fitness": fitness,
         "fit_param": {"gaussian_vs": 4.0 * N * mu * T, "quadratic": 8.0}.get(fitness, 1.0), "p_neutral": p_neutral,
         "kmax": 0, "q1": rng.random() < 0.8}
    if kind == "growth":
        c.update(N0=max(2, int(N * rng.uniform(0.03, 0.5))), G=rng.randint(8, 40))
    if kind == "run":
        c.update(G=rng.choice([1, 5, 10, 25]), read=rng.choice(["rows", "margins"]) if N < 5_000 else "margins")
    return c


# ---------------------------------------------------------------------------------------------------------
def _thresholds(rng, S, A, kmax):
    """Carrier probabilities k/S as 32-bit thresholds, P(k) ~ 1/k for k in [1, kmax or S-1]."""
    top = min(kmax or S - 1, S - 1)
    cdf = np.cumsum(1.0 / np.arange(1, top + 1, dtype=np.float64))
    k = np.minimum(np.searchsorted(cdf, rng.random(A) * cdf[-1], side="right") + 1, top)
    return np.minimum(np.floor(k / S * 2.0 ** 32), 2.0 ** 32 - 1).astype(np.uint32)


def _effects(rng, A, T, p_neutral):
    e = rng.standard_normal((A, T)).astype(np.float32)
    e[rng.random((A, T)) < p_neutral] = 0.0
    return e


def _start(c, seed):
    """Host arrays of the seeded start: positions, effects, thresholds, the rows' hash seed."""
    rng = np.random.default_rng([seed, c["A0"], c["N"]])
    pos = rng.random(c["A0"])
    eff = _effects(rng, c["A0"], c.get("T", 1), c.get("p_neutral", 0.0))
    return pos, eff, _thresholds(rng, 2 * c["N"], c["A0"], c.get("kmax", 0)), 1000 + seed


def _population(c, seed, **more):
    pop = cg.Population(c["N"], c["cap"], c.get("T", 1), seed=77 + seed, fitness=c.get("fitness", "constant"),
                        fit_param=c.get("fit_param", 1.0), mu=c.get("mu", 0.0), rho=c.get("rho", 0.0),
                        p_neutral=c.get("p_neutral", 0.0), q1=c.get("q1", True), max_fixed=max(c["cap"], 1 << 16), **more)
    pos, eff, thr, hash_seed = _start(c, seed)
    pop.seed_population(c["N"], pos, eff.reshape(-1), thr, hash_seed)
    return pop


def _tapes(c, seed, n):
    rng = np.random.default_rng([seed, 5, c["N"]])
    return [neutral_tape(rng, c["N"], c["mu"], c["rho"], T=c["T"], p_neutral=c["p_neutral"]) for _ in range(n)]


TAPES = 4


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        jobs = serving.synthetic_jobs(c["pops"], 1.0, seed=seed, N_range=(c["N_lo"], c["N_hi"]), G_range=(100, 200))
        batch = cg.Batch([j.desc() for j in jobs])
        batch.init()
        batch.run(c["burn"])
        batch.sync()
        return {"case": c, "batch": batch, "read": list(range(0, c["pops"], c["read_every"]))}
    if kind in ("tape", "staged"):
        tapes = _tapes(c, seed, TAPES)
        pop = _population(c, seed, max_events=max(64, max(int(t.ev_off[-1]) for t in tapes)),
                          max_mutations=max(64, max(t.M for t in tapes)))
        return {"case": c, "pop": pop, "tapes": tapes}
    s = {"case": c, "pop": _population(c, seed)}
    if kind == "growth":
        s["sizes"] = np.linspace(c["N0"], c["N"], c["G"]).astype(np.uint32)
    if kind == "pairwise":
        s["rows"] = np.random.default_rng([seed, 9]).choice(2 * c["N"], size=c["n"], replace=False).astype(np.uint32)
    return s


def _whole(info):
    return np.array([v for v in info.values() if isinstance(v, int)], np.int64)


def _slots(c):
    """Allele slots that a population of this capacity has room for: rows come in 64-word steps."""
    return (c["cap"] + 4095) // 4096 * 4096


def _columns(col, c):
    """Carriers per slot, as long as the capacity (the slots in use differ from run to run)."""
    out = np.zeros(_slots(c), np.uint32)
    out[: col.size] = col
    return out


def _genomes(pop, c):
    rows = pop.rows()
    out = np.zeros((rows.shape[0], _slots(c) // 64), np.int64)
    out[:, : rows.shape[1]] = rows.view(np.int64)
    return out


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "batch":
        batch = state["batch"]
        batch.run(c["G"])
        batch.sync()
        infos = [batch.info(i) for i in range(c["pops"])]
        stats = [batch.stats(i, 64) for i in state["read"]]
        return {"info": np.stack([_whole(i) for i in infos]), "fitness": np.array([i["mean_fitness"] for i in infos]),
                "sfs": np.stack([s["sfs"] for s in stats]), "segregating": np.array([s["segregating"] for s in stats]),
                "heterozygosity": np.array([s["heterozygosity"] for s in stats])}
    pop = state["pop"]
    if kind == "run":
        pop.run_philox(c["N"], c["G"])
        if c["read"] == "rows":
            return {"info": _whole(pop.info()), "genomes": _genomes(pop, c), "phenotypes": pop.phenotypes()}
        col, row = pop.margins()
        return {"columns": _columns(col, c), "rows": row, "fitness": pop.fitness()}
    if kind == "growth":
        pop.run_philox_schedule(state["sizes"])
        col, row = pop.margins()
        return {"info": _whole(pop.info()), "columns": _columns(col, c), "rows": row, "phenotypes": pop.phenotypes(),
                "fitness": pop.fitness()}
    if kind in ("tape", "staged"):
        fitness = []
        for tape in state["tapes"]:
            (pop.simulate if kind == "tape" else pop.simulate_staged)(tape)
            fitness.append(pop.fitness())
        out = {"info": _whole(pop.info()), "fitness": fitness, "phenotypes": pop.phenotypes()}
        if kind == "staged":
            out["genomes"] = _genomes(pop, c)
        else:
            col, out["rows"] = pop.margins()
            out["columns"] = _columns(col, c)
        return out
    if kind == "sample":
        col, row = pop.margins()
        st = pop.stats(c["sfs"])
        return {"columns": _columns(col, c), "rows": row, "sfs": st["sfs"],
                "counts": np.array([st["segregating"], st["fixed_now"]], np.int64),
                "means": np.array([st["heterozygosity"], st["mean_fitness"], *st["mean_phenotype"]])}
    d = pop.pairwise_difference(state["rows"], distances=c["distances"])
    out = {"counts": np.array([d["min"], d["max"], d["count"], d["total"]], np.int64),
           "moments": np.array([d["mean"], d["variance"]])}
    if c["distances"]:
        out["distances"] = d["distances"]
    return out


# ---------------------------------------------------------------------------------------------------------
def _words(A):
    return (A + 511) // 512 * 8


def work(case):
    """Bytes: per generation every child row written and one parent strand's worth read, per analysis the
    rows read once, tapes and results; operations: one XOR, one count and one add per pair and word."""
    c, kind = case, case["kind"]
    if kind == "batch":
        mean = (c["N_hi"] - c["N_lo"]) / math.log(c["N_hi"] / c["N_lo"])
        return {"bytes": c["pops"] * c["G"] * 2.0 * mean * 16 * 8, "flops": 0.0}
    S, W = 2.0 * c["N"], _words(c["A0"])
    if kind == "run":
        return {"bytes": c["G"] * S * W * 16 + S * W * 8, "flops": 0.0}
    if kind == "growth":
        return {"bytes": c["G"] * (c["N0"] + c["N"]) * W * 16 + S * W * 8, "flops": 0.0}
    if kind in ("tape", "staged"):
        tape = S * (4 + 1 + 4 + 8 * c["rho"] + c["mu"] * (4 + 8 + 4 * c["T"]))
        return {"bytes": TAPES * (S * W * 16 + tape + c["N"] * 8) + S * W * 8, "flops": 0.0}
    if kind == "sample":
        return {"bytes": S * W * 8 + S * 4 + c["A0"] * 4, "flops": 0.0}
    pairs = c["n"] * (c["n"] - 1) / 2
    return {"bytes": c["n"] * W * 8 + (4 * pairs if c["distances"] else 0), "flops": 3.0 * pairs * W}


# ---------------------------------------------------------------------------------------------------------
def _hash_bits(hash_seed, rows, thr, device):
    """The seeded start's bits of the given rows, bool [rows, A]: a 64-bit mix of (seed, row, slot) against
    the slot's threshold, in integers."""
    def i64(v):
        return v - (1 << 64) if v >= 1 << 63 else v

    def shr(x, n):
        return (x >> n) & ((1 << (64 - n)) - 1)

    A = thr.numel()
    key = (rows[:, None] << 32) + torch.arange(1, A + 1, device=device)[None, :]
    x = key * i64(0x9E3779B97F4A7C15) + hash_seed
    x = (x ^ shr(x, 30)) * i64(0xBF58476D1CE4E5B9)
    x = (x ^ shr(x, 27)) * i64(0x94D049BB133111EB)
    x = x ^ shr(x, 31)
    return shr(x, 32) < thr[None, :]


def _blocks(n, cells):
    step = max(1, int(cells))
    return ((i, min(n, i + step)) for i in range(0, n, step))


def _fitness64(c, z, N):
    """The fitness metrics in 64 bits: z [N, T]."""
    sig = math.sqrt(4.0 * N * c.get("mu", 0.0))
    if c["fitness"] == "gaussian":
        return 0.398942280401432677939946059934 / sig * torch.exp(-z[:, 0] ** 2 / (2.0 * sig * sig))
    if c["fitness"] == "quadratic":
        return torch.clamp(1.0 - (z[:, 0] / (c["fit_param"] * sig)) ** 2, min=0.0)
    if c["fitness"] == "gaussian_vs":
        return torch.exp(-(z ** 2).sum(1) / (2.0 * c["fit_param"]))
    return torch.ones(N, dtype=torch.float64, device=z.device)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("run", "growth", "batch"):
        return None  # drawn generation after generation on the device: no plain form of a few seconds
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    N, A, T = c["N"], c["A0"], c.get("T", 1)
    S = 2 * N
    pos, eff, thr, hash_seed = _start(c, seed)
    thr_d = torch.from_numpy(thr.astype(np.int64)).to(dev)
    eff_d = torch.from_numpy(eff.astype(np.float64)).to(dev)
    if kind == "pairwise":
        rows = torch.from_numpy(np.random.default_rng([seed, 9]).choice(2 * N, size=c["n"], replace=False)).to(dev)
        bits = torch.cat([_hash_bits(hash_seed, rows[i:j], thr_d, dev).half() for i, j in _blocks(c["n"], 2e8 / A)])
        ones = bits.sum(1, dtype=torch.float64)
        # products of 0 and 1 over at most 2^16 columns at a time: whole numbers, exact in 32 bits
        common = sum((bits[:, i:j].float() @ bits[:, i:j].float().T).double() for i, j in _blocks(A, 65_536))
        d = (ones[:, None] + ones[None, :] - 2.0 * common)[tuple(torch.triu_indices(c["n"], c["n"], 1, device=dev))]
        mean = float(d.mean())
        out = {"counts": None, "moments": np.array([mean, max(0.0, float((d * d).mean()) - mean * mean)])}
        if c["distances"]:
            out["distances"] = None
        return out
    if kind == "sample":
        col, z = torch.zeros(A, dtype=torch.float64, device=dev), torch.zeros(S, T, dtype=torch.float64, device=dev)
        for i, j in _blocks(S, 2e8 / A):
            b = _hash_bits(hash_seed, torch.arange(i, j, device=dev), thr_d, dev).double()
            col += b.sum(0)
            z[i:j] = b @ eff_d
        f = col / S
        zi = z[0::2] + z[1::2]
        # every fitness value is 1
        return {"columns": None, "rows": None, "sfs": None, "counts": None,
                "means": np.array([float((2.0 * f * (1.0 - f)).sum()), 1.0, *zi.mean(0).tolist()])}
    # the tapes' generations: the parents' rows, the breakpoints' parity, the new alleles (a column each; the
    # slots that they reuse do not matter here)
    if S * A > 1.0e10:
        return None  # over twenty seconds
    rows = torch.cat([_hash_bits(hash_seed, torch.arange(i, j, device=dev), thr_d, dev) for i, j in _blocks(S, 2e8 / A)])
    pos_d = torch.from_numpy(pos).to(dev)
    fitness = []
    for t in _tapes(c, seed, TAPES):
        keep = ~rows.all(0)  # fixed alleles leave
        rows, pos_d, eff_d = rows[:, keep], pos_d[keep], eff_d[keep]
        E = np.diff(t.ev_off.astype(np.int64))
        if c["q1"]:
            E[1::2] = 0  # the second gamete of a pair does not recombine
        ev = np.full((S, max(1, int(E.max()))), np.inf)
        for k in range(ev.shape[1]):
            has = E > k
            ev[has, k] = t.ev_pos[t.ev_off[:-1][has].astype(np.int64) + k]
        ev_d = torch.from_numpy(ev).to(dev)
        par = torch.from_numpy(t.pairs.astype(np.int64)).to(dev)
        top = 2 * par + torch.from_numpy(t.swap.astype(np.int64)).to(dev)
        child = torch.zeros(S, pos_d.numel() + t.M, dtype=torch.bool, device=dev)
        for i, j in _blocks(S, 1e8 / A):
            side = torch.zeros(j - i, pos_d.numel(), dtype=torch.bool, device=dev)
            for k in range(ev.shape[1]):
                side ^= ev_d[i:j, k, None] <= pos_d[None, :]
            child[i:j, : pos_d.numel()] = torch.where(side, rows[top[i:j] ^ 1], rows[top[i:j]])
        child[torch.from_numpy(t.mut_seq.astype(np.int64)).to(dev), torch.arange(t.M, device=dev) + pos_d.numel()] = True
        rows = child
        pos_d = torch.cat([pos_d, torch.from_numpy(t.mut_pos).to(dev)])
        eff_d = torch.cat([eff_d, torch.from_numpy(t.mut_eff.reshape(t.M, T).astype(np.float64)).to(dev)])
        z = torch.cat([rows[i:j].double() @ eff_d for i, j in _blocks(S, 2e8 / A)])
        zi = z[0::2] + z[1::2]
        if not bool((eff_d != 0.0).any()):
            zi = torch.ones_like(zi)  # no trait weight at all: the constant phenotype
        fitness.append(_fitness64(c, zi, N).cpu().numpy())
    out = {"info": None, "fitness": fitness, "phenotypes": zi.cpu().numpy()}
    return out | ({"genomes": None} if kind == "staged" else {"columns": None, "rows": None})
