"""What a user of the sampler has it do, as measurable cases.

Kinds of case, each one pass through the public entry points (the C ABI
behind gpuropolis_gb300.Sampler):

  block    one iteration of the sampling loop (main.cu:1156-1239) with the
           chains resident on the device: a block of MH steps, then the
           re-draw of the chains below the cutoff
  outer    the same iteration with the state read back to the host, as a
           program that writes every block's samples does
  batched  the same for many datasets of uneven size behind one handle, the
           blocks replayed from a captured graph, the re-draw per dataset
  hmc      a block whose constant moves are Hamiltonian
  grad     d log-likelihood / d constants of every chain
  score    prior and likelihood of every chain, without stepping
  select   what follows a block: the MAP chain, the candidates for the k best
           lines, and the re-draw below the quantile

Populations are drawn like the sampler's own initial state (ops uniform,
constants 10^U{-4..3} N(0, 1)) and stepped a little before they are handed
over, so that a pass meets a running population; the score, gradient and
Hamiltonian cases fit models of a fixed form.
"""
import ctypes
import math

import numpy as np
import torch

import gpuropolis_gb300 as g

OPS = {
    "reference": g.OPSET_REFERENCE,                         # all 27 ops of the default build
    "basic": g.OPSET_BASIC,                                 # + - * / log exp pow x const
    "multi": [g.CONST, g.A, g.B, g.PLUS, g.MINUS, g.TIMES, g.DIV, g.SIN, g.COS,
              g.X1, g.X2, g.X3, g.EXP],                     # three input variables
}
RNG = {"lcg": g.RNG_LCG, "philox": g.RNG_PHILOX}
MOVES = {"reference": g.CONST_REFERENCE, "walk": g.CONST_RANDOM_WALK, "hmc": g.CONST_HMC}


def listed():
    return [
        # a try-out: a handful of chains on a small table of data, the default build's options
        dict(name="block_64", kind="block", chains=64, length=31, points=50, data="quad", ops="reference",
             moves="reference", rng="lcg", steps=20, burn=20),
        # the small everyday run: 1,024 chains of the quadratic, blocks of 1000 steps
        dict(name="block_1k", kind="block", chains=1024, length=31, points=101, data="quad", ops="basic",
             moves="walk", rng="lcg", steps=1000, burn=200),
        # a mid-size run on awkward sizes: odd chain count, long programs, the counter-based stream
        dict(name="block_10k_odd", kind="block", chains=10007, length=127, points=1501, data="expdecay",
             ops="reference", moves="reference", rng="philox", steps=60, burn=40),
        # the large run: 131,072 chains, 250 points
        dict(name="block_131k", kind="block", chains=131072, length=63, points=250, data="expdecay", ops="basic",
             moves="walk", rng="lcg", steps=400, burn=100),
        # data too large to stage: 65,536 points of three variables
        dict(name="block_3var_16k", kind="block", chains=16384, length=127, points=65536, data="multivar",
             ops="multi", moves="walk", rng="lcg", steps=20, burn=20),
        # the command-line tool's loop: every block's state comes back to the host
        dict(name="outer_32k", kind="outer", chains=32768, length=31, points=500, data="quad", ops="reference",
             moves="reference", rng="lcg", steps=200, burn=100),
        # 256 datasets of 8 to 4,096 points in one launch, captured blocks
        dict(name="batched_256", kind="batched", chains=131072, length=47, sets=256, smallest=8, largest=4096,
             ops="basic", moves="walk", rng="lcg", steps=100, blocks=2, burn=100),
        # gradient moves of the constants of one model: 8 leapfrog steps
        dict(name="hmc_65k", kind="hmc", chains=65536, length=31, points=1024, form="rational", every=0, leap=8,
             rng="lcg", steps=10, burn=4),
        # gradient moves beside structure moves, three variables
        dict(name="hmc_3var_2k", kind="hmc", chains=2048, length=63, points=16384, form="free", every=5, leap=8,
             rng="lcg", steps=5, burn=10),
        # an external optimiser's gradient of a population's constants
        dict(name="grad_65k", kind="grad", chains=65536, length=31, points=1024),
        # scores of a saved population on another, larger dataset
        dict(name="score_131k", kind="score", chains=131072, length=31, points=4096),
        # between two blocks: MAP, best lines, re-draw
        dict(name="select_131k", kind="select", chains=131072, length=63, best=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "outer", "batched", "hmc", "grad", "score", "select"])
    c = dict(kind=kind, chains=_log_int(rng, 64, 131072), length=rng.choice([15, 31, 63, 127]))
    if kind in ("block", "outer"):
        data = rng.choice(["quad", "expdecay", "multivar"] if kind == "block" else ["quad", "expdecay"])
        c.update(points=_log_int(rng, 30, 20000), data=data,
                 ops="multi" if data == "multivar" else rng.choice(["reference", "basic"]),
                 moves=rng.choice(["reference", "walk"]), rng=rng.choice(["lcg", "philox"]),
                 burn=rng.randrange(10, 50))
        # about as much work as a large listed case at most
        room = 6e9 / (c["chains"] * (c["points"] + 20.0 * c["length"]))
        c["steps"] = int(max(1, min(500, _log_int(rng, 10, 500), room)))
        c["burn"] = int(max(1, min(c["burn"], room)))
        if kind == "outer":
            c["chains"] = min(c["chains"], 40000)
    elif kind == "batched":
        c["sets"] = rng.choice([5, 16, 60, 256])
        c["chains"] = c["sets"] * _log_int(rng, 8, 131072 // c["sets"])
        c.update(length=rng.choice([31, 47, 63]), smallest=8, largest=_log_int(rng, 100, 4096), ops="basic",
                 moves=rng.choice(["reference", "walk"]), rng=rng.choice(["lcg", "philox"]),
                 steps=rng.randrange(10, 60), blocks=rng.randrange(1, 4), burn=rng.randrange(5, 30))
    elif kind == "hmc":
        c.update(points=_log_int(rng, 50, 4096), form=rng.choice(["rational", "free"]), leap=rng.choice([1, 4, 8]),
                 rng=rng.choice(["lcg", "philox"]), burn=2)
        c["every"] = 0 if c["form"] == "rational" else 5
        c["length"] = 31 if c["form"] == "rational" else rng.choice([31, 63])
        c["chains"] = min(c["chains"], 65536, int(6e7 / c["points"]) + 64)
        c["steps"] = rng.randrange(2, 9)
    elif kind in ("grad", "score"):
        c.update(length=rng.choice([31, 63]), points=_log_int(rng, 30, 4096))
        c["chains"] = min(c["chains"], 65536) if kind == "grad" else c["chains"]
        if kind == "grad":
            c["chains"] = min(c["chains"], int(6.7e7 / c["points"]) + 64)
    else:
        c["best"] = rng.randrange(1, 64)
    return c


# ---- data ------------------------------------------------------------------

def _quad(r, n):
    x = r.uniform(0, 10, n)
    return x, 2.5 * x ** 2 - 1.3 * x + 0.7 + r.normal(0, 0.1, n), np.full(n, 0.1)


def _expdecay(r, n):
    x = r.uniform(0, 50, n)
    f = r.uniform(50, 150) * np.exp(-r.uniform(0.01, 0.2) * x) + r.uniform(-5, 5)
    s = 0.05 * np.std(f)
    return x, f + r.normal(0, s, n), np.full(n, s)


def _multivar(r, n):
    x1, x2, x3 = r.normal(0, 1, (3, n))
    return x1, x2, x3, np.sin(x1) * x2 + np.exp(-x3 ** 2) + r.normal(0, 0.05, n), np.full(n, 0.05)


def _f32(cols):
    return [np.ascontiguousarray(c, np.float32) for c in cols]


def _dataset(name, r, n):
    return _f32({"quad": _quad, "expdecay": _expdecay, "multivar": _multivar}[name](r, n))


# ---- populations -----------------------------------------------------------

def _initial(r, chains, length, ops):
    ops = np.asarray(ops, np.int32)
    P = ops[r.integers(0, len(ops) - 1, (length, chains), dtype=np.int32)]
    C = r.standard_normal((length, chains), np.float32)
    C *= (10.0 ** np.arange(-4, 4)).astype(np.float32)[r.integers(0, 8, (length, chains), dtype=np.int8)]
    return P, C


# Models of a fixed form over the full op set: (heap node, op) of the nodes
# that are read, and the constants' typical values by node; a path that ends
# at node 16, 18, ... goes on through A nodes to the input variable.
FORMS = {
    # (c2 + x (c9 + c18 x)) / (1 + x (c15 + c30 x))
    "rational": ([(1, g.DIV), (2, g.CPLUS), (4, g.TIMES), (8, g.A), (9, g.CPLUS), (18, g.CTIMES), (3, g.PLUS),
                  (6, g.ONE), (7, g.TIMES), (14, g.A), (15, g.CPLUS), (30, g.CTIMES)],
                 {2: 1.0, 9: 0.5, 18: -0.7, 15: 0.1, 30: 0.3}, (16, 36, 28, 60)),
    # c1 + c2 exp(c8 x)
    "decay": ([(1, g.CPLUS), (2, g.CTIMES), (4, g.EXP), (8, g.CTIMES)], {1: 0.3, 2: 1.5, 8: -0.4}, (16,)),
    # c1 + c2 sin(c8 + c16 x)
    "wave": ([(1, g.CPLUS), (2, g.CTIMES), (4, g.SIN), (8, g.CPLUS), (16, g.CTIMES)],
             {1: 0.2, 2: 1.2, 8: 0.5, 16: 1.7}, (32,)),
    # c1 + c2 (c8 + x)^c4
    "power": ([(1, g.CPLUS), (2, g.CTIMES), (4, g.CPOW), (8, g.CPLUS)], {1: -0.5, 2: 0.2, 4: 1.3, 8: 5.0}, (16,)),
}


def _value(form, c, x):
    if form == "rational":
        return (c[2] + x * (c[9] + c[18] * x)) / (1 + x * (c[15] + c[30] * x))
    if form == "decay":
        return c[1] + c[2] * torch.exp(c[8] * x)
    if form == "wave":
        return c[1] + c[2] * torch.sin(c[8] + c[16] * x)
    return c[1] + c[2] * (c[8] + x) ** c[4]


def _form_length(form):
    """Description length: a leaf 1, a unary node 1 more than its child, one with a constant 2, a binary 1."""
    ops = dict(FORMS[form][0])

    def length(j):
        o = ops.get(j, g.A)
        if o == g.ONE or (o == g.A and 2 * j not in ops):
            return 1                     # 1, or A nodes down to the input variable
        if o == g.A:
            return length(2 * j)
        if o in (g.CPLUS, g.CTIMES, g.CPOW):
            return 2 + length(2 * j)
        if o in (g.EXP, g.SIN):
            return 1 + length(2 * j)
        return 1 + length(2 * j) + length(2 * j + 1)
    return length(1)


def _modelled(r, chains, length, forms):
    """Chains of the given forms in turn, constants 5% around the typical
    values; nodes that are not read hold random ops and constants."""
    P, C = _initial(r, chains, length, OPS["reference"])
    C = np.clip(C, -100.0, 100.0)
    for k, form in enumerate(forms):
        ops, consts, inputs = FORMS[form]
        for j, o in ops:
            P[j - 1, k::len(forms)] = o
        for j in inputs:
            while j <= length:
                P[j - 1, k::len(forms)] = g.A
                j *= 2
        n = len(range(k, chains, len(forms)))
        for j, v in consts.items():
            C[j - 1, k::len(forms)] = v * (1 + 0.05 * r.standard_normal(n))
    return np.ascontiguousarray(P), np.ascontiguousarray(C)


def _model_data(r, n, forms):
    """Data of the first form with its typical constants."""
    x = r.uniform(-3, 3, n)
    c = {j: torch.tensor(v, dtype=torch.float64) for j, v in FORMS[forms[0]][1].items()}
    f = _value(forms[0], c, torch.from_numpy(x)).numpy()
    return _f32((x, f + r.normal(0, 0.02, n), np.full(n, 0.02)))


def _rows(case, r):
    """(programs, constants, data) of a score or grad case."""
    forms = ["rational"] if case["kind"] == "grad" else list(FORMS)
    data = _model_data(r, case["points"], forms)
    P, C = _modelled(r, case["chains"], case["length"], forms)
    return forms, P, C, data


# ---- states ----------------------------------------------------------------

class _View:
    """A device array of the handle, for torch (the handle lives as long as the view)."""

    def __init__(self, sampler, pointer, shape, kind):
        self.sampler = sampler
        self.__cuda_array_interface__ = dict(data=(pointer, False), shape=shape, typestr=kind, version=2)


def _device_state(s):
    """P, C, prior, likelihood of a handle as tensors on the device (gpr_device_state)."""
    p = [ctypes.c_void_p() for _ in range(4)]
    s._check(s.lib.gpr_device_state(s.h, *[ctypes.byref(v) for v in p]))
    shapes = [(s.PL, s.N), (s.PL, s.N), (s.N,), (s.N,)]
    return [torch.as_tensor(_View(s, v.value, sh, k), device="cuda")
            for v, sh, k in zip(p, shapes, ("<i4", "<f4", "<f8", "<f8"))]


_stream = None


def _sampler(case, **kw):
    """A handle on the one stream that a program steps its chains on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return g.Sampler(case["chains"], program_length=case["length"], stream=_stream.cuda_stream, **kw)


def prepare(case, seed):
    r = np.random.default_rng(seed)
    kind = case["kind"]
    state = dict(kind=kind, seed=int(seed) % 1000000, steps=case.get("steps"))
    if kind in ("block", "outer", "batched"):
        three = case.get("data") == "multivar"
        s = _sampler(case, ops=OPS[case["ops"]], rng=RNG[case["rng"]], const_proposal=MOVES[case["moves"]],
                     rw_sd=0.1, n_vars=3 if three else 1)
        if kind == "batched":
            # sizes log-uniform over the range, the ends among them
            lo, hi, n = case["smallest"], case["largest"], case["sets"]
            sizes = np.exp(r.uniform(np.log(lo), np.log(hi), n)).round().astype(int)
            sizes[0], sizes[-1] = lo, hi
            s.set_batched_data([_dataset("expdecay" if i % 2 else "quad", r, k) for i, k in enumerate(sizes)])
        elif three:
            s.set_data3(*_dataset("multivar", r, case["points"]))
        else:
            s.set_data(*_dataset(case["data"], r, case["points"]))
        s.set_state(*_initial(r, case["chains"], case["length"], OPS[case["ops"]]))
        s.run_block(case["burn"], state["seed"])
        if kind == "batched":
            s.capture_blocks(case["blocks"], case["steps"])
            state["blocks"] = case["blocks"]
    elif kind == "hmc":
        if case["form"] == "rational":
            P, C = _modelled(r, case["chains"], case["length"], ["rational"])
            s = _sampler(case, ops=OPS["reference"], rng=RNG[case["rng"]], const_proposal=MOVES["hmc"])
            s.set_data(*_model_data(r, case["points"], ["rational"]))
        else:
            P, C = _initial(r, case["chains"], case["length"], OPS["multi"])
            s = _sampler(case, ops=OPS["multi"], rng=RNG[case["rng"]], const_proposal=MOVES["hmc"], n_vars=3)
            s.set_data3(*_dataset("multivar", r, case["points"]))
        s.set_moves(case["every"], 0.0005, case["leap"])
        s.set_state(P, C)
        s.run_block(case["burn"], state["seed"])
    elif kind in ("grad", "score"):
        _, P, C, data = _rows(case, r)
        s = _sampler(case)
        s.set_data(*data)
        s.set_state(P, C)
    else:
        s = _sampler(case, ops=OPS["basic"])
        s.set_state(*_initial(r, case["chains"], case["length"], OPS["basic"]))
        s.set_scores(*_scores(r, case["chains"]))
        state["best"] = case["best"]
    s.sync()
    state["s"] = s
    return state


def _scores(r, n):
    """Priors and likelihoods of a population: likelihoods over many decades, some chains invalid."""
    prior = -r.gamma(40.0, 5.0, n)
    lik = -np.abs(r.normal(0, 1e3, n)) * 10.0 ** r.integers(-2, 4, n)
    lik[r.random(n) < 0.05] = -np.inf
    prior[r.random(n) < 0.01] = np.nan
    return prior, lik


def run(state):
    s, kind = state["s"], state["kind"]
    if kind in ("block", "outer"):
        state["seed"] += 1
        s.run_block(state["steps"], state["seed"])
        if kind == "outer":
            redrawn, cutoff = s.resample(0, 0.5, state["seed"])
            P, C, prior, lik = s.get_state()
            return dict(redrawn=redrawn, cutoff=cutoff, P=P, C=C, prior=prior, lik=lik)
        s._check(s.lib.gpr_resample(s.h, 0, 0.5, state["seed"], None, None))     # queued, nothing read back
        return _device_state(s)
    if kind == "batched":
        state["seed"] += state["blocks"]
        s.run_captured([state["seed"] + b for b in range(state["blocks"])])
        s._check(s.lib.gpr_resample_datasets(s.h, 0, 0.5, state["seed"], None, None))
        return _device_state(s)
    if kind == "hmc":
        state["seed"] += 1
        s.run_block(state["steps"], state["seed"])
        return _device_state(s)
    if kind == "grad":
        grad, lik = s.loglik_grad()
        return dict(grad=grad, lik=lik)
    if kind == "score":
        prior, lik = s.evaluate()
        return dict(prior=prior, lik=lik)
    chain, post = s.map_chain()
    chains, count, threshold = s.top_chains(state["best"], 1e-3, capacity=4 * state["best"] + 1000)
    redrawn, cutoff = s.resample(0, 0.5, state["seed"])
    P, C, _, _ = _device_state(s)
    return dict(chain=chain, post=post, chains=chains, count=count, threshold=threshold, redrawn=redrawn,
                cutoff=cutoff, P=P, C=C)


def work(case):
    """Bytes: the state, the data and the scores read or written once.  Flops: per step and chain, a program
    of about five nodes at every point with its Gaussian term, and the proposal of every constant."""
    n, pl, kind = case["chains"], case["length"], case["kind"]
    state = 8.0 * pl * n
    if kind == "select":
        return dict(bytes=32.0 * n + state / 2, flops=0)
    if kind == "batched":
        lo, hi = case["smallest"], case["largest"]
        points = (hi - lo) / math.log(hi / lo)           # mean of a log-uniform size
        data, steps = 12.0 * points * case["sets"], case["steps"] * case["blocks"]
    else:
        points, steps = case["points"], case.get("steps", 1)
        data = points * (20.0 if case.get("data") == "multivar" or case.get("form") == "free" else 12.0)
    if kind in ("grad", "score"):
        per = (3 if kind == "grad" else 1) * 9.0 * points
        out = 8.0 * n * (pl + 1 if kind == "grad" else 2)
        return dict(bytes=state + data + out, flops=per * n)
    if kind == "hmc":
        return dict(bytes=2 * state + data + 16.0 * n, flops=steps * n * case["leap"] * 3 * 9.0 * points)
    return dict(bytes=2 * state + data + 16.0 * n, flops=steps * n * (9.0 * points + 60.0 * pl))


def exact(case, seed):
    kind = case["kind"]
    r = np.random.default_rng(seed)
    if kind == "select":
        _initial(r, case["chains"], case["length"], OPS["basic"])
        prior, lik = _scores(r, case["chains"])
        post = prior + lik
        up = np.sort(np.where(np.isnan(post), -np.inf, post))    # NaN lowest: -inf and NaN are below every cutoff
        cut = up[int(len(up) * 0.5)]
        return dict(chain=None, post=float(up[-1]), chains=None, count=None, threshold=float(up[len(up) - case["best"]]),
                    redrawn=None, cutoff=float(cut), P=None, C=None)
    if kind not in ("grad", "score"):
        return None                                              # a stochastic trajectory has no closed form
    forms, P, C, data = _rows(case, r)
    x, y, sd = [torch.from_numpy(v).cuda().double() for v in data]
    C64 = torch.from_numpy(C).cuda().double()
    n, pl = case["chains"], case["length"]
    lik = torch.empty(n, dtype=torch.float64, device="cuda")
    grad = torch.zeros((pl, n), dtype=torch.float64, device="cuda")
    norm = float((0.5 * math.log(2 * math.pi) + torch.log(sd)).sum())
    for k, form in enumerate(forms):
        nodes = list(FORMS[form][1])
        idx = torch.arange(k, n, len(forms), device="cuda")
        for part in torch.split(idx, max(1, (1 << 24) // max(1, len(x)))):
            c = {j: C64[j - 1, part][:, None].requires_grad_(kind == "grad") for j in nodes}
            res = (_value(form, c, x[None, :]) - y) / sd
            ll = -0.5 * (res * res).sum(1)
            if kind == "grad":
                for j, d in zip(nodes, torch.autograd.grad(ll.sum(), [c[j] for j in nodes])):
                    grad[j - 1, part] = d[:, 0]
            lik[part] = ll.detach() - norm
    if kind == "grad":
        return dict(grad=grad.cpu().numpy(), lik=lik.cpu().numpy())
    length = torch.tensor([_form_length(f) for f in forms], dtype=torch.float64, device="cuda")
    length = length[torch.arange(n, device="cuda") % len(forms)]
    prior = -length * math.log(len(OPS["reference"]) + 1.0) - (math.log(math.pi) + torch.log1p(C64 * C64)).sum(0)
    return dict(prior=prior.cpu().numpy(), lik=lik.cpu().numpy())
