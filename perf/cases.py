"""The work that a user of this library has it do, as cases for timing.

Every case is one call (or the two calls of a split run) on an instance of the library's own workload generators:
strings evaluated ('chain', 'prob'), exact samples drawn ('sample', 'hybrid'), a run split by a table dump ('resume'),
a batch of instances that share prefixes ('batch') and a loss with its gradient ('grad').  The sizes are those of the
benchmark, the tests and the configurations: n = 20 (width at most 10) to n = 70 (width 30, an arena of 8.6 or 17.2 GB).
Circuits come from the case, strings and uniforms from the seed.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "exact-graphstate-sampling_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

import adjoint  # noqa: E402
import gsb  # noqa: E402
import workloads  # noqa: E402

FREE = 16           # '?' bits at the end of a hybrid or resumed string (the hybrid driver's suffix length)
NPRE, NSUF = 16, 4  # prefixes per instance and suffixes per prefix of a batch


def listed():
    return [
        # one probability of a small graph state, the smallest call: latency and launches
        dict(name="prob_1_n20_c64", kind="prob", graph="gnp", n=20, circuit=1, precision=64, count=1),
        # the n = 20 configuration: a table of amplitudes, and exact samples
        dict(name="chain_1024_n20_c128", kind="chain", graph="gnp", n=20, circuit=1, precision=128, count=1024),
        dict(name="sample_100_n20_c128", kind="sample", graph="gnp", n=20, circuit=1, precision=128, count=100),
        # a sliced run's two halves on an odd size: a table dumped half way, then resumed with a sampled end
        dict(name="resume_n41_c64", kind="resume", graph="matching", n=41, circuit=3, precision=64, count=1),
        # scoring measured strings on a medium instance (width 20)
        dict(name="chain_50_n48_c64", kind="chain", graph="matching", n=48, circuit=8, precision=64, count=50),
        # exact samples of a medium instance, the targets of the gradient workload
        dict(name="sample_50_n48_c128", kind="sample", graph="matching", n=48, circuit=8, precision=128, count=50),
        # hybrid rejection sampling: forced prefix, exactly sampled end
        dict(name="hybrid_12_n60_c64", kind="hybrid", graph="matching", n=60, circuit=5, precision=64, count=12),
        # the headline instance (width 30) in both precisions: amplitudes, samples
        dict(name="chain_3_n70_c64", kind="chain", graph="matching", n=70, circuit=2, precision=64, count=3),
        dict(name="sample_2_n70_c64", kind="sample", graph="matching", n=70, circuit=2, precision=64, count=2),
        dict(name="chain_2_n70_c128", kind="chain", graph="matching", n=70, circuit=2, precision=128, count=2),
        # many instances of uneven width in one launch (the batched configuration's mix, qubits in index order)
        dict(name="batch_96_c64", kind="batch", graph="qubit", n=40, circuit=0, precision=64, count=96),
        # a training step of the n = 48 rotation layer
        dict(name="grad_128_n48", kind="grad", graph="rotations", n=48, circuit=7, precision=128, count=128),
    ]


def draw(rng):
    kind = rng.choice(["prob", "chain", "sample", "resume", "chain", "sample", "hybrid", "batch", "grad"])
    precision = 128 if kind == "grad" else rng.choice([64, 128])
    circuit = rng.randrange(1, 1000)
    if kind == "batch":
        return dict(kind=kind, graph="qubit", n=rng.randrange(24, 41), circuit=circuit, precision=precision,
                    count=round(2 ** rng.uniform(2, 6.5)))
    n = rng.randrange(20, 50) if kind == "grad" else rng.randrange(FREE + 2, 66)
    graph = "rotations" if kind == "grad" else "gnp" if n <= 32 and rng.random() < 0.5 else "matching"
    count = 1 if kind == "resume" else round(2 ** rng.uniform(0, 10))
    # seconds of one string on one GPU, roughly: the launches, and a dozen passes over a table of width 0.45 n
    one = 1e-4 + (24 if kind != "chain" else 12) * 2.0 ** (0.45 * n) * precision / 8 / 3e12
    return dict(kind=kind, graph=graph, n=n, circuit=circuit, precision=precision,
                count=max(1, min(count, int(0.03 / one))))


# ---- instances (planned once per process: a program plans a circuit once and evaluates many strings) ----

@functools.lru_cache(maxsize=None)
def instance(graph, n, circuit):
    if graph == "gnp":
        return workloads.graph_state_instance(n, 0.5, seed=circuit)
    if graph == "rotations":
        return workloads.rotation_instance(n, n, seed=circuit, order_seed=12, iters=20000)
    if graph == "qubit":
        return workloads.qubit_order_instance(n, n, circuit)
    return workloads.matching_instance(n, n, circuit, 12, 60000)


@functools.lru_cache(maxsize=None)
def batch_instances(count, nmax, circuit):
    sizes = np.random.default_rng(circuit).integers(16, nmax + 1, size=count)
    return [instance("qubit", int(n), circuit * 100003 + i) for i, n in enumerate(sizes)]


def inputs(case, seed):
    """The seed's inputs: what a user has on the host before the call."""
    rng = np.random.default_rng([seed, 20])
    kind, count = case["kind"], case["count"]
    if kind == "batch":
        ws = batch_instances(count, case["n"], case["circuit"])
        K = [len(w["steps"]) // 2 for w in ws]
        return dict(ws=ws, K=K, pre=[rng.integers(0, 2, (NPRE, k), dtype=np.int8) for k in K],
                    suf=[rng.integers(0, 2, (NPRE, NSUF, len(w["steps"]) - k), dtype=np.int8) for w, k in zip(ws, K)])
    w = instance(case["graph"], case["n"], case["circuit"])
    bits = rng.integers(0, 2, (count, len(w["steps"])), dtype=np.int8)
    ns = len(w["steps"])
    got = dict(w=w, bits=bits, K=ns // 2 if kind == "resume" else ns - FREE, seed=int(rng.integers(1 << 40)))
    if kind in ("hybrid", "resume"):
        bits[:, max(got["K"], ns - FREE):] = -1
    if kind == "grad":
        got["theta"] = torch.tensor(rng.uniform(0, 2 * math.pi, (case["n"], 3)), device="cuda")
    return got


def prepare(case, seed):
    s = inputs(case, seed)
    s["kind"], s["precision"] = case["kind"], case["precision"]
    if case["kind"] == "batch":
        s["engine"] = gsb.Batch([w["plan"] for w in s["ws"]], precision=case["precision"])
    elif case["kind"] == "grad":
        s["theta"].requires_grad_(True)
        s["engine"] = gsb.GradSweep(s["w"]["plan"], every=4)
    else:
        s["engine"] = gsb.Engine.from_text(s["w"]["plan"], precision=case["precision"])
        if case["kind"] == "hybrid":
            s["engine"].set_hybrid_prefix(s["K"])
    return s


def run(s):
    eng, kind = s["engine"], s["kind"]
    # complex64 engines report single-precision results in double arrays: kept here as what they are
    own = (lambda a: np.asarray(a, np.float32)) if s["precision"] == 64 else (lambda a: a)
    if kind == "prob":
        return own(eng.prob(s["bits"]))
    if kind == "chain":
        lp, cond = eng.chain(s["bits"])
        return own(lp), own(cond)
    if kind == "sample":
        bits, lp = eng.sample(len(s["bits"]), s["seed"])
        return bits, own(lp)
    if kind == "hybrid":
        bits, lp, cond = eng.hybrid(s["bits"], s["seed"])
        return bits, own(lp), own(cond)
    if kind == "resume":
        dump, scale, lpre = eng.prefix(s["bits"][0], s["K"])
        bits, lp, _, cond = eng.resume(s["bits"][0], s["K"], s["seed"], 0, [dump], [scale])
        return dump, own(2.0 ** scale), own(lpre), bits, own(lp), own(cond[s["K"]:])
    if kind == "batch":
        eng.set_strings(s["K"], s["pre"], s["suf"])
        return own(eng.run()[0])
    s["theta"].grad = None
    lp = adjoint.log2_prob(s["theta"], s["w"]["M0"], s["w"]["step_vertices"], s["bits"], eng)
    (-lp.mean()).backward()
    return lp.detach(), s["theta"].grad


def work(case):
    """Floating operations of the DP (two complex products and two additions per written entry; the branch norms of a
    sampled step, two products and a square per read entry; a reverse step, four products per entry), and the bytes
    of the inputs and outputs, with the widest table written and read once where it is larger than the 126 MB L2."""
    kind, e = case["kind"], case["precision"] // 8
    if kind == "batch":
        ws = batch_instances(case["count"], case["n"], case["circuit"])
        flops = 0
        for w in ws:
            st, k = w["steps"], len(w["steps"]) // 2
            flops += NPRE * sum(16 * 2.0 ** s["rn"] * (1 if i < k else NSUF) for i, s in enumerate(st))
        return dict(bytes=sum(len(w["plan"]) + NPRE * NSUF * (len(w["steps"]) + 8) for w in ws), flops=flops)
    w = instance(case["graph"], case["n"], case["circuit"])
    st, ns, c = w["steps"], len(w["steps"]), case["count"]
    first = {"prob": 0, "sample": 0, "hybrid": ns - FREE, "resume": max(ns // 2, ns - FREE)}.get(kind, ns)   # first sampled step
    flops = sum(16 * 2.0 ** s["rn"] + (18 * 2.0 ** s["r"] if i >= first else 0) + (64 * 2.0 ** s["r"] if kind == "grad" else 0)
                for i, s in enumerate(st))
    table = 2.0 ** w["width"] * e
    moved = len(w["plan"]) / c + 10 * ns + 8 + (2 * table if table > 126e6 else 0)
    if kind == "resume":
        moved += 2 * 2.0 ** st[ns // 2]["r"] * e
    if kind == "grad":
        moved += 64 * case["n"] / c
    return dict(bytes=c * moved, flops=c * flops)


# ---- the same results in plain torch, complex128 ----

def parse(text):
    """Steps of an in-place plan: kept address columns, written slots, sign mask, terms (offset, x, output, parity), M."""
    rows = [r.split() for r in text.strip().split("\n")]
    n, _, R = (int(x) for x in rows[0])
    steps = []
    for r in rows[1:]:
        _, nk, m, g, rhoc, nt = (int(x) for x in r[:6])
        t = [int(x) for x in r[6 + nk:6 + nk + 4 * nt]]
        M = torch.tensor([float(x) for x in r[6 + nk + 4 * nt:]], dtype=torch.float64).view(2, 2, 2)
        steps.append(dict(tk=[int(x) for x in r[6:6 + nk]], nk=nk, m=m, g=g, rhoc=rhoc,
                          terms=[tuple(t[4 * i:4 * i + 4]) for i in range(nt)], M=torch.view_as_complex(M)))
    return n, R, steps


def cosets(st, c0, count):
    """Base address and sign of the cosets c0 .. c0 + count - 1 (a power of two dividing c0)."""
    base = torch.zeros(1, dtype=torch.int64, device="cuda")
    odd = torch.zeros(1, dtype=torch.bool, device="cuda")
    for j in range(st["nk"]):
        if 1 << j < count:
            base = torch.cat([base, base ^ st["tk"][j]])
            odd = torch.cat([odd, odd ^ bool(st["rhoc"] >> j & 1)])
        elif c0 >> j & 1:
            base, odd = base ^ st["tk"][j], odd ^ bool(st["rhoc"] >> j & 1)
    return base, 1.0 - 2.0 * odd.to(torch.float64)


def sums(st, mem, base, sign):
    """S[x][tau]: the x = 0 and signed x = 1 sums of the cosets, for each row of mem."""
    S = [[0] * st["m"] for _ in (0, 1)]
    for tq, x, tau, par in st["terms"]:
        v = mem[:, base ^ tq]
        S[x][tau] = S[x][tau] + (v * (sign * (-1) ** par) if x else v)
    return S


def outputs(S, m0, m1):
    return [m0[:, None] * a + m1[:, None] * b for a, b in zip(*S)]


def sweep(text, bits, u=None, keep=None):
    """Rows of step bits (-1: drawn with the uniform of `u`) through every step: bits, conditionals, log2 Pr, and the
    table before step `keep` with the norm of the one before it."""
    n, R, steps = parse(text)
    bits = torch.as_tensor(np.array(bits, np.int64), device="cuda")
    B = len(bits)
    mem = torch.zeros(B, 1 << R, dtype=torch.complex128, device="cuda")
    mem[:, 0] = 1
    cond = torch.zeros(bits.shape, dtype=torch.float64, device="cuda")
    prev, before, kept = torch.ones(B, dtype=torch.float64, device="cuda"), None, None
    chunk = 1 << 24
    for k, st in enumerate(steps):
        if k == keep:
            offs = sorted({t[0] for t in st["terms"]})
            base, _ = cosets(st, 0, 1 << st["nk"])
            kept = torch.stack([mem[0, base ^ o] for o in offs], 1).reshape(-1), before
        M, N = st["M"].cuda(), 1 << st["nk"]
        spans = [(c, min(chunk, N)) for c in range(0, N, chunk)]
        if bool((bits[:, k] < 0).any()):
            nb = torch.zeros(2, B, dtype=torch.float64, device="cuda")
            for c, ln in spans:
                S = sums(st, mem, *cosets(st, c, ln))
                for b in (0, 1):
                    for o in outputs(S, M[b, 0].expand(B), M[b, 1].expand(B)):
                        nb[b] += torch.view_as_real(o).square().sum((1, 2))
            drawn = (torch.as_tensor(u[:, k], device="cuda") < nb[1] / (nb[0] + nb[1])).to(torch.int64)
            bits[:, k] = torch.where(bits[:, k] < 0, drawn, bits[:, k])
        nb = torch.zeros(B, dtype=torch.float64, device="cuda")
        for c, ln in spans:
            base, sign = cosets(st, c, ln)
            row = M[bits[:, k]]
            for tau, o in enumerate(outputs(sums(st, mem, base, sign), row[:, 0], row[:, 1])):
                nb += torch.view_as_real(o).square().sum((1, 2))
                mem[:, base ^ st["g"] if tau else base] = o
        cond[:, k] = nb / (2 * prev)
        before, prev = prev, nb
    return bits, cond, torch.log2(prev) - n, kept


def mt19937_64(seed, count):
    """`count` uniforms in [0, 1) of a 64-bit Mersenne Twister (Matsumoto and Nishimura's mt19937-64), count <= 312."""
    mask, low = (1 << 64) - 1, (1 << 31) - 1
    s = [seed & mask]
    for i in range(1, 312):
        s.append((6364136223846793005 * (s[-1] ^ s[-1] >> 62) + i) & mask)
    out = []
    for i in range(count):
        x = (s[i] & ~low & mask) | (s[(i + 1) % 312] & low)
        s[i] = s[(i + 156) % 312] ^ x >> 1 ^ (0xB5026F5AA96619E9 if x & 1 else 0)
        y = s[i]
        y ^= y >> 29 & 0x5555555555555555
        y ^= y << 17 & 0x71D67FFFEDA60000 & mask
        y ^= y << 37 & 0xFFF7EEE000000000 & mask
        out.append(min((y ^ y >> 43) / 2.0 ** 64, 1 - 2.0 ** -53))
    return out


def uniforms(case, x):
    """The library's draws: string i from the stream seeded seed + i, one per drawn step."""
    u = np.zeros((case["count"], len(x["w"]["steps"])))
    for i in range(case["count"]):
        free = np.flatnonzero((x["bits"][i] < 0) | (case["kind"] == "sample"))
        u[i, free] = mt19937_64(x["seed"] + i, len(free))
    return u


def exact(case, seed):
    x, kind = inputs(case, seed), case["kind"]
    if kind == "batch":
        rows = []
        for w, K, pre, suf in zip(x["ws"], x["K"], x["pre"], x["suf"]):
            b = np.concatenate([np.repeat(pre[:, None], NSUF, 1), suf], 2).reshape(NPRE * NSUF, -1)
            rows.append(sweep(w["plan"], b)[2].view(NPRE, NSUF))
        return torch.stack(rows)
    if kind == "grad":
        return exact_grad(x)
    plan, bits, u = x["w"]["plan"], x["bits"], None
    if kind == "sample":
        bits = np.full_like(bits, -1)
    if kind in ("sample", "hybrid", "resume"):
        u = uniforms(case, x)
    keep = x["K"] if kind == "resume" else None
    at_once = max(1, min(1 << 10, (1 << 28) >> x["w"]["width"]))
    got = [sweep(plan, bits[i:i + at_once], None if u is None else u[i:i + at_once], keep)
           for i in range(0, len(bits), at_once)]
    bits, cond, lp = (torch.cat([g[i] for g in got]) for i in range(3))
    if kind == "prob":
        return lp
    if kind == "chain":
        return lp, cond
    if kind == "sample":
        return bits.to(torch.int8), lp
    if kind == "hybrid":
        return bits.to(torch.int8), lp, cond
    table, before = got[0][3]   # stored over the root of the norm before its last step: that is its scale
    scale = torch.sqrt(before[0])
    return (table / scale, float(scale), float(torch.log2(cond[0, :keep]).sum()), bits[0].to(torch.int8),
            float(lp[0]), cond[0, keep:])


def exact_grad(x):
    """log2 Pr and the gradient of -mean log2 Pr by automatic differentiation of the sweep, one string at a time."""
    n, R, steps = parse(x["w"]["plan"])
    theta = x["theta"].clone().requires_grad_(True)
    th, ph, la = theta.unbind(1)
    c, s = torch.cos(th / 2).to(torch.complex128), torch.sin(th / 2).to(torch.complex128)
    eph, ela = torch.exp(1j * ph), torch.exp(1j * la)
    U = torch.stack([torch.stack([c, -ela * s], 1), torch.stack([eph * s, eph * ela * c], 1)], 1)
    M = (U @ torch.as_tensor(np.asarray(x["w"]["M0"]), dtype=torch.complex128, device="cuda"))[x["w"]["step_vertices"]]
    where = [cosets(st, 0, 1 << st["nk"]) for st in steps]
    grad, lps = torch.zeros_like(M), []
    for row in x["bits"]:
        Ms = M.detach().requires_grad_(True)
        mem = torch.zeros(1, 1 << R, dtype=torch.complex128, device="cuda")
        mem[0, 0] = 1
        for k, st in enumerate(steps):
            base, sign = where[k]
            m = Ms[k, int(row[k])]
            for tau, o in enumerate(outputs(sums(st, mem, base, sign), m[0:1], m[1:2])):
                mem = mem.index_copy(1, base ^ st["g"] if tau else base, o)
        lp = torch.log2(torch.view_as_real(mem[0, 0]).square().sum()) - n
        (-lp / len(x["bits"])).backward()
        grad += Ms.grad
        lps.append(lp.detach())
    M.backward(grad)
    return torch.stack(lps), theta.grad
