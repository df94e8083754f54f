"""The calls that a prover makes through this package, as cases to be timed.

A halo2 prover over BN254 calls the library in seven ways, and each is a kind
of case here:

ntt       one transform of a device vector in place (forward, inverse with its
          n^-1, or coset), the call behind every change of basis;
host      the same three transforms through the reference-compatible symbols
          on a pageable host array, as the Rust caller makes them: the copies
          are part of the call;
lde       Lagrange values -> evaluations on the extended coset, on the device;
quotient  one quotient step on extended vectors: h = (a b) y + a, divided by
          X^n - 1 on the coset and taken back to coefficients;
msm       one commitment: scalars times bases on the device, one scalar in ten
          below 2^16 (selector and lookup columns are mostly small);
batch     many transforms of uneven sizes and directions, one graph launch;
serve     a burst of mixed jobs with host buffers through the serving loop.

Elements are uniform below the modulus in their Montgomery words, which is
what committed polynomials look like.  A state holds what a program keeps
(constants, bases, a batch handle, a running server) and its input buffers.
"""
import functools
import random

import numpy as np
import torch

import zk_gpu_b200 as zk

R_MOD = 21888242871839275222246405745257275088548364400416034343698204186575808495617
TOP = R_MOD >> 192  # top 64-bit word of the modulus
WORD = (1 << 64) - 1
DIRECTIONS = ("forward", "inverse", "coset")
PRODUCT = 256  # 32-bit multiply-adds of one 254-bit Montgomery product


# ---- constants --------------------------------------------------------------
def mont(x):
    """x in Montgomery form, 4 little-endian 64-bit words."""
    m = (x << 256) % R_MOD
    return np.array([(m >> (64 * j)) & WORD for j in range(4)], dtype=np.uint64)


def root(log_n):
    """A root of unity of order 2^log_n: the field's generator 7 raised to the cofactor."""
    return pow(7, (R_MOD - 1) >> log_n, R_MOD)


def inverse(x):
    return pow(x, -1, R_MOD)


def lde_constants(k, e):
    """(omega_n^-1, n^-1, coset generator, omega of the extended domain)"""
    return mont(inverse(root(k))), mont(inverse(1 << k)), mont(7), mont(root(k + e))


@functools.lru_cache(maxsize=1)
def small_table():
    """Montgomery forms of 0 .. 2^16 - 1."""
    step, x, out = (1 << 256) % R_MOD, 0, []
    for _ in range(1 << 16):
        out.append(x)
        x = (x + step) % R_MOD
    raw = b"".join(v.to_bytes(32, "little") for v in out)
    return np.frombuffer(raw, dtype=np.int64).reshape(-1, 4).copy()


# ---- inputs -----------------------------------------------------------------
def elements(n, seed):
    """n uniform elements on the GPU: (n, 4) int64, each below the modulus."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randint(-(1 << 63), (1 << 63) - 1, (n, 4), generator=g, device="cuda", dtype=torch.int64)
    a[:, 3] = torch.randint(0, TOP, (n,), generator=g, device="cuda", dtype=torch.int64)
    return a


def scalars(n, seed):
    """n scalars on the GPU, about one in ten of them below 2^16."""
    a = elements(n, seed)
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    at = torch.nonzero(torch.rand(n, generator=g, device="cuda") < 0.1).reshape(-1)
    v = torch.randint(0, 1 << 16, (at.numel(),), generator=g, device="cuda")
    a[at] = torch.from_numpy(small_table()).cuda()[v]
    return a


def bases(n, seed):
    """n points, seeded multiples of the generator."""
    out = torch.empty((n, 8), dtype=torch.int64, device="cuda")
    zk.g1_mul_fixed_dev(elements(n, seed), out)
    return out


def on_host(t, pinned=False):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=pinned)
    h.copy_(t)
    return h.numpy().view(np.uint64)


def direction(log_n, way):
    """omega, coset shift and output scale of one transform."""
    w = root(log_n)
    if way == "inverse":
        return {"omega": mont(inverse(w)), "scale": mont(inverse(1 << log_n))}
    if way == "coset":
        return {"omega": mont(w), "coset": mont(7)}
    return {"omega": mont(w)}


def batch_sizes(case):
    """The sizes and directions of a batch or burst: part of the case, not of its inputs."""
    r = random.Random(case["mix"])
    return [(r.randint(case["lo"], case["hi"]), r.choice(DIRECTIONS)) for _ in range(case["jobs"])]


def burst(case):
    """Kind and size of each job of a burst: 35 % NTT, 35 % LDE (x4), 30 % MSM."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["jobs"]):
        kind = r.choices(("ntt", "lde", "msm"), (35, 35, 30))[0]
        out.append((kind, r.randint(max(case["lo"], 14) if kind == "msm" else case["lo"], case["hi"])))
    return out


# ---- the cases --------------------------------------------------------------
def listed():
    return [
        # the smallest transform of a batch run alone: launch and table-lookup latency
        {"name": "ntt 2^10", "kind": "ntt", "log_n": 10, "way": "forward"},
        # an odd power of two, interpolation of one column of a mid-sized circuit
        {"name": "ntt 2^21 inverse", "kind": "ntt", "log_n": 21, "way": "inverse"},
        # one column of the largest circuit
        {"name": "ntt 2^24", "kind": "ntt", "log_n": 24, "way": "forward"},
        # one part of the extended domain as the Rust caller asks for it, host array in and out
        {"name": "host coset 2^16", "kind": "host", "log_n": 16, "way": "coset"},
        # LDE of a small circuit's column: latency again, two transforms deep
        {"name": "lde 2^13 x4", "kind": "lde", "log_n": 13, "e": 2},
        # the largest LDE, the benchmark's headline
        {"name": "lde 2^24 x4", "kind": "lde", "log_n": 24, "e": 2},
        # a quotient step of a mid-sized circuit: element-wise passes and the way back to coefficients
        {"name": "quotient 2^20", "kind": "quotient", "log_n": 18, "e": 2},
        # commitments: a small circuit, one whose column is no power of two, the largest
        {"name": "msm 2^14", "kind": "msm", "n": 1 << 14},
        {"name": "msm 300007", "kind": "msm", "n": 300007},
        {"name": "msm 2^22", "kind": "msm", "n": 1 << 22},
        # all columns of a circuit's phases at once, 2^10 .. 2^20 mixed
        {"name": "batch of 512", "kind": "batch", "jobs": 512, "lo": 10, "hi": 20, "mix": 77},
        # requests that arrive together at the serving loop
        {"name": "burst of 24", "kind": "serve", "jobs": 24, "lo": 12, "hi": 18, "mix": 99},
    ]


def log_uniform(rng, lo, hi):
    """A whole number between 2^lo and 2^hi, spread over the logarithm, hardly ever a power of two."""
    return int(2 ** rng.uniform(lo, hi))


def draw(rng):
    kind = rng.choices(("ntt", "host", "lde", "quotient", "msm", "batch", "serve"), (5, 2, 4, 2, 5, 2, 1))[0]
    if kind == "ntt":
        return {"kind": kind, "log_n": rng.randint(10, 24), "way": rng.choice(DIRECTIONS)}
    if kind == "host":
        return {"kind": kind, "log_n": rng.randint(10, 20), "way": rng.choice(DIRECTIONS)}
    if kind == "lde":
        e = rng.randint(1, 3)
        return {"kind": kind, "log_n": rng.randint(10, 26 - e), "e": e}
    if kind == "quotient":
        e = rng.randint(1, 3)
        return {"kind": kind, "log_n": rng.randint(10, 23 - e), "e": e}
    if kind == "msm":
        return {"kind": kind, "n": log_uniform(rng, 10, 22)}
    if kind == "batch":
        return {"kind": kind, "jobs": log_uniform(rng, 4, 9), "lo": 10, "hi": rng.randint(16, 20), "mix": rng.randint(1, 10**6)}
    return {"kind": kind, "jobs": rng.randint(8, 24), "lo": 12, "hi": 18, "mix": rng.randint(1, 10**6)}


# ---- preparing --------------------------------------------------------------
def prepare_batch(case, seed):
    sizes = batch_sizes(case)
    slab = elements(sum(1 << k for k, _ in sizes), seed)
    jobs, at = [], 0
    for k, way in sizes:
        jobs.append({"tensor": slab[at:at + (1 << k)], "log_n": k, **direction(k, way)})
        at += 1 << k
    return {"data": slab, "batch": zk.NttBatch(jobs)}


def prepare_serve(case, seed):
    plan = burst(case)
    largest = max([1 << s for kind, s in plan if kind == "msm"] or [1 << 14])
    server = zk.Server(hbm_budget=4 * 10**9, max_wave_jobs=64)
    basis = server.add_bases(on_host(bases(largest, seed)))
    jobs, outs, keep = [], [], []
    for i, (kind, s) in enumerate(plan):
        n = 1 << s
        shape = (12,) if kind == "msm" else (n if kind == "ntt" else 4 * n, 4)
        inp = on_host(scalars(n, seed + 10 + 2 * i) if kind == "msm" else elements(n, seed + 10 + 2 * i), pinned=True)
        out = torch.zeros(shape, dtype=torch.int64, pin_memory=True)
        view = out.numpy().view(np.uint64)
        if kind == "ntt":
            d = direction(s, DIRECTIONS[i % 3])
            jobs.append(zk.ntt_job(inp, view, s, d["omega"], d.get("coset"), d.get("scale")))
        elif kind == "lde":
            jobs.append(zk.lde_job(inp, view, s, s + 2, *lde_constants(s, 2)))
        else:
            jobs.append(zk.msm_job(inp, view, n, basis))
        keep.append(inp)
        outs.append(out)
    return {"server": server, "jobs": jobs, "outs": outs, "keep": keep}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        state = prepare_batch(case, seed)
    elif kind == "serve":
        state = prepare_serve(case, seed)
    elif kind == "msm":
        state = {"scalars": scalars(case["n"], seed), "bases": bases(case["n"], seed + 7),
                 "out": torch.zeros(12, dtype=torch.int64, device="cuda")}
    else:
        k = case["log_n"]
        if kind == "ntt":
            state = {"data": elements(1 << k, seed), "log_n": k, **direction(k, case["way"])}
        elif kind == "host":
            state = {"data": on_host(elements(1 << k, seed)), "log_n": k, "way": case["way"], **direction(k, case["way"])}
        elif kind == "lde":
            state = {"values": elements(1 << k, seed), "log_n": k, "log_ext": k + case["e"],
                     "ext": torch.empty((1 << (k + case["e"]), 4), dtype=torch.int64, device="cuda"),
                     "constants": lde_constants(k, case["e"])}
        else:
            K = k + case["e"]
            state = {"a": elements(1 << K, seed), "b": elements(1 << K, seed + 1), "y": mont(987654321),
                     "h": torch.empty((1 << K, 4), dtype=torch.int64, device="cuda"),
                     "coeffs": torch.empty(((1 << K) - (1 << k), 4), dtype=torch.int64, device="cuda"),
                     "log_n": k, "log_ext": K, "g": mont(7), "omega_ext": mont(root(K)),
                     "back": (mont(inverse(root(K))), mont(inverse(1 << K)), mont(inverse(7)))}
    state["kind"] = kind
    return state


# ---- one pass ---------------------------------------------------------------
def run_host(s):
    a, k = s["data"], s["log_n"]
    if s["way"] == "inverse":
        rc = zk.parallel_ifft_api(0, a, s["omega"], None, 1 << k, k, 0, s["scale"])
    elif s["way"] == "coset":
        rc = zk.parallel_coeff_to_extended_part_api(0, a, s["omega"], None, 1 << k, k, 0, s["coset"])
    else:
        rc = zk.parallel_fft_api(0, a, s["omega"], None, 1 << k, k, 0)
    if rc:
        raise zk.ZkGpuError(rc, "host transform")
    return a.view(np.int64)


def run(s):
    kind = s["kind"]
    if kind == "ntt":
        zk.ntt_dev(s["data"], s["log_n"], s["omega"], coset=s.get("coset"), post_scale=s.get("scale"))
        return s["data"]
    if kind == "host":
        return run_host(s)
    if kind == "lde":
        zk.lagrange_to_extended_dev(s["values"], s["ext"], s["log_n"], s["log_ext"], *s["constants"])
        return s["ext"]
    if kind == "quotient":
        zk.ew_dev(zk.EW_MUL, s["h"], s["a"], s["b"])
        zk.ew_dev(zk.EW_AXPY, s["h"], s["h"], s["a"], s["y"])
        zk.divide_by_vanishing_dev(s["h"], s["log_n"], s["log_ext"], s["g"], s["omega_ext"])
        zk.extended_to_coeff_dev(s["h"], s["coeffs"], s["log_ext"], *s["back"])
        return {"h": s["h"], "coeffs": s["coeffs"]}
    if kind == "msm":
        zk.msm_dev(s["scalars"], s["bases"], s["out"])
        return s["out"]
    if kind == "batch":
        s["batch"].run()
        return s["data"]
    tickets = [s["server"].submit(j) for j in s["jobs"]]
    for t in tickets:
        s["server"].wait(t)
    return s["outs"]


# ---- what a pass cannot do without -------------------------------------------
def ntt_products(k):
    return (1 << k) * k / 2


def msm_products(n):
    """Additions into the buckets of the best window width, six products each."""
    return min(6.0 * n * -(-254 // c) + 28.0 * (1 << (c - 1)) * -(-254 // c) for c in range(4, 21))


def work(case):
    kind = case["kind"]
    if kind in ("ntt", "host"):
        k = case["log_n"]
        b, p = 64 << k, ntt_products(k)
    elif kind == "lde":
        k, K = case["log_n"], case["log_n"] + case["e"]
        b, p = (32 << k) + (32 << K), ntt_products(k) + ntt_products(K) + (2 << k)
    elif kind == "quotient":
        K = case["log_n"] + case["e"]
        b, p = (4 * 32 << K) - (32 << case["log_n"]), ntt_products(K) + (3 << K)
    elif kind == "msm":
        b, p = 96 * case["n"], msm_products(case["n"])
    elif kind == "batch":
        b = sum(64 << k for k, _ in batch_sizes(case))
        p = sum(ntt_products(k) for k, _ in batch_sizes(case))
    else:
        b = p = 0
        for what, k in burst(case):
            if what == "msm":
                b, p = b + (32 << k), p + msm_products(1 << k)
            elif what == "ntt":
                b, p = b + (64 << k), p + ntt_products(k)
            else:
                b, p = b + (160 << k), p + ntt_products(k) + ntt_products(k + 2)
    return {"bytes": float(b), "flops": float(PRODUCT * p)}


# ---- the answer from plain integers -------------------------------------------
def exact(case, seed):
    """One small transform by the radix-2 recursion on Python integers; larger cases would take too long."""
    if case["kind"] != "ntt" or case["log_n"] > 14:
        return None
    n = 1 << case["log_n"]
    raw = elements(n, seed).cpu().numpy().tobytes()
    x = [int.from_bytes(raw[32 * i:32 * i + 32], "little") for i in range(n)]
    w, scale = root(case["log_n"]), 1
    if case["way"] == "inverse":
        w, scale = inverse(w), inverse(n)
    elif case["way"] == "coset":
        c = 1
        for i in range(n):
            x[i] = x[i] * c % R_MOD
            c = c * 7 % R_MOD

    def dft(v, w):
        if len(v) == 1:
            return v
        even, odd, t, lo, hi = dft(v[::2], w * w % R_MOD), dft(v[1::2], w * w % R_MOD), 1, [], []
        for a, b in zip(even, odd):
            b = b * t % R_MOD
            lo.append((a + b) % R_MOD)
            hi.append((a - b) % R_MOD)
            t = t * w % R_MOD
        return lo + hi

    out = b"".join((v * scale % R_MOD).to_bytes(32, "little") for v in dft(x, w))
    return torch.from_numpy(np.frombuffer(out, dtype=np.int64).reshape(n, 4).copy())
