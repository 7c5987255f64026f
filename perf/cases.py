"""The work that users of this library have it do, as measured cases.

A case is one evaluation through a public entry point: the reference's own
Python call (``callTreedriver``, host arrays, FP64), the pointer call on
device arrays (``treecode_ptr``), a batch of systems, a session (fixed
particles, new charges per evaluation) and the FP64 direct sum.  Sizes,
distributions, kernels, degrees and leaf sizes are those of the benchmark's
five configurations, of the reference's Python test and of this repository's
tests, with odd particle counts among them.

``draw`` gives further cases of the same families over the ranges in between.
"""
import math

import numpy as np
import torch

import barytree_b200 as B
from barytree_b200 import selector

COULOMB, YUKAWA, REGULARIZED = int(B.Kernel.COULOMB), int(B.Kernel.YUKAWA), int(B.Kernel.REGULARIZED_COULOMB)
LAGRANGE, HERMITE = int(B.Approximation.LAGRANGE), int(B.Approximation.HERMITE)
PC, CP, CC = (int(c) for c in (B.ComputeType.PARTICLE_CLUSTER, B.ComputeType.CLUSTER_PARTICLE,
                               B.ComputeType.CLUSTER_CLUSTER))
FP64, MIXED = "fp64", "mixed"


def _case(name, call, n, **kw):
    """One case with the defaults spelled out.  nt = 0: the targets are the
    sources (n particles); otherwise nt targets of their own and n sources."""
    c = dict(name=name, call=call, n=n, nt=0, dist="cube", kernel=COULOMB, kp=0.0, approx=LAGRANGE, ctype=PC,
             theta=0.7, degree=8, leaf=2000, size_check=1.0, precision=FP64, learned=False, subtraction=False,
             systems=0)
    c.update(kw)
    if not name:
        del c["name"]
    return c


def listed():
    return [
        # the reference's Python test: a small system with singularity
        # subtraction, one call from host arrays; latency counts
        _case("call_5k_yukawa_subtraction", "host", 5000, dist="unit", kernel=YUKAWA, kp=0.5, theta=0.8, degree=4,
              leaf=50, subtraction=True),
        # a script that moved over from the reference by changing its import
        _case("call_100k_coulomb", "host", 100_000),
        # the same with the reference's fastest method, an odd particle count
        _case("call_300k_cc_yukawa", "host", 300_007, kernel=YUKAWA, kp=0.5, ctype=CC, theta=0.8),
        # potentials of a smaller charge set at many field points (a visualisation grid's worth)
        _case("call_cp_fields", "host", 30_011, nt=250_003, kernel=REGULARIZED, kp=1e-2, ctype=CP, degree=6,
              leaf=1000),
        # Hermite interpolation in FP64, Gaussian cloud of +-1 charges
        _case("call_200k_hermite", "host", 200_003, dist="gauss", approx=HERMITE, degree=6, leaf=1000,
              size_check=4.0),
        # mixed precision on device arrays: one time step of a 100k simulation
        _case("device_100k_mixed", "device", 100_000, precision=MIXED),
        # cluster-cluster Yukawa at 1M
        _case("device_1m_cc_yukawa_mixed", "device", 1_000_000, kernel=YUKAWA, kp=0.5, ctype=CC, theta=0.8,
              precision=MIXED),
        # Hermite at scale, Gaussian cloud
        _case("device_2m_hermite_mixed", "device", 2_000_003, dist="gauss", approx=HERMITE, degree=6, leaf=1000,
              size_check=4.0, precision=MIXED),
        # many independent systems per call, a thousand to two hundred thousand particles each
        _case("batch_64_systems", "batch", 200_000, dist="unit", kernel=REGULARIZED, kp=1e-3, degree=7,
              precision=MIXED, systems=64),
        # the flagship: 16M clustered particles, a learned degree per interaction
        _case("device_16m_learned", "device", 16_000_000, dist="blobs", degree=10, precision=MIXED, learned=True),
        # the matrix-vector product of an iterative solver: fixed particles, new charges from the host
        _case("session_150k_mixed", "session", 150_001, precision=MIXED),
        # the accuracy check of a run: FP64 direct sum at sampled targets
        _case("direct_10k_targets", "direct", 500_000, nt=10_000),
    ]


def _between(rng, lo, hi):
    """A whole number spread evenly in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["host", "host", "host", "device", "device", "device", "batch", "session", "direct"])
    kernel = rng.choice([COULOMB, COULOMB, YUKAWA, REGULARIZED])
    kp = {COULOMB: 0.0, YUKAWA: round(rng.uniform(0.1, 2.0), 3), REGULARIZED: 10.0 ** -rng.randint(2, 4)}[kernel]
    if call == "direct":
        return _case("", call, _between(rng, 20_000, 1_000_000), nt=_between(rng, 1000, 20_000), kernel=kernel, kp=kp)
    theta = round(rng.uniform(0.5, 0.85), 2)
    leaf = rng.choice([250, 500, 1000, 2000])
    degree = rng.randint(3, 10)
    if call == "batch":
        return _case("", call, _between(rng, 20_000, 200_000), dist="unit", kernel=kernel, kp=kp, theta=theta,
                     degree=degree, leaf=leaf, precision=rng.choice([FP64, MIXED]), systems=rng.randint(4, 48))
    ctype = rng.choice([PC, PC, CC, CP])
    approx = LAGRANGE if ctype != PC else rng.choice([LAGRANGE, LAGRANGE, HERMITE])
    size_check = 1.0
    if approx == HERMITE:
        degree, size_check = rng.randint(3, 7), 4.0
    dist = rng.choice(["cube", "gauss", "blobs"])
    if call == "host":
        n = _between(rng, 2000, 400_000)
        nt = rng.choice([0, 0, _between(rng, 2000, 400_000)])
        sub = kernel != REGULARIZED and approx == LAGRANGE and rng.random() < 0.2
        return _case("", call, n, nt=nt, dist=dist, kernel=kernel, kp=1.0 if sub and kernel == COULOMB else kp,
                     approx=approx, ctype=ctype, theta=theta, degree=degree, leaf=leaf, size_check=size_check,
                     subtraction=sub)
    n = _between(rng, 20_000, 2_000_000)
    if call == "session":
        n = min(n, 1_000_000)
    learned = call == "device" and ctype == PC and approx == LAGRANGE and kernel == COULOMB and rng.random() < 0.5
    if learned:
        theta, degree = 0.7, 10
    return _case("", call, n, dist=dist, kernel=kernel, kp=kp, approx=approx, ctype=ctype, theta=theta,
                 degree=degree, leaf=leaf, size_check=size_check, precision=MIXED, learned=learned)


def _sizes(case):
    """Particle counts of a batch's systems: log-uniform from 1,000 to n."""
    u = np.random.default_rng(case["systems"]).uniform(math.log(1000), math.log(case["n"]), case["systems"])
    return np.round(np.exp(u)).astype(np.int64)


def _counts(case):
    """(targets, sources) of the whole call."""
    if case["call"] == "batch":
        n = int(_sizes(case).sum())
        return n, n
    return case["nt"] or case["n"], case["n"]


def _positions(dist, n, g):
    if dist == "unit":
        return torch.rand(3, n, generator=g, device="cuda", dtype=torch.float64)
    if dist == "gauss":
        return (0.25 * torch.randn(3, n, generator=g, device="cuda", dtype=torch.float64)).clamp_(-1, 1)
    p = 2 * torch.rand(3, n, generator=g, device="cuda", dtype=torch.float64) - 1
    if dist == "blobs":
        # 80 % in 8 Gaussian blobs, the rest uniform
        m = int(0.8 * n) // 8
        c = 1.4 * torch.rand(8, 3, generator=g, device="cuda", dtype=torch.float64) - 0.7
        s = 0.05 * 6.0 ** torch.rand(8, generator=g, device="cuda", dtype=torch.float64)
        for i in range(8):
            b = torch.randn(3, m, generator=g, device="cuda", dtype=torch.float64) * s[i] + c[i][:, None]
            p[:, i * m:(i + 1) * m] = b.clamp_(-1, 1)
    return p


def _inputs(case, seed):
    """Device tensors: targets (3, nt), sources (3, ns), charges, and for the
    subtraction target charges and source weights; targets is sources where
    the case has no targets of its own."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    nt, ns = _counts(case)
    s = _positions(case["dist"], ns, g)
    t = _positions(case["dist"], nt, g) if case["nt"] else s
    u = torch.rand(ns, generator=g, device="cuda", dtype=torch.float64)
    q = torch.where(u < 0.5, -1.0, 1.0).to(torch.float64) if case["dist"] == "gauss" else 2 * u - 1
    w = tq = None
    if case["subtraction"]:
        # the subtraction multiplies source charges and target charges of the
        # same density: one array where the targets are the sources
        w = 0.5 + torch.rand(ns, generator=g, device="cuda", dtype=torch.float64)
        tq = q if not case["nt"] else 2 * torch.rand(nt, generator=g, device="cuda", dtype=torch.float64) - 1
    return t, s, q, w, tq


def _options(case):
    return dict(kernel=case["kernel"], kernel_param=case["kp"], approximation=case["approx"],
                compute_type=case["ctype"], theta=case["theta"], degree=case["degree"], max_source_leaf=case["leaf"],
                max_target_leaf=case["leaf"], size_check=case["size_check"],
                precision=B.PRECISION_MIXED if case["precision"] == MIXED else B.PRECISION_FP64,
                degree_policy=B.DEGREE_LEARNED if case["learned"] else B.DEGREE_FIXED)


def prepare(case, seed):
    t, s, q, w, tq = _inputs(case, seed)
    if case["learned"]:
        selector.install_default()
    call = case["call"]
    if call in ("host", "direct"):
        host = lambda a: None if a is None else a.cpu().numpy()  # noqa: E731
        hs = [host(a) for a in s]
        ht = hs if t is s else [host(a) for a in t]
        return case, (ht, hs, host(q), host(w), host(tq))
    if call == "session":
        hs = [a.cpu().numpy() for a in s]
        hq = q.cpu().numpy()
        sess = B.Session([(*hs, *hs, hq)], **_options(case))
        return case, (sess, hq, np.empty(len(hq)))
    torch.cuda.synchronize()                 # the library works on its own stream
    off = np.concatenate([[0], np.cumsum(_sizes(case))]).astype(np.int64) if call == "batch" else None
    return case, (t.contiguous(), s.contiguous(), q, torch.empty(t.shape[1], device="cuda", dtype=torch.float64), off)


def run(state):
    case, st = state
    call = case["call"]
    if call == "host":
        t, s, q, w, tq = st
        return B.callTreedriver(len(t[0]), len(s[0]), *t, tq, *s, q, w, case["kernel"], 1, [case["kp"]],
                                B.Singularity.SUBTRACTION if case["subtraction"] else B.Singularity.SKIPPING,
                                case["approx"], case["ctype"], theta=case["theta"], degree=case["degree"],
                                sourceLeafSize=case["leaf"], targetLeafSize=case["leaf"],
                                sizeCheck=case["size_check"])
    if call == "direct":
        t, s, q, _, _ = st
        return B.direct(*t, *s, q, case["kernel"], case["kp"])
    if call == "session":
        sess, q, out = st
        sess.evaluate(q, out=out)
        return out
    t, s, q, out, off = st
    ptr = [a.data_ptr() for a in (*t, *s, q, out)]
    if call == "batch":
        B.treecode_batch_ptr(len(off) - 1, off, off, *ptr, inputs_on_device=True, **_options(case))
    else:
        B.treecode_ptr(t.shape[1], s.shape[1], *ptr, inputs_on_device=True, **_options(case))
    return out


def _evaluations(nt, ns, case):
    """Kernel evaluations of one system by the treecode, estimated: leaves hold
    about 0.6 of the leaf limit, a target sees directly the leaves within the
    acceptance distance sqrt(3)/theta leaf widths, and on every coarser level
    the clusters of the shell between two levels' distances (about a third of
    them: the domain ends) through (degree + 1)^3 grid points each; a learned
    selection mostly picks degrees around 6."""
    if case["call"] == "direct":
        return float(nt) * ns
    leaf = 0.6 * case["leaf"]
    ball = 4.0 / 3.0 * math.pi * (math.sqrt(3.0) / case["theta"]) ** 3
    near = min(float(ns), ball * leaf)
    levels = max(0.0, math.log(max(1.0, ns / (ball * leaf)), 8.0))
    points = (7 if case["learned"] else case["degree"] + 1) ** 3
    far = 0.3 * 7.0 * ball * levels * points
    if case["ctype"] == CC:
        far /= max(1.0, leaf / points)
    return nt * (near + min(far, float(ns)))


def work(case):
    nt, ns = _counts(case)
    same = case["nt"] == 0
    values = (4 * ns + nt) if same else (4 * ns + 4 * nt)
    if case["subtraction"]:
        values += nt + ns
    if case["call"] == "session":
        values = ns + nt
    # a kernel evaluation: 3 differences, 5 for the squared distance, 2 for
    # the multiply-add of the charge (the reciprocal root and exp not counted)
    per = 10.0 + (3.0 if case["kernel"] == YUKAWA else 1.0 if case["kernel"] == REGULARIZED else 0.0)
    if case["call"] == "batch":
        ev = sum(_evaluations(int(n), int(n), case) for n in _sizes(case))
    else:
        ev = _evaluations(nt, ns, case)
    return {"bytes": 8.0 * values, "flops": per * ev}


def tolerance(case):
    # measured: the same system with its particles in another order (sums in
    # another order) moves FP64 potentials by up to 3.6e-14 (largest single
    # value 1.5e-13), mixed ones by up to 6e-7 (3.6e-6); mixed against FP64 by
    # up to 4.6e-7.  Drawn systems cancel more or less than these.
    if case["precision"] == FP64:
        return {"rel": 3e-13, "max": 3e-12}
    return {"rel": 2.5e-6, "max": 4e-5}


def _direct64(t, s, q, case, w=None, tq=None):
    """The direct sum in FP64 with plain torch operations."""
    nt, ns = t.shape[1], s.shape[1]
    out = torch.zeros(nt, device="cuda", dtype=torch.float64)
    k, kp = case["kernel"], case["kp"]
    cs = min(ns, 8192)
    ct = max(1, min(nt, 4_000_000 // cs))
    for a in range(0, nt, ct):
        x = t[:, a:a + ct]
        acc = torch.zeros(x.shape[1], device="cuda", dtype=torch.float64)
        for b in range(0, ns, cs):
            y = s[:, b:b + cs]
            r2 = (x[0][:, None] - y[0]).square_()
            d = x[1][:, None] - y[1]
            r2.addcmul_(d, d)
            torch.sub(x[2][:, None], y[2], out=d)
            r2.addcmul_(d, d)
            if k == REGULARIZED:
                acc += r2.add_(kp * kp).rsqrt_() @ q[b:b + cs]
                continue
            hole = r2 == 0.0
            kv = r2.rsqrt()
            if k == YUKAWA:
                kv.mul_(torch.exp(r2.sqrt().mul_(-kp)))
            kv.masked_fill_(hole, 0.0)
            if w is None:
                acc += kv @ q[b:b + cs]
                continue
            acc += kv @ (q[b:b + cs] * w[b:b + cs])
            if k == COULOMB:
                kv.mul_(torch.exp(r2.mul_(-1.0 / (kp * kp))))
            acc -= tq[a:a + ct] * (kv @ w[b:b + cs])
        out[a:a + ct] = acc
    if w is not None:
        # what the subtracted term integrates to over the whole space
        out += tq * (4.0 * math.pi / (kp * kp) if k == YUKAWA else 2.0 * math.pi * kp * kp)
    return out


def exact(case, seed):
    """The untruncated sums in 64 bits; None above 3e11 pairs (about 10 s)."""
    if case["call"] == "batch":
        sizes = [int(n) for n in _sizes(case)]
        if sum(n * n for n in sizes) > 3e11:
            return None
        t, s, q, _, _ = _inputs(case, seed)
        off = np.concatenate([[0], np.cumsum(sizes)])
        return torch.cat([_direct64(s[:, a:b], s[:, a:b], q[a:b], case) for a, b in zip(off[:-1], off[1:])])
    nt, ns = _counts(case)
    if float(nt) * ns > 3e11:
        return None
    t, s, q, w, tq = _inputs(case, seed)
    out = _direct64(t, s, q, case, w, tq)
    return out if case["call"] == "device" else out.cpu().numpy()
