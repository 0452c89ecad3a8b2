"""The work a prover has this library do, as timed cases: multi-scalar multiplications over G1 and
G2, number-theoretic transforms over Fr, and the two chains a Groth16 prover is made of.

A case is a dict of plain values:
  kind   "msm"      sum s_i P_i over `n` resident bases; `group` 1 or 2; `scalars` the mix of
                    scalar values; `table` whether the key is held as a fixed-base table
         "ntt"      in-place transforms of `count` vectors of 2^log_n elements in turn; `inverse` their
                    direction
         "witness"  the quotient polynomial's chain of seven transforms of 2^log_n elements on the
                    coset of `coset`
         "proof"    one served proving request of 2^log_m constraints, the third G1 MSM `short` points
                    shorter than the key; host memory to host memory
Scalars and elements are seeded draws from [0, r); bases are [k_i]G with seeded k_i, 0.1% of them
the point at infinity, resident in Montgomery form as a proving key is. Every output is an exact
integer: affine coordinates of the sum as a program reads them (the projective words behind them
depend on the order of the additions), or the transformed elements in their buffer.
"""
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "zk-gpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from zk_gpu import CosetShift, Gpu, Group, Msm, Ntt, xyzz_to_affine, xyzz_to_affine_g2  # noqa: E402
from zk_gpu.host import FR, inverse as mod_inverse  # noqa: E402
from zk_gpu.serving import ProofInputs, Server  # noqa: E402
from zk_gpu.synthetic import generator_multiples  # noqa: E402

COSET = 7  # the usual coset generator of the witness map
_gpu = None


def gpu():
    """The process's one context, as a program has it."""
    global _gpu
    if _gpu is None:
        _gpu = Gpu(0)
    return _gpu


def _msm(name, n, group=1, scalars="uniform", table=False):
    return {"name": name, "kind": "msm", "n": n, "group": group, "scalars": scalars, "table": table}


def listed():
    return [
        # the smallest circuits and the commitments of a handful of values: one call's latency
        _msm("g1 1000", 1000),
        # a small circuit's key, the size of the single-call configuration
        _msm("g1 2^16", 1 << 16),
        # a medium circuit: the witness is 30% zeros and 30% small values, and no power of two long
        _msm("g1 300007 sparse", 300007, scalars="sparse"),
        # the ordinary large circuit
        _msm("g1 2^20", 1 << 20),
        # the largest circuits: the quotient polynomial's MSM
        _msm("g1 2^24", 1 << 24),
        # the one G2 MSM of a proof, for a small and for an ordinary large circuit
        _msm("g2 2^14", 1 << 14, group=2),
        _msm("g2 2^20", 1 << 20, group=2),
        # a short transform (latency), an ordinary one back from evaluations, the largest circuits'
        {"name": "ntt 2^12", "kind": "ntt", "log_n": 12, "inverse": False, "count": 1},
        {"name": "intt 2^20", "kind": "ntt", "log_n": 20, "inverse": True, "count": 1},
        {"name": "ntt 2^24", "kind": "ntt", "log_n": 24, "inverse": False, "count": 1},
        # a proof's polynomial part: coset transforms, quotient, back to coefficients
        {"name": "witness 2^18", "kind": "witness", "log_n": 18, "coset": COSET},
        # a whole small proof through the server: three G1 MSMs, one G2 MSM and the chain above
        {"name": "proof 2^14", "kind": "proof", "log_m": 14, "short": 1024},
    ]


def draw(rng):
    kind = rng.choice(["g1", "g1", "g1", "g2", "ntt", "ntt", "witness", "proof"])
    if kind in ("g1", "g2"):
        top = 24.0 if kind == "g1" else 21.0
        n = min(int(2.0 ** rng.uniform(9.5, top)), 1 << int(top))
        # a table holds a row of the key per window: tables are for keys that stay small
        table = kind == "g1" and n <= (1 << 19) and rng.random() < 0.25
        return {"kind": "msm", "n": n, "group": 1 if kind == "g1" else 2,
                "scalars": rng.choice(["uniform", "uniform", "sparse", "r-1"]), "table": table}
    if kind == "ntt":
        log_n = rng.randint(10, 24)
        return {"kind": "ntt", "log_n": log_n, "inverse": rng.random() < 0.5,
                "count": rng.randint(1, 8 if log_n <= 21 else 4)}
    if kind == "witness":
        return {"kind": "witness", "log_n": rng.randint(11, 21), "coset": rng.randint(3, 9999)}
    return {"kind": "proof", "log_m": rng.randint(11, 17), "short": rng.randint(0, 1024)}


# ------------------------------------------------------------------ inputs

def _elements(n, gen):
    """n elements of Fr, (n, 8) little-endian 32-bit words on the GPU: uniform below the multiple of
    2^224 next below r."""
    w = torch.randint(-(1 << 31), 1 << 31, (n, 8), dtype=torch.int64, device="cuda", generator=gen).to(torch.int32)
    w[:, 7] = torch.randint(0, FR >> 224, (n,), dtype=torch.int64, device="cuda", generator=gen).to(torch.int32)
    return w


def _scalars(n, mix, gen):
    w = _elements(n, gen)
    if mix == "uniform":
        return w
    u = torch.rand(n, device="cuda", generator=gen)
    if mix == "sparse":  # 30% zero, 30% below 2^64
        w[u < 0.6, 2:] = 0
        w[u < 0.3] = 0
    else:  # 5% equal to r - 1
        minus_one = np.array([((FR - 1) >> (32 * i)) & 0xFFFFFFFF for i in range(8)], dtype=np.uint32).view(np.int32)
        w[u < 0.05] = torch.from_numpy(minus_one).cuda()
    return w


def _words(t):
    return t.cpu().numpy().view(np.uint32).reshape(-1)


def _bases(n, group, gen):
    k = _elements(n, gen)
    k[torch.rand(n, device="cuda", generator=gen) < 0.001] = 0
    return generator_multiples(gpu(), group, _words(k), mont256=True)


class _DeviceWords:
    """A library buffer's memory for torch.as_tensor (it copies nothing)."""

    def __init__(self, buf):
        self.buf = buf
        self.__cuda_array_interface__ = {"shape": (buf.words(),), "typestr": "<i4", "data": (buf.device_ptr(), False),
                                         "version": 3}


def _tensor(buf):
    return torch.as_tensor(_DeviceWords(buf), device="cuda")


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    g = gpu()
    s = {"case": case}
    if case["kind"] == "msm":
        n, group = case["n"], Group(case["group"])
        c = Msm.default_window(n)
        s["plan"] = Msm.for_group(g, group, n, c)
        s["bases"] = _bases(n, group, gen)
        s["scalars"] = g.buffer(_words(_scalars(n, case["scalars"], gen)))
        if case["table"]:
            s["bases"] = Msm.fixed_base_table(g, group, s["bases"], n, c)
            s["plan"].set_fixed_base()
    elif case["kind"] == "ntt":
        s["plan"] = Ntt(g, case["log_n"])
        s["data"] = [g.buffer(_words(_elements(1 << case["log_n"], gen))) for _ in range(case["count"])]
        s["out"] = [_tensor(b) for b in s["data"]]
    elif case["kind"] == "witness":
        n = 1 << case["log_n"]
        s["plan"] = Ntt(g, case["log_n"])
        s["shift"] = CosetShift(g, case["log_n"], case["coset"])
        s["unshift"] = CosetShift(g, case["log_n"], mod_inverse(case["coset"], FR))
        s["polys"] = [g.buffer(_words(_elements(n, gen))) for _ in range(3)]
        s["out"] = _tensor(s["polys"][2])
    else:
        m = 1 << case["log_m"]
        s["server"] = Server(g, lanes=8, coset_g=COSET)
        s["server"].add_key(m, _bases(m, Group.G1, gen), _bases(m, Group.G2, gen))
        s["server"].reserve(case["log_m"], 1)
        counts = [m, m, m - case["short"]]
        s["request"] = ProofInputs(case["log_m"], counts).fill(
            [_words(_elements(k, gen)) for k in counts], _words(_elements(m, gen)),
            [_words(_elements(2 * m, gen)) for _ in range(3)])
    g.wait()
    return s


# ------------------------------------------------------------------ passes

def _point(words, group):
    xy = xyzz_to_affine(words) if group == 1 else xyzz_to_affine_g2(words)
    if xy is None:
        return np.zeros(8 * group, dtype=np.int64)
    return np.array(xy, dtype=np.uint64).reshape(-1).view(np.int64)


def run(s):
    case, g = s["case"], gpu()
    if case["kind"] == "msm":
        out = s["plan"].run(g, s["bases"], s["scalars"])
        return _point(g.read(out, Group(case["group"]).xyzz_words()), case["group"])
    if case["kind"] == "ntt":
        transform = s["plan"].inverse if case["inverse"] else s["plan"].forward
        for data in s["data"]:
            transform(g, data)
        return s["out"]
    if case["kind"] == "witness":
        plan, (a, b, c) = s["plan"], s["polys"]
        for p in (a, b, c):
            plan.inverse_coset(g, p, s["shift"])
        plan.forward(g, a)
        plan.forward(g, b)
        plan.forward_quotient(g, c, a, b, case["coset"])
        plan.inverse_coset(g, c, s["unshift"])
        return s["out"]
    server, req = s["server"], s["request"]
    server.wait(server.submit(req))
    pts = req.points()
    return [_point(pts[32 * j: 32 * j + 32], 1) for j in range(3)] + [_point(pts[96:160], 2), req.h().view(np.int32)]


def exact(case, seed):
    """Every output is a whole number and has no rounding error to measure."""
    return None


# ------------------------------------------------------------------ work

PRODUCT = 2 * 2 * 64  # 32-bit multiplications and additions of a 256-bit modular product: operand and reduction half


def _msm_work(n, group):
    """One addition of a bucket method per point and 16-bit window of a 254-bit scalar, six products
    each (three times that in the quadratic extension); scalars and points read once."""
    return {"bytes": n * (32 + 64 * group), "flops": n * 16 * 6 * (3 if group == 2 else 1) * PRODUCT}


def _ntt_work(log_n, count=1):
    """The elements in and out once, half a product per element and stage."""
    n = 1 << log_n
    return {"bytes": count * 64 * n, "flops": count * n * log_n // 2 * PRODUCT}


def work(case):
    if case["kind"] == "msm":
        return _msm_work(case["n"], case["group"])
    if case["kind"] == "ntt":
        return _ntt_work(case["log_n"], case["count"])
    if case["kind"] == "witness":
        return _ntt_work(case["log_n"], 7)
    m = 1 << case["log_m"]
    parts = [_msm_work(m, 1), _msm_work(m, 1), _msm_work(m - case["short"], 1), _msm_work(m, 2), _ntt_work(case["log_m"] + 1, 7)]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
