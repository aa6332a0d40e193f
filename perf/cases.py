"""Timed cases of the prover: what a user's program has this package do.

Kinds, each through a public entry point:

* proof   update proofs of resident sessions (DynaverseEngine.submit / wait)
* msm     one MSM: host buffers, device buffers, or fresh scalars over a
          registered SRS with its window table; G1 and G2
* sparse  a sparse-index MSM over a registered SRS (an update's delta)
* ntt     one Fr transform on device buffers, any of the four kinds
* setup   SRS generation: G1 and checked G2 fixed-base points, host buffers
* batch   one replay of a batch plan of uneven MSMs and transforms

All values are uniform field elements, as in every real input of the path
(witnesses, blinded polynomials, deltas of fresh values).  Results are exact
integers modulo a prime, given as bytes.
"""
import functools
import importlib
import random

import numpy as np
import torch

dv = importlib.import_module("zkp-dynaverse_b200")

FQ_MUL, FQ_SQR = 136, 108  # 32x32-bit multiply-accumulates of one product and one square


def listed():
    return [
        # one user, one small session: the smallest whole call, all latency
        {"name": "proof_n256_one", "kind": "proof", "n": 256, "sessions": 1, "gates": 4},
        # one update of a large session, called and waited for by itself
        {"name": "proof_n65536_one", "kind": "proof", "n": 65536, "sessions": 1, "gates": 100},
        # a server's queue: updates of 1 to 1024 gates, the largest re-anchor
        {"name": "proof_n65536_x32", "kind": "proof", "n": 65536, "sessions": 32, "gates": 1024},
        # a small commitment through the operator interface (host buffers)
        {"name": "msm_g1_host_1000", "kind": "msm", "points": 1000, "g2": False, "form": "host"},
        # a full commitment with both inputs on the device
        {"name": "msm_g1_device_2p20", "kind": "msm", "points": 1 << 20, "g2": False, "form": "device"},
        # commitments against a kept SRS, of a length that is no power of two
        {"name": "msm_g1_resident_300001", "kind": "msm", "points": 300001, "g2": False, "form": "resident"},
        # the verifier-side group
        {"name": "msm_g2_device_2p16", "kind": "msm", "points": 1 << 16, "g2": True, "form": "device"},
        # the delta of a middling update against a kept SRS
        {"name": "sparse_256", "kind": "sparse", "bases": 65536, "entries": 256},
        # a small transform: latency
        {"name": "ntt_forward_2p12", "kind": "ntt", "log": 12, "transform": 0},
        # a large one with the coset scaling, the quotient's way back
        {"name": "ntt_coset_inverse_2p22", "kind": "ntt", "log": 22, "transform": 3},
        # SRS generation with validation, host buffers in and out
        {"name": "setup_100000", "kind": "setup", "g1": 100000, "g2": 10000},
        # uneven commitments and transforms of one proving step as one plan
        {"name": "batch_128", "kind": "batch", "msms": 128, "top": 16, "ntts": 64, "ntt_top": 18, "shape": 4004},
    ]


def draw(rng):
    def size(lo, hi):  # log-uniform, odd sizes among them
        return max(lo, min(hi, int(lo * (hi / lo) ** rng.random())))

    kind = rng.choice(["proof", "proof", "msm", "msm", "msm", "sparse", "ntt", "ntt", "setup", "batch"])
    if kind == "proof":
        n = rng.choice([256, 1024, 4096, 16384, 65536])
        return {"kind": kind, "n": n, "sessions": size(1, 32), "gates": size(1, min(n, 1024))}
    if kind == "msm":
        g2 = rng.random() < 0.25
        form = rng.choice(["host", "device"] if g2 else ["host", "device", "resident"])
        return {"kind": kind, "points": size(200, 1 << 16 if g2 else 1 << 20), "g2": g2, "form": form}
    if kind == "sparse":
        return {"kind": kind, "bases": 65536, "entries": size(1, 4096)}
    if kind == "ntt":
        return {"kind": kind, "log": rng.randint(8, 22), "transform": rng.randrange(4)}
    if kind == "setup":
        return {"kind": kind, "g1": size(100, 100000), "g2": size(10, 10000)}
    return {"kind": kind, "msms": size(8, 128), "top": rng.randint(11, 16), "ntts": size(4, 64),
            "ntt_top": rng.randint(12, 18), "shape": rng.randrange(1 << 20)}


# ---------------------------------------------------- what a program keeps
@functools.lru_cache(maxsize=None)
def _backend():
    return dv.DvgpuBackend()


@functools.lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()


@functools.lru_cache(maxsize=None)
def _engine():
    return dv.DynaverseEngine(120 << 30, 64)


@functools.lru_cache(maxsize=None)
def _params(n):
    rng, m = random.Random(9900 + n), 8 * n
    while True:  # the setup's own conditions on the two trapdoors
        x, y = rng.randrange(1, dv.R_MODULUS), rng.randrange(1, dv.R_MODULUS)
        if (x != y and pow(x, m, dv.R_MODULUS) != 1 and pow(y, m, dv.R_MODULUS) != 1
                and x != pow(y, 8, dv.R_MODULUS)):
            return _engine().params_create(n, x, y)


@functools.lru_cache(maxsize=None)
def _srs(n, c):
    """A registered G1 SRS of n bases with its window table (c = 0: the
    library's width)."""
    b = _backend()
    h = b.register_bases(_bases(n, False, 2812).cpu().numpy().tobytes())
    b.precompute_bases(h, c)
    return h


@functools.lru_cache(maxsize=None)
def _plan(msms, top, ntts, ntt_top, shape):
    """A batch plan over a kept SRS: MSMs of 2^U points, U uniform in
    [8, top], and transforms of 2^floor(U) elements, U uniform in
    [10, ntt_top]."""
    b = _backend()
    rng = np.random.default_rng(shape)
    sizes = [min(1 << top, int(2 ** u)) for u in rng.uniform(8, top, msms)]
    logs = [int(u) for u in rng.uniform(10, ntt_top, ntts)]
    h = b.register_bases(_bases(1 << top, False, 2812).cpu().numpy().tobytes())
    plan, _ = b.batch_plan_create(h, sizes, logs)
    return plan, b.batch_plan_buffers(plan), sum(sizes), sum(1 << x for x in logs)


class _DeviceBytes:
    def __init__(self, ptr, nbytes):
        self.__cuda_array_interface__ = {"shape": (nbytes,), "typestr": "|u1", "data": (ptr, False), "version": 3}


def _view(ptr, nbytes):
    return torch.as_tensor(_DeviceBytes(ptr, nbytes), device="cuda")


def _fr(seed, n):
    out = torch.empty(32 * n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    _backend().random_fr_device(seed, n, out.data_ptr(), _stream().cuda_stream)
    torch.cuda.synchronize()
    return out


def _bases(n, g2, seed):
    """[tau^i] of the generator, affine."""
    b, s = _backend(), _stream().cuda_stream
    tau, powers = _fr(seed, 1), torch.empty(32 * n, dtype=torch.uint8, device="cuda")
    out = torch.empty((128 if g2 else 64) * n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    b.fr_powers_device(tau.data_ptr(), n, powers.data_ptr(), s)
    b.fixed_base_device(powers.data_ptr(), n, g2, out.data_ptr(), s)
    torch.cuda.synchronize()
    return out


class _Sessions:
    """Open sessions on one valid instance, and two update sets that passes
    take in turn, so that every pass changes values."""

    def __init__(self, case, seed):
        n, r = case["n"], dv.R_MODULUS
        rng = random.Random(seed)
        left, right, mul = ([rng.randrange(r) for _ in range(n)] for _ in range(3))
        total = [(x + y) % r for x, y in zip(left, right)]
        prod = [x * y % r for x, y in zip(total, mul)]
        enc = [b"".join(v.to_bytes(32, "little") for v in col) for col in (left, right, total, mul, prod)]
        witness = enc[0] + enc[1] + enc[2] + enc[2] + enc[3] + enc[4]
        self.engine, self.turn = _engine(), 0
        params = _params(n)
        self.ids = [self.engine.open_session(params, enc[0], witness)[0] for _ in range(case["sessions"])]
        self.updates = []
        supports = []
        for k in range(case["sessions"]):
            # one session: the case's own support; several: log-uniform up to
            # it, half of them inside a window of 64 gates
            g = case["gates"]
            if case["sessions"] > 1:
                g = min(n, max(1, int(g ** ((k + 0.5) / case["sessions"]))))
            if k % 2 and g <= 64 < n:
                at = rng.randrange(n - 64)
                supports.append([at + i for i in rng.sample(range(64), g)])
            else:
                supports.append(rng.sample(range(n), g))
        for _ in range(2):
            one = []
            for gates in supports:
                idx, vals = [], []
                for i in gates:
                    u = rng.randrange(r)
                    idx += [4 * n + i, 5 * n + i]
                    vals += [u.to_bytes(32, "little"), (total[i] * u % r).to_bytes(32, "little")]
                one.append((idx, b"".join(vals)))
            self.updates.append(one)

    def step(self):
        ups = self.updates[self.turn]
        self.turn ^= 1
        tickets = [self.engine.submit(s, idx, vals) for s, (idx, vals) in zip(self.ids, ups)]
        return b"".join(self.engine.wait(t)[0] for t in tickets)

    def __del__(self):
        for s in getattr(self, "ids", []):
            self.engine.close_session(s)


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "proof":
        st["sessions"] = _Sessions(case, seed)
    elif kind == "msm":
        n, g2 = case["points"], case["g2"]
        scalars = _fr(3 * seed + 1, n)
        if case["form"] == "resident":
            st["handle"] = _srs(n, 0)
        else:
            points = _bases(n, g2, 3 * seed + 2)
            st["points"] = points.cpu().numpy().tobytes() if case["form"] == "host" else points
        st["scalars"] = scalars.cpu().numpy().tobytes() if case["form"] == "host" else scalars
    elif kind == "sparse":
        st["handle"] = _srs(case["bases"], 8)
        rng = np.random.default_rng(seed)
        st["index"] = rng.choice(case["bases"], size=case["entries"], replace=False).astype(np.uint64)
        st["values"] = _fr(3 * seed + 1, case["entries"]).cpu().numpy().tobytes()
    elif kind == "ntt":
        st["values"] = _fr(3 * seed + 1, 1 << case["log"])
        st["out"] = torch.empty_like(st["values"])
    elif kind == "setup":
        st["g1"] = _fr(3 * seed + 1, case["g1"]).cpu().numpy().tobytes()
        st["g2"] = _fr(3 * seed + 2, case["g2"]).cpu().numpy().tobytes()
        _backend()
    else:
        plan, buf, points, elements = _plan(case["msms"], case["top"], case["ntts"], case["ntt_top"], case["shape"])
        st["plan"] = plan
        st["scalars"], st["values"] = _fr(3 * seed + 1, points), _fr(3 * seed + 2, elements)
        st["plan_scalars"] = _view(buf.scalars, buf.scalar_bytes)
        st["plan_values"] = _view(buf.ntt_values, buf.ntt_bytes)
        st["plan_sums"] = _view(buf.msm_results, buf.msm_result_bytes)
        st["plan_out"] = _view(buf.ntt_results, buf.ntt_bytes)
    return st


def _array(data):
    return np.frombuffer(data, dtype=np.uint8)


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "proof":
        return _array(state["sessions"].step())
    b, s = _backend(), _stream().cuda_stream
    if kind == "msm":
        if case["form"] == "host":
            call = b.msm_g2_host if case["g2"] else b.msm
            return _array(call(state["points"], state["scalars"]))
        if case["form"] == "device":
            return _array(b.msm_device(state["points"].data_ptr(), state["scalars"].data_ptr(), case["points"],
                                       g2=case["g2"], stream=s))
        return _array(b.msm_resident(state["handle"], state["scalars"].data_ptr(), case["points"], stream=s))
    if kind == "sparse":
        return _array(b.sparse_msm_resident(state["handle"], state["index"], state["values"],
                                            [0, case["entries"]])[0])
    if kind == "ntt":
        b.ntt_device(state["values"].data_ptr(), 1 << case["log"], case["transform"], state["out"].data_ptr(), s)
        return state["out"]
    if kind == "setup":
        g2, report = b.fixed_base_g2_checked(state["g2"], 3)
        return {"g1": _array(b.fixed_base_g1(state["g1"])), "g2": _array(g2),
                "invalid": int(report.invalid_points)}
    # the plan's buffers are shared by every caller of the plan
    with torch.cuda.stream(_stream()):
        state["plan_scalars"].copy_(state["scalars"])
        state["plan_values"].copy_(state["values"])
        b.batch_plan_launch(state["plan"], s)
        return state["plan_sums"].clone(), state["plan_out"].clone()


# ------------------------------------------------------------------- work
def _msm_macs(n, g2=False, windows=None):
    scale = 2.95 if g2 else 1.0  # G2 products are three, squares two
    madd, add = (8 * FQ_MUL + 2 * FQ_SQR) * scale, (12 * FQ_MUL + 2 * FQ_SQR) * scale
    return min(-(-254 // c) * (n * madd + (1 << c) * add) for c in range(2, 23))


def work(case):
    kind = case["kind"]
    if kind == "proof":
        # three dense quotients, their transforms, and 50 pairing equations
        n, k = case["n"], case["sessions"]
        macs = k * (3 * _msm_macs(n) + 6 * n * max(1, n.bit_length() - 1) * FQ_MUL / 2 + 50 * 12000 * FQ_MUL)
        return {"bytes": k * (3 * n * 32 + 9304), "flops": 2 * macs}
    if kind == "msm":
        n, g2 = case["points"], case["g2"]
        size = 32 + (0 if case["form"] == "resident" else 128 if g2 else 64)
        return {"bytes": n * size + (128 if g2 else 64), "flops": 2 * _msm_macs(n, g2)}
    if kind == "sparse":
        return {"bytes": case["entries"] * (40 + 64) + 64, "flops": 2 * _msm_macs(case["entries"])}
    if kind == "ntt":
        n = 1 << case["log"]
        products = n // 2 * case["log"] + (0, n, n, 2 * n)[case["transform"]]
        return {"bytes": 64 * n, "flops": 2 * products * FQ_MUL}
    if kind == "setup":
        # 16 mixed additions and a shared inversion a point; the subgroup check
        g1 = case["g1"] * (16 * (8 * FQ_MUL + 2 * FQ_SQR) + 10 * FQ_MUL)
        g2 = case["g2"] * (2.95 * 16 * (8 * FQ_MUL + 2 * FQ_SQR) + 30 * FQ_MUL + 2733 * FQ_MUL)
        return {"bytes": case["g1"] * 96 + case["g2"] * 160, "flops": 2 * (g1 + g2)}
    rng = np.random.default_rng(case["shape"])
    sizes = [min(1 << case["top"], int(2 ** u)) for u in rng.uniform(8, case["top"], case["msms"])]
    logs = [int(u) for u in rng.uniform(10, case["ntt_top"], case["ntts"])]
    macs = sum(_msm_macs(n) for n in sizes) + sum((1 << x) // 2 * x for x in logs) * FQ_MUL
    return {"bytes": 32 * sum(sizes) + 64 * len(sizes) + sum(64 << x for x in logs), "flops": 2 * macs}


def exact(case, seed):
    """No output is a rounded number: results are residues and curve points
    as bytes, and have to be equal."""
    return None
