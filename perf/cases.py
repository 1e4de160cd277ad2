"""Performance cases of the triples library, each one pass through its public entry points.

What a user of the library has it do:
  * a reference-style program calls the drop-in body once per (i, j, k) triple on host arrays, in the
    reference driver's k loop (omp/test.c:160-176), in double or (the gpu-omp variant) single precision;
  * a program with its own device buffers runs one triple without any allocation;
  * a batched program keeps a plan and its tensors on the device and runs every triple of a system, of
    several systems or of several virtual indices a, in the fused, plain or emulated form, and reads
    the totals (and, where it prints or checkpoints them, the per-triple records);
  * a program whose tensors live on the host uploads them overlapped with the kernels.

The inputs follow the library's own synthetic distributions (T2 in [-0.05, 0.05], T1-like amplitudes in
[-0.02, 0.02], integrals in [-0.1, 0.1] or log-uniform magnitudes in [1e-6, 1], occupied energies in
[-2, -0.5], virtual ones in [0.2, 3], a = the first virtual orbital).
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

# imported with the repository's root as the working folder
_PKG = os.path.join(os.getcwd(), "nwchem-ccsd-trpdrv_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import trpdrv_b200 as T  # noqa: E402

MODES = {"fused": T.MODE_FUSED, "plain": T.MODE_PLAIN, "emulated": T.MODE_EMULATED}
VECS = ("dintc", "dintx", "t1v")


# ------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------
def _body(name, nocc, nvir, kind="body", ncor=0, calls=8):
    return {"name": name, "kind": kind, "ncor": ncor, "nocc": nocc, "nvir": nvir, "calls": calls}


def _plan(name, sizes, mode="fused", ncor=0, nkpass=1, a_count=1, slices=7, dist="uniform", records=True, host=False):
    return {"name": name, "kind": "plan", "mode": mode, "sizes": " ".join("%dx%d" % s for s in sizes), "ncor": ncor,
            "nkpass": nkpass, "a_count": a_count, "slices": slices, "dist": dist, "records": records, "host": host}


def listed():
    return [
        # the reference driver's k loop at the size of its known answers (test_c99 10 60): latency of a call
        _body("dropin_10_60", 10, 60, calls=10),
        # the same loop at a production size, one k chunk of 8 calls
        _body("dropin_40_300", 40, 300),
        # the single-precision variant's driver (gpu-omp/test.c) at its known-answer size
        _body("dropin_fp32_10_60", 10, 60, kind="body32", calls=10),
        # one triple on an application's own device buffers, no allocation
        _body("noalloc_20_200", 20, 200, kind="noalloc", calls=1),
        # the reference's structure on the device, triple by triple, with per-triple records
        _plan("plain_20_200", [(20, 200)], mode="plain"),
        # the smallest system a program runs whole; totals only
        _plan("fused_10_60", [(10, 60)], records=False),
        # tensors in pinned host memory, copied under the kernels; totals only
        _plan("host_20_200", [(20, 200)], records=False, host=True),
        # odd sizes with core orbitals and a chunked k loop, as basis sets give them
        _plan("fused_odd_13_151", [(13, 151)], ncor=5, nkpass=2),
        # uneven molecules in one launch
        _plan("batch_uneven", [(8, 80), (12, 150), (16, 220), (24, 310)], records=False),
        # the headline size: every triple of one a
        _plan("fused_40_300", [(40, 300)]),
        # emulated form, a sweep over two virtual indices
        _plan("emulated_sweep_20_200", [(20, 200)], mode="emulated", a_count=2),
        # emulated form on the precision workload (log-uniform integrals); totals only
        _plan("emulated_30_400", [(30, 400)], mode="emulated", dist="loguniform", records=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["body", "body", "body32", "noalloc", "plain", "fused", "fused", "batch", "host", "emulated",
                       "emulated"])
    ncor = rng.choice([0, 0, rng.randint(1, 12)])
    if kind in ("body", "body32"):
        nocc, nvir = _log(rng, 4, 40), _log(rng, 24, 320)
        c = _body("", nocc, nvir, kind=kind, ncor=ncor, calls=rng.randint(1, min(10, nocc)))
    elif kind == "noalloc":
        c = _body("", _log(rng, 2, 64), _log(rng, 16, 256), kind=kind, ncor=ncor, calls=1)
    else:
        dist = rng.choice(["uniform", "uniform", "loguniform"])
        records = rng.random() < 0.5
        a_count = rng.choice([1, 1, 2, 3])
        if kind == "batch":
            sizes = [(_log(rng, 4, 20), _log(rng, 24, 260)) for _ in range(rng.randint(2, 10))]
            c = _plan("", sizes, ncor=ncor, dist=dist, records=records)
        elif kind == "plain":
            c = _plan("", [(_log(rng, 4, 18), _log(rng, 24, 200))], mode="plain", ncor=ncor, dist=dist, records=records)
        elif kind == "host":
            c = _plan("", [(_log(rng, 4, 24), _log(rng, 24, 320))], ncor=ncor, dist=dist, records=records, host=True)
        elif kind == "fused":
            c = _plan("", [(_log(rng, 4, 28), _log(rng, 24, 320))], ncor=ncor, nkpass=rng.choice([1, 1, 2, 4]),
                      a_count=a_count, dist=dist, records=records)
        else:
            c = _plan("", [(_log(rng, 4, 24), _log(rng, 24, 400))], mode="emulated", ncor=ncor, a_count=a_count,
                      slices=rng.choice([7, 7, 7, 5, 6, 8]), dist=dist, records=records)
    del c["name"]
    return c


def _sizes(case):
    return [tuple(int(v) for v in s.split("x")) for s in case["sizes"].split()]


def _flops(o, v, same):
    """One triple's contractions; where i == k the eight t products are the eight n products."""
    return 16.0 * v * v * (v + o) * (0.5 if same else 1.0)


def work(case):
    if case["kind"] != "plan":
        o, v, n = case["nocc"], case["nvir"], case["calls"]
        w = 4 if case["kind"] == "body32" else 8
        flops = sum(_flops(o, v, case["kind"] != "noalloc" and q == o - 1) for q in range(o - n, o))
        # the i blocks once, the k blocks of every call
        return {"bytes": w * ((1 + n) * (3.0 * v * v + 4.0 * o * v + 3.0 * v) + case["ncor"] + o + v + 2 * n), "flops": flops}
    na, by, fl = case["a_count"], 0.0, 0.0
    for o, v in _sizes(case):
        nt = o * o * (o + 1) // 2
        by += 8.0 * (o * o * v * v + 2 * o * o * o * v + 2 * o * o * v + na * (2 * o * v * v + 3 * o * v)
                     + case["ncor"] + o + v + 2 + (4 * nt * na if case["records"] else 0))
        fl += na * ((nt - o * o) * _flops(o, v, False) + o * o * _flops(o, v, True))
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _uniform(g, n, lo, hi):
    return torch.empty(n, dtype=torch.float64, device="cuda").uniform_(lo, hi, generator=g)


def _integrals(g, n, dist):
    if dist == "uniform":
        return _uniform(g, n, -0.1, 0.1)
    sign = torch.randint(0, 2, (n,), device="cuda", generator=g).to(torch.float64).mul_(2.0).sub_(1.0)
    return _uniform(g, n, math.log(1e-6), 0.0).exp_().mul_(sign)


def _tensors(ncor, o, v, a_count, dist, seed, jblocks=None):
    """The tensors of one system in the library's slice layout, on the GPU (jblocks: that many j blocks)."""
    g = torch.Generator(device="cuda").manual_seed(1_000_003 * seed + 1009 * o + v)
    nj = o if jblocks is None else jblocks
    eorb = torch.cat([_uniform(g, ncor, -20.0, -5.0).sort()[0], _uniform(g, o, -2.0, -0.5).sort()[0],
                      _uniform(g, v, 0.2, 3.0).sort()[0]])
    t = {"eorb": eorb, "t2": _uniform(g, nj * o * v * v, -0.05, 0.05)}
    for n in ("jvv", "kvv"):
        t[n] = _integrals(g, a_count * o * v * v, dist)
    for n in ("tov", "xov"):
        t[n] = _uniform(g, o * v * o, -0.02, 0.02)
    for n in ("jov", "kov"):
        t[n] = _integrals(g, nj * o * o * v, dist)
    for n in ("dintc", "dintx"):
        t[n] = _integrals(g, a_count * o * v, dist)
    t["t1v"] = _uniform(g, a_count * o * v, -0.02, 0.02)
    return t


def _case_tensors(case, seed):
    if case["kind"] == "plan":
        return [_tensors(case["ncor"], o, v, case["a_count"], case["dist"], seed + 7919 * q)
                for q, (o, v) in enumerate(_sizes(case))]
    return [_tensors(case["ncor"], case["nocc"], case["nvir"], 1, "uniform", seed, jblocks=1)]


def _triples(o, nkpass=1):
    """(i, j, k) of every triple, 0-based, in the order of the library's records."""
    return T.enumerate_triples(o, nkpass)[:, :3].astype(np.int64) - 1


def _body_triples(case):
    """The calls of a body case: i = nocc, j = 1, the last `calls` values of k (one k chunk); 0-based."""
    o, n = case["nocc"], case["calls"]
    if case["kind"] == "noalloc":
        return [(o - 1, 0, max(0, o - 2))]
    return [(o - 1, 0, k) for k in range(o - n, o)]


# ------------------------------------------------------------------------------------------------
# prepare and run
# ------------------------------------------------------------------------------------------------
_fp32 = None


def _body_fn(kind):
    """The reference-signature body: double from the main library, float from the single-precision one."""
    global _fp32
    if kind == "body":
        return T.lib.ccsd_trpdrv_omp_cbody_
    if _fp32 is None:
        lib = C.CDLL(os.path.join(os.path.dirname(T.LIB_PATH), "libtrpdrv_b200_fp32.so"))
        _fp32 = lib.ccsd_trpdrv_omp_cbody_
        fp, ip = C.POINTER(C.c_float), C.POINTER(C.c_int)
        _fp32.restype = None
        _fp32.argtypes = [fp] * 9 + [ip] * 3 + [fp] * 2 + [ip] * 5 + [fp] * 20
    return _fp32


def _prepare_body(case, seed):
    o, v, ncor = case["nocc"], case["nvir"], case["ncor"]
    single = case["kind"] == "body32"
    dt, ct = (np.float32, C.c_float) if single else (np.float64, C.c_double)
    h = {n: np.ascontiguousarray(x.cpu().numpy().astype(dt)) for n, x in _case_tensors(case, seed)[0].items()}
    f = np.zeros((8, v * v), dtype=dt)
    trip = _body_triples(case)
    emp = np.zeros((len(trip), 2), dtype=dt)
    klo = trip[0][2] + 1
    pt = C.POINTER(ct)

    def at(name, off):
        return C.cast(h[name].ctypes.data + off * h[name].itemsize, pt)

    ints = [C.c_int(q) for q in (ncor, o, v)]
    vv, ov = v * v, o * v
    calls = []
    for q, (i, j, k) in enumerate(trip):
        idx = [C.c_int(x) for x in (ncor + o + 1, i + 1, j + 1, k + 1, klo)]
        kl = klo - 1
        args = [C.cast(f[x].ctypes.data, pt) for x in range(8)] + [at("eorb", 0)] + [C.byref(x) for x in ints]
        args += [C.cast(emp[q, x:].ctypes.data, pt) for x in range(2)] + [C.byref(x) for x in idx]
        args += [at("t2", i * vv), at("t2", kl * vv), at("tov", i * ov), at("tov", kl * ov), at("xov", i * ov),
                 at("xov", kl * ov), at("jvv", i * vv), at("jvv", kl * vv), at("kvv", i * vv), at("kvv", kl * vv),
                 at("jov", i * ov), at("jov", kl * ov), at("kov", i * ov), at("kov", kl * ov)]
        args += [at(n, i * v) for n in VECS] + [at(n, k * v) for n in VECS]
        calls.append((args, idx))
    return {"kind": "body", "fn": _body_fn(case["kind"]), "calls": calls, "emp": emp, "keep": (h, f, ints)}


def _prepare_noalloc(case, seed):
    o, v = case["nocc"], case["nvir"]
    t = _case_tensors(case, seed)[0]
    i, j, k = _body_triples(case)[0]
    vv, ov = v * v, o * v
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    s = {}
    for role, x in (("i", i), ("k", k)):
        s["t%sj" % role] = t["t2"][x * vv:]
        for n, src, size in (("t%sa", "tov", ov), ("x%sa", "xov", ov), ("j%sa", "jvv", vv), ("k%sa", "kvv", vv),
                             ("j%sj", "jov", ov), ("k%sj", "kov", ov)):
            s[n % role] = t[src][x * size:]
        for n in VECS:
            s[n + ("1" if role == "i" else "2")] = t[n][x * v:]
    # each slice in a buffer of its own, as an application holds it
    sizes = {n: vv for n in ("tij", "tkj", "jia", "jka", "kia", "kka")}
    keep = {n: x[:sizes.get(n, v if n[-1] in "12" else ov)].clone() for n, x in s.items()}
    keep["eorb"] = t["eorb"]
    args = T.BodyDeviceArgs()
    args.ncor, args.nocc, args.nvir, args.a = case["ncor"], o, v, case["ncor"] + o + 1
    args.i, args.j, args.k = i + 1, j + 1, k + 1
    for n in T.BODY_DEVICE_FIELDS:
        setattr(args, n, C.c_void_p((out if n == "out4" else keep[n]).data_ptr()))
    return {"kind": "noalloc", "args": args, "out": out, "keep": keep}


def prepare(case, seed):
    if case["kind"] in ("body", "body32"):
        return _prepare_body(case, seed)
    if case["kind"] == "noalloc":
        return _prepare_noalloc(case, seed)
    ten = _case_tensors(case, seed)
    systems = []
    for (o, v), t in zip(_sizes(case), ten):
        s = T.System(case["ncor"], o, v, case["ncor"] + o + 1, a_count=case["a_count"])
        if case["host"]:
            s.arrays = {}
            for n, x in t.items():
                p = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
                p.copy_(x)
                s.arrays[n] = p.numpy()
        systems.append(s)
    opt = {"mode": MODES[case["mode"]], "nkpass": case["nkpass"]}
    if case["mode"] == "emulated":
        opt["slices"] = case["slices"]
    plan = T.Plan(systems, **opt)
    torch.cuda.synchronize()
    if not case["host"]:
        plan.bind_device([{n: x.data_ptr() for n, x in t.items()} for t in ten])
    return {"kind": "plan", "plan": plan, "host": case["host"], "records": case["records"], "n": len(systems),
            "keep": None if case["host"] else ten}


def run(state):
    if state["kind"] == "body":
        fn, emp = state["fn"], state["emp"]
        emp.fill(0.0)  # each call's emp4 and emp5 by itself
        for args, _ in state["calls"]:
            fn(*args)
        return {"emp4": emp[:, 0].copy(), "emp5": emp[:, 1].copy()}
    if state["kind"] == "noalloc":
        rc = T.lib.trpdrv_body_device_noalloc(C.byref(state["args"]), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise RuntimeError(T.last_error()[1])
        return {"out4": state["out"]}
    plan = state["plan"]
    if state["host"]:
        plan.upload_execute()
    else:
        plan.execute()
    e4, e5 = plan.energies()
    got = {"emp4": e4, "emp5": e5}
    if state["records"]:
        got["records"] = [plan.triple_energies(q) for q in range(state["n"])]
    return got


# ------------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ------------------------------------------------------------------------------------------------
def _records(t, ncor, o, v, ai, tri, nj):
    """emp4i, emp5i, emp4k, emp5k of the triples `tri` (n, 3), of virtual index block ai."""
    dev = t["t2"].device
    t2 = t["t2"].view(nj, o, v, v)
    jov, kov = (t[n].view(nj, o, v, o) for n in ("jov", "kov"))
    jvv, kvv = (t[n].view(-1, o, v, v)[ai] for n in ("jvv", "kvv"))
    tov, xov = (t[n].view(o, o, v) for n in ("tov", "xov"))
    dintc, dintx, t1v = (t[n].view(-1, o, v)[ai] for n in VECS)
    e = t["eorb"]
    ev = e[ncor + o:]
    out = torch.empty(len(tri), 4, dtype=torch.float64, device=dev)
    step = max(1, int(3e7 / (v * v * 8)))
    tri = torch.from_numpy(np.ascontiguousarray(tri)).to(dev)
    for s in range(0, len(tri), step):
        i, j, k = tri[s:s + step].T

        def group(x, y):
            # f[c, b] of f1..f4 with A operands of index x and B operands of (j, y)
            tt, kk, jj = t2[j, y], kov[j, y], jov[j, y]
            return [torch.matmul(tt.transpose(1, 2), jvv[x]) - torch.matmul(kk, tov[x]),
                    torch.matmul(tt.transpose(1, 2), kvv[x]) - torch.matmul(kk, xov[x]),
                    torch.matmul(tt, jvv[x]) - torch.matmul(jj, tov[x]),
                    torch.matmul(tt, kvv[x]) - torch.matmul(jj, xov[x])]

        n, m = group(i, k), group(k, i)
        nt, mt = [f.transpose(1, 2) for f in n], [f.transpose(1, 2) for f in m]
        ea = e[ncor + o + ai] - (e[ncor + i] + e[ncor + j] + e[ncor + k])
        den = -1.0 / (ev[None, None, :] + ev[None, :, None] + ea[:, None, None])

        def energies(n, nt, m, mt, x):
            # the i energies; the k energies are the same forms with the n and t families exchanged
            e4 = den * ((m[0] + nt[0] + mt[1] + n[2] + nt[3]) * (m[0] - 2 * m[1] - 2 * m[2] + m[3])
                        - (n[0] + mt[0] + nt[1] + nt[2]) * (2 * m[0] - m[1] - m[2] + 2 * m[3])
                        + 3 * (n[0] * (n[0] + nt[2] + 2 * mt[3]) + n[1] * mt[1] + n[2] * m[3]))
            e5 = den * t1v[x][:, None, :] * (
                dintx[x][:, :, None] * (m[0] + n[1] + nt[3] - 2 * (m[2] + n[3] + nt[1] + n[0] + m[1] + nt[2])
                                        + 4 * (n[2] + m[3] + nt[0]))
                + dintc[x][:, :, None] * (n[0] + n[3] + mt[0] - 2 * (n[1] + n[2] + mt[1])))
            return e4.sum((1, 2)), e5.sum((1, 2))

        out[s:s + step, 0], out[s:s + step, 1] = energies(n, nt, m, mt, i)
        out[s:s + step, 2], out[s:s + step, 3] = energies(m, mt, n, nt, k)
    return out


def exact(case, seed):
    ten = _case_tensors(case, seed)
    if case["kind"] != "plan":
        t = ten[0]
        if case["kind"] == "body32":
            t = {n: x.float().double() for n, x in t.items()}
        tri = np.array(_body_triples(case))
        r = _records(t, case["ncor"], case["nocc"], case["nvir"], 0, tri, 1).cpu().numpy()
        if case["kind"] == "noalloc":
            return {"out4": r[0]}
        both = (tri[:, 0] != tri[:, 2])[:, None]
        tot = r[:, :2] + np.where(both, r[:, 2:], 0.0)
        return {"emp4": tot[:, 0], "emp5": tot[:, 1]}
    e4, e5, recs = [], [], []
    for (o, v), t in zip(_sizes(case), ten):
        tri = _triples(o, case["nkpass"])
        r = np.concatenate([_records(t, case["ncor"], o, v, ai, tri, o).cpu().numpy() for ai in range(case["a_count"])])
        both = np.tile((tri[:, 0] != tri[:, 2])[:, None], (case["a_count"], 1))
        tot = r[:, :2] + np.where(both, r[:, 2:], 0.0)
        e4.append(math.fsum(tot[:, 0]))
        e5.append(math.fsum(tot[:, 1]))
        recs.append(r)
    got = {"emp4": np.array(e4), "emp5": np.array(e5)}
    if case["records"]:
        got["records"] = recs
    return got
