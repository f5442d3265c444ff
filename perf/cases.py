"""The multiplications a program has this library do, as measurable cases.

Every case goes through the public Python API (flint_b200) on the values such
a program holds: device-resident limb arrays for the integer, polynomial and
ring products, host arrays for the drop-in call that replaces FLINT's
mpn_ctx_mpn_mul.  Sizes are in 64-bit limbs or coefficients.

  listed()            the standing cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) inputs and handles, on the GPU (host arrays for "host")
  run(state)          one pass; returns the whole products
  work(case)          bytes in and out, and integer operations, of one pass
  exact(case, seed)   the products from Python's own integers, or None where
                      those would take too long
"""
import math

import numpy as np
import torch

import flint_b200 as fb

MASK64 = (1 << 64) - 1
# operands above this many limbs in all take Python's integers too long
EXACT_LIMBS = 60000


def listed():
    return [
        # A short product of uneven operands: the low end of the transform
        # route, one call at a time (latency and launches).
        {"name": "mpn_1k", "kind": "mpn", "an": 1000, "bn": 700},
        # 2^16 x 2^16 limbs, 4 Mbit operands: the usual size of a step in a
        # large-constant or factorial computation.
        {"name": "mpn_64k", "kind": "mpn", "an": 65536, "bn": 65536},
        # A ragged product between powers of two.
        {"name": "mpn_700k", "kind": "mpn", "an": 700001, "bn": 650003},
        # The largest balanced product a single transform takes (1 Gbit each).
        {"name": "mpn_16m", "kind": "mpn", "an": 1 << 24, "bn": 1 << 24},
        # A long operand times a much shorter one.
        {"name": "mpn_16m_by_1m", "kind": "mpn", "an": 1 << 24, "bn": 1 << 20},
        # A squaring (a powering ladder), ragged.
        {"name": "mpn_sqr_2m", "kind": "sqr", "an": 2000003},
        # The drop-in call on host arrays, as FLINT's callers make it.
        {"name": "mpn_host_200k", "kind": "host", "an": 200001, "bn": 150007},
        # Middle product of two polynomials mod a word-size n (Newton
        # iteration's step), window of the middle half.
        {"name": "nmod_mid_1m", "kind": "nmod", "an": 1 << 20, "bn": 1 << 20, "zl": 1 << 19, "zh": 3 << 19,
         "n": (1 << 61) + 15},
        # Integer polynomials with 2000-bit signed coefficients.
        {"name": "fmpz_10k", "kind": "fmpz", "an": 10007, "bn": 9001, "w": 32},
        # A planned batch of uneven products, replayed on new operand values.
        {"name": "batch_256", "kind": "batch", "count": 256, "lo": 10.0, "hi": 17.0, "ratio": 4.0, "sizes": 5},
        # The pointwise stage of a Schoenhage-Strassen convolution.
        {"name": "ring_47104", "kind": "ring", "N": 47104, "count": 4096},
        # One operand's transform kept and multiplied by a new one.
        {"name": "op_300k", "kind": "op", "an": 300007, "bn": 200003},
    ]


def _log_int(rng, lo, hi):
    return max(1, int(round(2.0 ** rng.uniform(math.log2(lo), math.log2(hi)))))


def draw(rng):
    kind = rng.choice(["mpn", "mpn", "mpn", "mpn", "sqr", "host", "nmod", "fmpz", "batch", "ring", "op"])
    if kind in ("mpn", "op"):
        an = _log_int(rng, 600, 1 << 24 if kind == "mpn" else 1 << 21)
        bn = max(1, int(an / 2.0 ** rng.uniform(0.0, 4.0)))
        if rng.random() < 0.5:
            an, bn = bn, an
        return {"kind": kind, "an": an, "bn": bn}
    if kind == "sqr":
        return {"kind": kind, "an": _log_int(rng, 600, 1 << 23)}
    if kind == "host":
        an = _log_int(rng, 600, 1 << 20)
        return {"kind": kind, "an": an, "bn": max(1, int(an / 2.0 ** rng.uniform(0.0, 3.0)))}
    if kind == "nmod":
        an = _log_int(rng, 500, 1 << 21)
        bn = max(1, int(an / 2.0 ** rng.uniform(0.0, 3.0)))
        zn = an + bn - 1
        if rng.random() < 0.5:
            zl, zh = 0, zn
        else:
            zl = min(an, bn) - 1
            zh = max(an, bn)
        n = rng.getrandbits(rng.choice([20, 31, 50, 62, 64])) | 3
        return {"kind": kind, "an": an, "bn": bn, "zl": zl, "zh": zh, "n": n}
    if kind == "fmpz":
        w = rng.randint(1, 65)
        total = _log_int(rng, 1 << 13, 1 << 22)     # chunk positions of the product
        an = max(2, int(total / (2 * w) * rng.uniform(0.3, 0.7)))
        bn = max(2, int(total / (2 * w)) - an)
        return {"kind": kind, "an": an, "bn": bn, "w": w}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(32, 300), "lo": 10.0, "hi": rng.uniform(13.0, 17.0),
                "ratio": rng.uniform(0.0, 4.0), "sizes": rng.randint(1, 1 << 20)}
    # ring products: N = m b with m = 1024 digits or 4096 digits of odd size
    m = rng.choice([256, 1024, 4096])
    N = m * rng.randint(20, 60)
    return {"kind": "ring", "N": N, "count": _log_int(rng, 8, min(8192, (1 << 28) // N))}


# --- inputs ---------------------------------------------------------------

def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed & ((1 << 62) - 1))
    return g


def _limbs(g, n, device="cuda"):
    """n uniform 64-bit limbs as int64, the top one non-zero."""
    x = torch.randint(-(1 << 63), (1 << 63) - 1, (n,), dtype=torch.int64, generator=g, device=device)
    x[-1] |= 1
    return x


def _below(g, count, n):
    """`count` values in [0, n) as int64 bit patterns."""
    if n < (1 << 62):
        return torch.randint(0, n, (count,), dtype=torch.int64, generator=g, device="cuda")
    x = torch.randint(0, (1 << 63) - 1, (count,), dtype=torch.int64, generator=g, device="cuda")
    return x % n if n < (1 << 63) else x


def _batch_sizes(case):
    rng = np.random.default_rng(case["sizes"])
    U = rng.uniform(case["lo"], case["hi"], case["count"])
    V = rng.uniform(0.0, case["ratio"], case["count"])
    an = np.rint(np.exp2(U)).astype(np.int64)
    bn = np.maximum(1, np.rint(an / np.exp2(V))).astype(np.int64)
    return [(int(a), int(b)) for a, b in zip(an, bn)]


def _inputs(case, seed):
    k = case["kind"]
    if k == "host":
        g = _gen(seed, "cpu")
        return tuple(_limbs(g, n, "cpu").numpy().view(np.uint64) for n in (case["an"], case["bn"]))
    g = _gen(seed)
    if k in ("mpn", "op"):
        return _limbs(g, case["an"]), _limbs(g, case["bn"])
    if k == "sqr":
        return (_limbs(g, case["an"]),)
    if k == "nmod":
        return _below(g, case["an"], case["n"]), _below(g, case["bn"], case["n"])
    if k == "fmpz":
        # signed coefficients of up to 64 w - 1 bits
        return tuple(_limbs(g, n * case["w"]).view(n, case["w"]) for n in (case["an"], case["bn"]))
    if k == "batch":
        return tuple(_limbs(g, sum(s)) for s in zip(*_batch_sizes(case)))
    if k == "ring":
        n = case["N"] // 64
        out = []
        for _ in range(2):
            x = _limbs(g, case["count"] * (n + 1)).view(case["count"], n + 1)
            x[:, n] = 0
            out.append(x)
        return tuple(out)
    raise ValueError(k)


def prepare(case, seed):
    ins = _inputs(case, seed)
    k = case["kind"]
    ctx = fb.MpnCtx()
    st = {"kind": k, "case": case, "ctx": ctx, "in": ins}

    def empty(*shape):
        return torch.empty(shape, dtype=torch.int64, device="cuda")

    if k in ("mpn", "op"):
        st["z"] = empty(case["an"] + case["bn"])
    elif k == "sqr":
        st["z"] = empty(2 * case["an"])
    elif k == "host":
        st["z"] = np.empty(case["an"] + case["bn"], dtype=np.uint64)
    elif k == "nmod":
        st["z"] = empty(case["zh"] - case["zl"])
    elif k == "fmpz":
        st["zw"] = 2 * case["w"] + 1
        st["z"] = empty(case["an"] + case["bn"] - 1, st["zw"])
    elif k == "batch":
        sizes = _batch_sizes(case)
        st["z"] = empty(sum(a + b for a, b in sizes))
        reqs, oa, ob, oz = [], 0, 0, 0
        for an, bn in sizes:
            reqs.append((st["z"].data_ptr() + 8 * oz, ins[0].data_ptr() + 8 * oa, an,
                         ins[1].data_ptr() + 8 * ob, bn))
            oa, ob, oz = oa + an, ob + bn, oz + an + bn
        st["batch"] = fb.MpnBatch(ctx, reqs)
        st["batch"].ctx = ctx       # the context outlives its batch
    elif k == "ring":
        st["ring"] = fb.Mulmod2expp1(ctx, case["N"])
        st["z"] = empty(case["count"], case["N"] // 64 + 1)
    if k == "op":
        plan = fb.FftPlan.mpn(ctx, case["an"], case["bn"])
        st["plan"] = plan
        st["B"], st["A"] = plan.op(), plan.op()
        st["B"].fft(ins[1].data_ptr(), case["bn"], torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    return st


def run(st):
    k, c, ctx, ins, z = st["kind"], st["case"], st["ctx"], st["in"], st["z"]
    if k == "host":
        return ctx.mpn_mul(ins[0], ins[1], out=z)
    s = torch.cuda.current_stream().cuda_stream
    if k == "mpn":
        ctx.mpn_mul_device(z.data_ptr(), ins[0].data_ptr(), c["an"], ins[1].data_ptr(), c["bn"], s)
    elif k == "sqr":
        ctx.mpn_mul_device(z.data_ptr(), ins[0].data_ptr(), c["an"], ins[0].data_ptr(), c["an"], s)
    elif k == "nmod":
        ctx.nmod_poly_mul_mid_device(z.data_ptr(), c["zl"], c["zh"], ins[0].data_ptr(), c["an"],
                                     ins[1].data_ptr(), c["bn"], c["n"], s)
    elif k == "fmpz":
        ctx.fmpz_poly_mul_device(z.data_ptr(), st["zw"], 0, c["an"] + c["bn"] - 1, ins[0].data_ptr(), c["w"],
                                 c["an"], ins[1].data_ptr(), c["w"], c["bn"], s)
    elif k == "batch":
        st["batch"].run(s)
    elif k == "ring":
        st["ring"].batch_device(z.data_ptr(), ins[0].data_ptr(), ins[1].data_ptr(), c["count"], None, s)
    else:
        plan, A = st["plan"], st["A"]
        A.fft(ins[0].data_ptr(), c["an"], s)
        plan.pointwise(fb.OP_MUL, A, A, st["B"], s)
        A.ifft(s)
        A.export_mpn(z.data_ptr(), c["an"] + c["bn"], s)
    return z


# --- what a pass cannot do without -----------------------------------------

def _product_ops(length, words=5, transforms=3):
    """Integer operations of a product of `length` coefficients by fast
    transforms: (length / 2) log2(length) butterflies (one multiplication, two
    additions) per transform and 32-bit residue word of a coefficient."""
    return 3.0 * transforms * words * 0.5 * length * math.log2(max(2, length))


def work(case):
    k = case["kind"]
    if k in ("mpn", "host", "op"):
        n = case["an"] + case["bn"]
        # the kept operand of "op" was transformed before the pass
        inb = 8 * n if k != "op" else 8 * case["an"] + 20 * n
        return {"bytes": inb + 8 * n, "flops": _product_ops(n, transforms=2 if k == "op" else 3)}
    if k == "sqr":
        return {"bytes": 24 * case["an"], "flops": _product_ops(2 * case["an"], transforms=2)}
    if k == "nmod":
        n = case["an"] + case["bn"]
        words = math.ceil((2 * case["n"].bit_length() + math.log2(n)) / 31)
        return {"bytes": 8 * (n + case["zh"] - case["zl"]), "flops": _product_ops(n, words)}
    if k == "fmpz":
        n = case["an"] + case["bn"] - 1
        zw = 2 * case["w"] + 1
        return {"bytes": 8 * (case["w"] * (case["an"] + case["bn"]) + zw * n),
                "flops": _product_ops(n * (2 * case["w"] - 1))}
    if k == "batch":
        sizes = _batch_sizes(case)
        return {"bytes": sum(16 * (a + b) for a, b in sizes), "flops": sum(_product_ops(a + b) for a, b in sizes)}
    n = case["N"] // 64 + 1
    return {"bytes": 24 * n * case["count"], "flops": case["count"] * _product_ops(2 * n)}


# --- exact results from Python's integers -----------------------------------

def _to_int(x):
    """A 1-D limb array as a Python integer."""
    if isinstance(x, torch.Tensor):
        x = x.cpu().numpy()
    return int.from_bytes(np.ascontiguousarray(x).tobytes(), "little")


def _from_int(v, n):
    return np.frombuffer((v & ((1 << (64 * n)) - 1)).to_bytes(8 * n, "little"), dtype=np.int64).copy()


def _unpack(v, slot, count):
    """count slots of `slot` bytes of a non-negative integer."""
    b = v.to_bytes(slot * count, "little")
    return [int.from_bytes(b[slot * i:slot * (i + 1)], "little") for i in range(count)]


def exact(case, seed):
    k = case["kind"]
    if k in ("mpn", "host", "op", "sqr"):
        an = case["an"]
        bn = case.get("bn", an)
        if an + bn > EXACT_LIMBS:
            return None
        ins = _inputs(case, seed)
        a, b = _to_int(ins[0]), _to_int(ins[-1])
        z = _from_int(a * b, an + bn)
        return z.view(np.uint64) if k == "host" else torch.from_numpy(z)
    if k == "nmod":
        an, bn, n = case["an"], case["bn"], case["n"]
        if 3 * (an + bn) > EXACT_LIMBS:
            return None
        slot = (2 * n.bit_length() + max(an, bn).bit_length()) // 8 + 1
        vals = []
        for x in _inputs(case, seed):
            c = [int(v) for v in x.cpu().numpy().view(np.uint64)]
            vals.append(int.from_bytes(b"".join(v.to_bytes(slot, "little") for v in c), "little"))
        out = [v % n for v in _unpack(vals[0] * vals[1], slot, an + bn - 1)]
        z = np.array(out[case["zl"]:case["zh"]], dtype=np.uint64)
        return torch.from_numpy(z.view(np.int64))
    if k == "fmpz":
        an, bn, w = case["an"], case["bn"], case["w"]
        if 2 * w * (an + bn) > EXACT_LIMBS:
            return None
        zw = 2 * w + 1
        slot = 8 * zw
        vals = []
        for x in _inputs(case, seed):
            # sum of signed coefficients c_i 2^(8 slot i)
            pos, neg = [], []
            for r in x.cpu().numpy():
                v = int.from_bytes(r.tobytes(), "little", signed=True)
                pos.append(max(v, 0).to_bytes(slot, "little"))
                neg.append(max(-v, 0).to_bytes(slot, "little"))
            vals.append(int.from_bytes(b"".join(pos), "little") - int.from_bytes(b"".join(neg), "little"))
        zn = an + bn - 1
        half = 1 << (8 * slot - 1)
        # a bias of half a slot everywhere makes every slot non-negative
        bias = half * (((1 << (8 * slot * zn)) - 1) // ((1 << (8 * slot)) - 1))
        out = [v - half for v in _unpack(vals[0] * vals[1] + bias, slot, zn)]
        z = np.concatenate([_from_int(v, zw) for v in out]).reshape(zn, zw)
        return torch.from_numpy(z)
    if k == "batch":
        sizes = _batch_sizes(case)
        if sum(a + b for a, b in sizes) > 16 * EXACT_LIMBS or max(a + b for a, b in sizes) > EXACT_LIMBS:
            return None
        A, B = (x.cpu().numpy() for x in _inputs(case, seed))
        out, oa, ob = [], 0, 0
        for an, bn in sizes:
            out.append(_from_int(_to_int(A[oa:oa + an]) * _to_int(B[ob:ob + bn]), an + bn))
            oa, ob = oa + an, ob + bn
        return torch.from_numpy(np.concatenate(out))
    N, count = case["N"], case["count"]
    n = N // 64
    if (n + 1) * count > 64 * EXACT_LIMBS:
        return None
    X, Y = (x.cpu().numpy() for x in _inputs(case, seed))
    mod = (1 << N) + 1
    rows = []
    for x, y in zip(X, Y):
        v = _to_int(x) * _to_int(y)
        v = (v & ((1 << N) - 1)) - (v >> N)
        rows.append(_from_int(v % mod, n + 1))
    return torch.from_numpy(np.stack(rows))
