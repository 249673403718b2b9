"""The work that users of this prover run on the GPU, as cases that can be timed.

A case names one call path of the public interface (the Python mirror of the C ABI)
and its sizes:

  ntt     one domain operation (FFT, iFFT, cosetFFT, icosetFFT) on a device vector
  msm     one multi-scalar multiplication over resident bases, scalars on the device
  prove   a witness in pinned host memory -> raw proof -> blinded proof
  batch   several proofs of a prepared key in one call, raw proofs out
  verify  a batch of proofs in host memory -> verdicts

Contexts, proving keys, verification keys and MSM bases are what a prover process
loads once and keeps; they are made once per circuit or size and do not depend on the
seed.  Witnesses, scalars, vectors, proof randomness and proofs come from the seed.
Every output is a vector of whole numbers (field elements in Montgomery limbs, affine
points in the libff Jacobian layout, verdicts).
"""
import functools
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nkr-zkp_b200"))
import nkr_b200 as nk  # noqa: E402

FR = 21888242871839275222246405745257275088548364400416034343698204186575808495617
FQ = 21888242871839275222246405745257275088696311157297823662689037894645226208583
FR_TOP = FR >> 192  # highest limb of the scalar field's modulus
G2_GEN = (10857046999023057135944570762232829481370756359578518086990519993285655852781,
          11559732032986387107991004021392285783925812861821192530917403151452391805634,
          8495653923123431417604973247489272438418190587263600148770280649306958101930,
          4082367875863433681332203403145435568316851327593401208105741076214120093531)
NTT_OPS = ("fft", "ifft", "coset_fft", "icoset_fft")


def listed():
    return [
        # a small domain: one call of a launch-bound transform
        {"name": "ntt_fft_2e10", "path": "ntt", "op": "fft", "logn": 10},
        # the domain of a 2^16-constraint circuit (matmul 32, sql-aggregate 64)
        {"name": "ntt_ifft_2e16", "path": "ntt", "op": "ifft", "logn": 16},
        # the domain of the large serving keys
        {"name": "ntt_icoset_2e22", "path": "ntt", "op": "icoset_fft", "logn": 22},
        # a few thousand bases, not a power of two: latency and short reductions
        {"name": "msm_g1_3001", "path": "msm", "group": 1, "n": 3001, "scalars": "uniform"},
        # a query of a mid-size circuit with the values of a sparse witness (zeros, ones,
        # 16-bit values, one in ten uniform)
        {"name": "msm_g1_200003_sparse", "path": "msm", "group": 1, "n": 200003, "scalars": "sparse"},
        # the quotient query of a 2^20-constraint circuit: uniform coefficients
        {"name": "msm_g1_2e20", "path": "msm", "group": 1, "n": 1 << 20, "scalars": "uniform"},
        # a G2 query, ragged
        {"name": "msm_g2_100001", "path": "msm", "group": 2, "n": 100001, "scalars": "uniform"},
        # the smallest circuit: 16 steps, a 2^4 domain
        {"name": "prove_fibonacci_16", "path": "prove", "circuit": "fibonacci", "param": 16, "density": 0},
        # dense random matrices: 2^16 domain, 3,072 public inputs, no repeated witness values
        {"name": "prove_matmul_32", "path": "prove", "circuit": "matmul", "param": 32, "density": 0},
        # the headline prove: 2^20 domain, sparse preimages, a witness that repeats values
        {"name": "prove_poseidon_2048", "path": "prove", "circuit": "poseidon", "param": 2048, "density": 2},
        # batched proving of a small circuit with half of its preimages set (2^15 domain)
        {"name": "batch_poseidon_64_x8", "path": "batch", "circuit": "poseidon", "param": 64, "density": 1,
         "count": 8},
        # a verifier's queue of proofs with four public inputs; one in eight is not valid
        {"name": "verify_sql_16_x4096", "path": "verify", "circuit": "sql-aggregate", "param": 16, "density": 0,
         "count": 4096},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _draw_circuit(rng, most):
    """A circuit of at most about 2^most constraints."""
    kind = rng.choice(("fibonacci", "matmul", "poseidon", "sql-aggregate"))
    if kind == "fibonacci":
        return {"circuit": kind, "param": _log_uniform(rng, 8, (1 << most) - 1), "density": 0}
    if kind == "matmul":
        return {"circuit": kind, "param": _log_uniform(rng, 2, int((1 << most) ** (1 / 3))),
                "density": rng.randrange(3)}
    if kind == "poseidon":
        return {"circuit": kind, "param": _log_uniform(rng, 1, (1 << most) // 440), "density": rng.randrange(3)}
    return {"circuit": kind, "param": 1 << rng.randrange(1, most - 9), "density": rng.randrange(3)}


def draw(rng):
    path = rng.choice(("ntt", "msm", "msm", "prove", "prove", "batch", "verify"))
    if path == "ntt":
        return {"path": path, "op": rng.choice(NTT_OPS), "logn": rng.randrange(4, 23)}
    if path == "msm":
        group = rng.choice((1, 1, 2))
        return {"path": path, "group": group, "n": _log_uniform(rng, 64, 1 << 20 if group == 1 else 1 << 17),
                "scalars": rng.choice(("uniform", "uniform", "sparse"))}
    if path == "prove":
        return {"path": path, **_draw_circuit(rng, 18)}
    if path == "batch":
        return {"path": path, **_draw_circuit(rng, 14), "count": rng.randrange(2, 13)}
    return {"path": path, "circuit": "sql-aggregate", "param": 1 << rng.randrange(1, 5),
            "density": rng.randrange(3), "count": _log_uniform(rng, 16, 8192)}


# ---------------------------------------------------------------------------
# what a process keeps
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _ctx():
    return nk.Context(0)


def _limbs(v):
    return np.frombuffer(int(v).to_bytes(32, "little"), np.uint64).copy()


def _ints(a):
    return [int.from_bytes(row.tobytes(), "little") for row in np.ascontiguousarray(a).reshape(-1, 4)]


@functools.lru_cache(maxsize=2)
def _key(circuit, param, density):
    """A prepared proving key, its public input count and the pieces of its verification
    key (setup on the GPU from fixed toxic waste)."""
    r1 = nk.generate(circuit, param, density, seed=1)
    rng = random.Random(77)
    pk, vk = nk.setup(_ctx(), r1, [_limbs(rng.randrange(1, FR)) for _ in range(5)])
    be = nk.Backend(_ctx())
    be.prepare(r1, pk)
    be._keep = None  # the device holds the key: a server drops the host copy
    return be, r1.public_inputs, vk


@functools.lru_cache(maxsize=2)
def _verifying_key(circuit, param, density):
    vk = _key(circuit, param, density)[2]
    return nk.VerifyingKey(_ctx(), vk["alpha_g1_beta_g2"], vk["gamma_g2"], vk["delta_g2"], vk["ic"])


def _generator(group):
    coords = (1, 2, 1) if group == 1 else G2_GEN + (1, 0)
    return np.concatenate([_limbs(v * (1 << 256) % FQ) for v in coords])


def _base_scalars(n):
    return _uniform_fr(n, torch.Generator("cuda").manual_seed(5)).cpu().numpy().view(np.uint64)


@functools.lru_cache(maxsize=2)
def _bases(group, n):
    """Resident bases k_i G with fixed uniform k_i."""
    gen = _generator(group)
    jac = _ctx().group_op(group, 2, np.tile(gen, (n, 1)), _base_scalars(n))
    return nk.MsmBases(_ctx(), group, jac)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _uniform_fr(n, gen):
    """n uniform field elements (limbs below the modulus) on the GPU."""
    a = torch.randint(-2**63, 2**63 - 1, (n, 4), dtype=torch.int64, device="cuda", generator=gen)
    a[:, 3] = torch.randint(0, FR_TOP, (n,), dtype=torch.int64, device="cuda", generator=gen)
    return a


@functools.lru_cache(maxsize=1)
def _small_values():
    """The Montgomery forms of 0 .. 2^16 - 1 on the GPU."""
    one = (1 << 256) % FR
    tab = np.stack([_limbs(v * one % FR) for v in range(1 << 16)])
    return torch.from_numpy(tab.view(np.int64)).cuda()


def _scalars(n, kind, gen):
    if kind == "uniform":
        return _uniform_fr(n, gen)
    # a sparse witness: 30% zero, 60% zero, one or a 16-bit value, 10% uniform, shuffled
    n_uni, n_zero = n // 10, (3 * n) // 10
    rest = n - n_uni - n_zero
    which = torch.randint(0, 3, (rest,), device="cuda", generator=gen)
    small = torch.randint(0, 1 << 16, (rest,), device="cuda", generator=gen)
    small = torch.where(which == 2, small, which)
    out = torch.zeros((n, 4), dtype=torch.int64, device="cuda")
    out[:n_uni] = _uniform_fr(n_uni, gen)
    out[n_uni + n_zero:] = _small_values()[small]
    return out[torch.randperm(n, device="cuda", generator=gen)].contiguous()


def _witness(case, seed):
    return nk.generate(case["circuit"], case["param"], case["density"], seed=2 + seed).witness


def _pinned(a):
    t = torch.empty(a.size, dtype=torch.int64, pin_memory=True)
    t.numpy()[:] = np.ascontiguousarray(a).reshape(-1).view(np.int64)
    return t


def _random_fr(rng):
    return _limbs(rng.randrange(1, FR))


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(1000 + seed)
    if case["path"] == "ntt":
        x = _uniform_fr(1 << case["logn"], gen)
        state = {"op": NTT_OPS.index(case["op"]), "x": x, "work": torch.empty_like(x), "y": torch.empty_like(x)}
    elif case["path"] == "msm":
        state = {"bases": _bases(case["group"], case["n"]), "scalars": _scalars(case["n"], case["scalars"], gen)}
    elif case["path"] == "prove":
        be = _key(case["circuit"], case["param"], case["density"])[0]
        rng = random.Random(seed)
        state = {"key": be, "witness": _pinned(_witness(case, seed)), "r": _random_fr(rng), "s": _random_fr(rng)}
    elif case["path"] == "batch":
        be = _key(case["circuit"], case["param"], case["density"])[0]
        state = {"keys": [be] * case["count"],
                 "witnesses": [_pinned(_witness(case, 64 * seed + i)) for i in range(case["count"])]}
    else:
        be, n_pub, _ = _key(case["circuit"], case["param"], case["density"])
        w = _witness(case, seed)
        raw = be.prove(w)
        rng, count = random.Random(seed), case["count"]
        # distinct blindings of one proof, repeated to the queue's length
        some = [np.frombuffer(bytes(be.blind(raw, _random_fr(rng), _random_fr(rng))), np.uint64)
                for _ in range(min(count, 256))]
        proofs = np.stack([some[i % len(some)] for i in range(count)])
        publics = np.ascontiguousarray(np.broadcast_to(w[1:1 + n_pub], (count, n_pub, 4)))
        # one in eight comes with another public input
        bad = np.array([rng.random() < 0.125 for _ in range(count)])
        publics[bad, 0] = _random_fr(rng)
        state = {"vk": _verifying_key(case["circuit"], case["param"], case["density"]), "proofs": proofs,
                 "publics": publics}
    state["path"] = case["path"]
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def _raw_array(raw):
    return np.frombuffer(bytes(raw), np.uint64).view(np.int64)


def run(state):
    if state["path"] == "ntt":
        # the transform uses up its input vector
        state["work"].copy_(state["x"])
        stream = torch.cuda.current_stream().cuda_stream
        _ctx().ntt_device(state["op"], state["work"].data_ptr(), state["y"].data_ptr(), state["x"].shape[0],
                          stream or None)
        return state["y"]
    if state["path"] == "msm":
        point, _ = state["bases"].run(None, scalars_ptr=state["scalars"].data_ptr())
        return point.view(np.int64)
    if state["path"] == "prove":
        raw = state["key"].prove(None, witness_ptr=state["witness"].data_ptr())
        proof = state["key"].blind(raw, state["r"], state["s"])
        return {"raw": _raw_array(raw), "proof": _raw_array(proof)}
    if state["path"] == "batch":
        raws = nk.prove_batch(state["keys"], witness_ptrs=[w.data_ptr() for w in state["witnesses"]])
        return np.stack([_raw_array(r) for r in raws])
    return state["vk"].verify_batch(state["publics"], state["proofs"])


# ---------------------------------------------------------------------------
# work and values
# ---------------------------------------------------------------------------

PRODUCT = 2 * 2 * 64  # multiply-adds of one Montgomery product in 32-bit words, two operations each


@functools.lru_cache(maxsize=None)
def _circuit_sizes(circuit, param, density):
    r1 = nk.generate(circuit, param, density, seed=1)
    return r1.rows, r1.cols, sum(x.size for x in r1.col_idx)


def work(case):
    """Bytes: inputs and resident tables read once, outputs written once.  flops: 32-bit
    multiplies and adds of the field products: n/2 log2 n for a transform, 16 digits of a
    point and scalar at 6 products each for an MSM (3 times that on G2)."""
    if case["path"] == "ntt":
        n = 1 << case["logn"]
        return {"bytes": 64 * n, "flops": PRODUCT * (n // 2 * case["logn"] + n)}
    if case["path"] == "msm":
        n = case["n"]
        return {"bytes": (32 + 64 * case["group"]) * n, "flops": PRODUCT * 16 * 6 * n * (1 if case["group"] == 1 else 3)}
    if case["path"] == "verify":
        # Miller loop and final exponentiation: about 20,000 field products a proof
        return {"bytes": (384 + 4 * 32) * case["count"], "flops": PRODUCT * 20000 * case["count"]}
    rows, cols, nnz = _circuit_sizes(case["circuit"], case["param"], case["density"])
    count = case.get("count", 1)
    logn = rows.bit_length() - 1
    points = 3 * cols + rows + 3 * cols  # three G1 queries, h, and the G2 query at three products
    return {"bytes": count * (32 * cols + 64 * (3 * cols + rows) + 128 * cols + 36 * nnz),
            "flops": count * PRODUCT * (7 * (rows // 2 * logn + rows) + 16 * 6 * points + nnz)}


def _fft(x, w):
    """Radix-2 transform of Python integers, natural order in and out."""
    n = len(x)
    if n == 1:
        return x
    even, odd, out, t = _fft(x[0::2], w * w % FR), _fft(x[1::2], w * w % FR), [0] * n, 1
    for i in range(n // 2):
        v = t * odd[i] % FR
        out[i], out[i + n // 2] = (even[i] + v) % FR, (even[i] - v) % FR
        t = t * w % FR
    return out


def _mul2(a, b):
    return ((a[0] * b[0] - a[1] * b[1]) % FQ, (a[0] * b[1] + a[1] * b[0]) % FQ)


def _inv2(a):
    d = pow(a[0] * a[0] + a[1] * a[1], -1, FQ)
    return (a[0] * d % FQ, -a[1] * d % FQ)


def _add(p, q):
    """Affine addition over Fq2 (Fq as its first coordinate); None is infinity."""
    if p is None or q is None:
        return q if p is None else p
    (x1, y1), (x2, y2) = p, q
    if x1 == x2:
        if y1 != y2:
            return None
        xx = _mul2(x1, x1)
        lam = _mul2((3 * xx[0], 3 * xx[1]), _inv2((2 * y1[0] % FQ, 2 * y1[1] % FQ)))
    else:
        lam = _mul2((y2[0] - y1[0], y2[1] - y1[1]), _inv2(((x2[0] - x1[0]) % FQ, (x2[1] - x1[1]) % FQ)))
    ll = _mul2(lam, lam)
    x3 = ((ll[0] - x1[0] - x2[0]) % FQ, (ll[1] - x1[1] - x2[1]) % FQ)
    d = _mul2(lam, (x1[0] - x3[0], x1[1] - x3[1]))
    return x3, ((d[0] - y1[0]) % FQ, (d[1] - y1[1]) % FQ)


def _point_exact(group, k):
    g = ((1, 0), (2, 0)) if group == 1 else (G2_GEN[:2], G2_GEN[2:])
    acc = None
    for bit in bin(k)[2:]:
        acc = _add(acc, acc)
        if bit == "1":
            acc = _add(acc, g)
    x, y, z = ((0, 0), (1, 0), (0, 0)) if acc is None else (acc[0], acc[1], (1, 0))
    take = 1 if group == 1 else 2
    return np.concatenate([_limbs(v * (1 << 256) % FQ) for c in (x, y, z) for v in c[:take]]).view(np.int64)


def exact(case, seed):
    """The same outputs from Python integers: transforms up to 2^16, every MSM
    ((sum of s_i k_i) G for the bases k_i G), verdicts as the queue was made."""
    if case["path"] == "ntt" and case["logn"] <= 16:
        n, op = 1 << case["logn"], case["op"]
        x = _ints(prepare(case, seed)["x"].cpu().numpy())
        w = pow(5, (FR - 1) >> 28 << (28 - case["logn"]), FR)
        if op == "coset_fft":
            x = [v * pow(5, i, FR) % FR for i, v in enumerate(x)]
        y = _fft(x, w if op in ("fft", "coset_fft") else pow(w, -1, FR))
        if op in ("ifft", "icoset_fft"):
            g = pow(5, -1, FR) if op == "icoset_fft" else 1
            ninv = pow(n, -1, FR)
            y = [v * ninv * pow(g, i, FR) % FR for i, v in enumerate(y)]
        return torch.from_numpy(np.stack([_limbs(v) for v in y]).view(np.int64))
    if case["path"] == "msm":
        gen = torch.Generator("cuda").manual_seed(1000 + seed)
        s = _ints(_scalars(case["n"], case["scalars"], gen).cpu().numpy())
        k = _ints(_base_scalars(case["n"]))
        total = sum(a * b for a, b in zip(s, k)) * pow(1 << 512, -1, FR) % FR  # both in Montgomery form
        return _point_exact(case["group"], total)
    return None
