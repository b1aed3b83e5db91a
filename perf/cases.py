"""What a user of this package has it do, as timed cases.

Every case goes through the package's public entry points on inputs that are
filled on the GPU from a seed.  All outputs are exact residues or bytes, so two
correct implementations agree on every bit.

Kinds (``case["kind"]``):

* ``commit``  -- one Ajtai commitment call of a batch of witnesses under a
  resident key (``GoldilocksAjtaiKey.commit`` or ``U32AjtaiKey.commit``):
  int8 / uint8 digits or residues, device tensors or, with ``host``, numpy
  arrays through the synchronous host call.
* ``packed``  -- a polynomial commitment of field elements: 22-bit packing of
  Goldilocks values into Q_32 ring elements and the commitment of the result.
* ``derive``  -- a verifier's recommitment: the key from its 32-byte seed, then
  one commitment under it.
* ``ntt``     -- batched negacyclic transforms, forward or inverse, over one u32
  modulus, the 4-prime CRT set or Goldilocks.
* ``batch``   -- a batch of uneven commitment jobs (``CommitBatch``).
* ``fold``    -- one folding step (``FoldPipeline``): byte digits of the witness,
  their commitments, and the CRT transforms of the witness.
* ``ring50``  -- products in Z_q[X]/(X^n + 1) for the 2^50 prime.
* ``labinius`` -- the binary-witness commitment over X^648 - X^324 + 1.
"""
import numpy as np
import torch

from lzx_b200 import (CRT_SET_30BIT, AjtaiParams, AjtaiPublicKey, GoldilocksAjtaiKey, GoldilocksNttTables, Modulus32,
                      NttTables, RingConfig, synth)
from lzx_b200.batch import CommitBatch, CommitJob, U32AjtaiKey
from lzx_b200.labinius import CommitmentKey, Modulus
from lzx_b200.packing import pack_field_elements
from lzx_b200.pipeline import FoldPipeline
from lzx_b200.ring50 import Q_50, RingConfig50

LIMBS = [Modulus.Q3889_FS_S, Modulus.Q2917_Q_S, Modulus.Q9721_FS_S]


def listed():
    return [
        # One small commitment (kappa = 8, 256 ring elements of int8 digits), the prover's smallest call: latency.
        dict(name="commit_one", kind="commit", ring="gl", log_d=6, kappa=8, m=256, batch=1, digits="i8", host=False),
        # 128 witnesses of 2^16 ring elements under one large key: the batched prover at its full size.
        dict(name="commit_128_witnesses", kind="commit", ring="gl", log_d=6, kappa=16, m=1 << 16, batch=128,
             digits="i8", host=False),
        # Witnesses that are already residues (no digits), an odd length and batch, degree 128.
        dict(name="commit_residues_odd", kind="commit", ring="gl", log_d=7, kappa=6, m=3001, batch=20,
             digits="residues", host=False),
        # The Q_32 commitment of the ring and commitment API's own benchmark (n = 256, k = 2, m = 16), whose callers
        # hold their ring elements in host memory.
        dict(name="commit_q32_host", kind="commit", ring="q32", log_d=8, kappa=2, m=16, batch=1, digits="residues",
             host=True),
        # A polynomial commitment's packed witness under a Q_32 key of two rows, several columns at once.
        dict(name="packed_commit_q32", kind="packed", log_d=6, kappa=2, m=7998, batch=16),
        # A verifier: the key again from its seed (k = 2, m = 2000, d = 64), and one commitment to compare.
        dict(name="derive_and_commit", kind="derive", log_d=6, kappa=2, m=2000),
        # The transform benchmark's forward half: 2^16 polynomials of degree 256 under each of the 4 CRT primes.
        dict(name="ntt_crt_forward", kind="ntt", ring="crt", log_n=8, count=1 << 16, inverse=False),
        # Back from evaluations over Goldilocks at a larger degree, and a count that fills no tile.
        dict(name="ntt_gl_inverse_odd", kind="ntt", ring="gl", log_n=10, count=30011, inverse=True),
        # Uneven commitment jobs in one run: degrees 64/128/256, lengths log-uniform, Goldilocks and CRT classes.
        dict(name="uneven_batch", kind="batch", jobs=128, log_max=16),
        # One folding step over a witness of 2^20 ring elements.
        dict(name="folding_step", kind="fold", m=1 << 20, kappa=16),
        # Ring products modulo the 2^50 prime.
        dict(name="ring50_products", kind="ring50", log_n=7, count=1 << 20),
        # The binary-witness commitment at its medium suite size: 2^18 field elements in 128 columns, two limbs.
        dict(name="labinius_commit", kind="labinius", columns=128, len_f162=2048, limbs=2),
    ]


def _log(rng, lo, hi):
    """An integer whose logarithm is uniform in [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["commit", "commit", "commit", "packed", "derive", "ntt", "ntt", "batch", "fold", "ring50", "labinius"])
    if kind == "commit":
        ring = rng.choice(["gl", "gl", "q32", "crt30"])
        log_d, kappa, batch = rng.choice([6, 6, 7, 8]), rng.randint(1, 16), _log(rng, 1, 128)
        top = min(1 << 16, (1 << 29) // (batch << log_d))
        m = _log(rng, 16, top)
        digits = rng.choice(["i8", "i8", "u8", "residues"])
        host = m * batch << log_d <= 1 << 20 and rng.random() < 0.5
        return dict(kind=kind, ring=ring, log_d=log_d, kappa=kappa, m=m, batch=batch, digits=digits, host=host)
    if kind == "packed":
        batch = _log(rng, 1, 64)
        return dict(kind=kind, log_d=rng.choice([6, 8]), kappa=rng.randint(1, 4), m=3 * _log(rng, 33, 4000), batch=batch)
    if kind == "derive":
        return dict(kind=kind, log_d=6, kappa=rng.randint(1, 4), m=_log(rng, 100, 8000))
    if kind == "ntt":
        ring, log_n = rng.choice(["q32", "crt", "gl", "gl"]), rng.randint(6, 10)
        if ring == "crt":
            log_n = min(log_n, 8)
        top = (1 << 26) >> (log_n + (2 if ring == "crt" else 0))
        return dict(kind=kind, ring=ring, log_n=log_n, count=_log(rng, 1, top), inverse=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, jobs=_log(rng, 12, 128), log_max=rng.choice([12, 13, 14, 15, 16]))
    if kind == "fold":
        return dict(kind=kind, m=_log(rng, 1 << 13, 1 << 20), kappa=rng.choice([4, 8, 12, 16]))
    if kind == "ring50":
        log_n = rng.randint(4, 7)
        return dict(kind=kind, log_n=log_n, count=_log(rng, 1, (1 << 27) >> log_n))
    return dict(kind=kind, columns=1 << rng.randint(1, 7), len_f162=4 * _log(rng, 8, 512), limbs=rng.randint(1, 3))


class Outputs(tuple):
    """Output tensors that are views of buffers which ``owner`` frees with itself."""

    def __new__(cls, owner, *tensors):
        self = super().__new__(cls, tensors)
        self.owner = owner
        return self


def _modulus(ring):
    return Modulus32.Q_32 if ring == "q32" else CRT_SET_30BIT[0]


def _residues(shape, ring, seed, stream):
    """A CUDA tensor of canonical residues."""
    gl = ring == "gl"
    t = torch.empty(shape, dtype=torch.int64 if gl else torch.int32, device="cuda")
    return synth.fill_device(t, "gl", seed, stream) if gl else synth.fill_device(t, "mod32", seed, stream, q=_modulus(ring).q)


def _bytes(shape, kind, seed, stream):
    t = synth.fill_device(torch.empty(shape, dtype=torch.int8, device="cuda"), "i8", seed, stream)
    return t.view(torch.uint8) if kind == "u8" else t


def _job_sizes(case):
    """(log d, Goldilocks or CRT set, rows, ring elements) of every job: the case's own, whatever the seed."""
    rng, lo, hi = np.random.default_rng(case["jobs"]), 10, case["log_max"]
    return [(6 + int(rng.integers(3)), bool(rng.integers(2)), int(rng.choice([8, 16])),
             int(2.0 ** (lo + (hi - lo) * rng.random()))) for _ in range(case["jobs"])]


def _prepare_batch(case, seed):
    """Key classes (three degrees, Goldilocks and the CRT set; kappa = 16) and the jobs' sizes, witnesses and outputs."""
    specs = [(ld, gl) for gl in (True, False) for ld in (6, 7, 8)]
    m = 1 << case["log_max"]
    classes = []
    for ci, (ld, gl) in enumerate(specs):
        shape = 16 * m << ld
        if gl:
            classes.append([GoldilocksAjtaiKey(ld, 16, m, _residues(shape, "gl", seed, 100 + ci))])
        else:
            a = torch.empty(shape, dtype=torch.int32, device="cuda")
            classes.append([U32AjtaiKey(mod, ld, 16, m, synth.fill_device(a, "mod32", seed, 100 + 8 * ci + pi, q=mod.q))
                            for pi, mod in enumerate(CRT_SET_30BIT)])
    sizes = _job_sizes(case)
    totals = [sum(kappa << ld if g else 4 * kappa << ld for ld, g, kappa, _ in sizes if g == gl) for gl in (True, False)]
    out = [torch.zeros(max(1, totals[0]), dtype=torch.int64, device="cuda"),
           torch.zeros(max(1, totals[1]), dtype=torch.int32, device="cuda")]
    jobs, at = [], [0, 0]
    for j, (ld, gl, kappa, n) in enumerate(sizes):
        shape, o = ((1 if gl else 4), kappa, 1 << ld), 0 if gl else 1
        size = shape[0] * kappa << ld
        jobs.append(CommitJob(specs.index((ld, gl)), kappa, n, _bytes((n, 1 << ld), "i8", seed, 1000 + j),
                              out[o][at[o]:at[o] + size].view(shape)))
        at[o] += size
    return dict(batch=CommitBatch(classes, jobs), out=out)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "commit":
        d, shape = 1 << case["log_d"], (case["batch"], case["m"], 1 << case["log_d"])
        A = _residues(case["kappa"] * case["m"] * d, case["ring"], seed, 1)
        if case["ring"] == "gl":
            key = GoldilocksAjtaiKey(case["log_d"], case["kappa"], case["m"], A)
        else:
            key = U32AjtaiKey(_modulus(case["ring"]), case["log_d"], case["kappa"], case["m"], A)
        if case["digits"] == "residues":
            w = _residues(shape, case["ring"], seed, 2)
        else:
            w = _bytes(shape, case["digits"], seed, 2)
        if case["host"]:
            w = w.cpu().numpy()
            if case["digits"] == "residues":
                w = w.view(np.uint64 if case["ring"] == "gl" else np.uint32)
        return dict(kind=kind, key=key, w=w)
    if kind == "packed":
        ring = RingConfig(Modulus32.Q_32, case["log_d"])
        d, k, m = 1 << case["log_d"], case["kappa"], case["m"]
        key = AjtaiPublicKey.from_seed(AjtaiParams(ring, k, m, 1 << 22), int(seed).to_bytes(32, "little"))
        values = _residues((case["batch"], m * d // 3), "gl", seed, 2)  # m is a multiple of 3: the columns pack back to back
        return dict(kind=kind, ring=ring, key=key, values=values, shape=(case["batch"], m, d))
    if kind == "derive":
        ring = RingConfig(Modulus32.Q_32, case["log_d"])
        w = _residues((1, case["m"], 1 << case["log_d"]), "q32", seed, 2)
        return dict(kind=kind, params=AjtaiParams(ring, case["kappa"], case["m"], 1 << 31), seed=int(seed).to_bytes(32, "little"), w=w)
    if kind == "ntt":
        n, count, ring = 1 << case["log_n"], case["count"], case["ring"]
        if ring == "crt":
            t = NttTables(CRT_SET_30BIT, case["log_n"])
            a = torch.empty((4, count, n), dtype=torch.int32, device="cuda")
            for i, mod in enumerate(CRT_SET_30BIT):
                synth.fill_device(a[i], "mod32", seed, i, q=mod.q)
        else:
            t = GoldilocksNttTables(case["log_n"]) if ring == "gl" else NttTables(_modulus(ring), case["log_n"])
            a = _residues((count, n), ring, seed, 1)
        return dict(kind=kind, fn=t.inverse_fast if case["inverse"] else t.forward_fast, a=a, out=torch.empty_like(a))
    if kind == "batch":
        return dict(kind=kind, **_prepare_batch(case, seed))
    if kind == "fold":
        m = case["m"]
        key = GoldilocksAjtaiKey(6, case["kappa"], m, _residues(case["kappa"] * m * 64, "gl", seed, 1))
        pipe = FoldPipeline(key, NttTables(CRT_SET_30BIT, 6))
        synth.fill_device(pipe.z, "gl", seed, 2)
        return dict(kind=kind, pipe=pipe)
    if kind == "ring50":
        n, count = 1 << case["log_n"], case["count"]
        a, b = (synth.fill_device(torch.empty((count, n), dtype=torch.int64, device="cuda"), "u64", seed, s) for s in (1, 2))
        return dict(kind=kind, ring=RingConfig50(case["log_n"]), a=(a & ((1 << 62) - 1)) % Q_50, b=(b & ((1 << 62) - 1)) % Q_50)
    limbs = LIMBS[:case["limbs"]]
    key = CommitmentKey.random(case["len_f162"], seed, limbs[0], limbs[1:])
    w = synth.fill_device(torch.empty((case["columns"] * case["len_f162"], 3), dtype=torch.int64, device="cuda"), "u64", seed, 1)
    w[:, 2] &= (1 << 34) - 1
    return dict(kind=kind, key=key, w=w, columns=case["columns"])


def run(state):
    kind = state["kind"]
    if kind == "commit":
        return state["key"].commit(state["w"])
    if kind == "packed":
        batch, m, _ = state["shape"]
        packed = pack_field_elements(state["ring"], state["values"], batch * m)
        return state["key"].commit_batch(packed.view(state["shape"]))
    if kind == "derive":
        return AjtaiPublicKey.from_seed(state["params"], state["seed"]).commit_batch(state["w"])
    if kind == "ntt":
        return state["fn"](state["a"], state["out"])
    if kind == "batch":
        state["batch"].run()
        return state["out"]
    if kind == "fold":
        p = state["pipe"]
        p.run()
        return Outputs(p, p.digits, p.commits, p.crt_ntt)
    if kind == "ring50":
        return state["ring"].mul(state["a"], state["b"])
    matrix, aux = state["key"].commit(state["w"], state["columns"])
    return matrix.value, aux.raw, aux.batches


def work(case):
    """Bytes: every input (the resident key with them) read once, every output written once.  Flops: two per
    coefficient product of the transform-domain sums, and per butterfly of the transforms (log2 n / 2 a value)."""
    kind = case["kind"]
    if kind in ("commit", "packed", "derive"):
        gl = case.get("ring") == "gl"
        d, k, m, b = 1 << case["log_d"], case["kappa"], case["m"], case.get("batch", 1)
        e = 8 if gl else 4
        if kind == "packed":
            wb = b * (m * d // 3) * 8
        else:
            wb = b * m * d * (e if case.get("digits", "residues") == "residues" else 1)
        key = 32 if kind == "derive" else k * m * d * e
        lg = case["log_d"]
        transforms = (b * (m + k) + (k * m if kind == "derive" else 0)) * d * lg
        return dict(bytes=wb + key + b * k * d * e, flops=2 * b * k * m * d + transforms)
    if kind == "ntt":
        values = case["count"] * (4 if case["ring"] == "crt" else 1) << case["log_n"]
        return dict(bytes=2 * values * (8 if case["ring"] == "gl" else 4), flops=values * case["log_n"])
    if kind == "batch":
        nb = fl = 0
        longest = {}
        for ld, gl, kappa, n in _job_sizes(case):
            keys, e = (1, 8) if gl else (4, 4)
            nb += (n << ld) + (keys * kappa * e << ld)
            fl += keys * (2 * kappa * n + n * ld) << ld
            longest[ld, gl] = max(longest.get((ld, gl), 0), keys * e * 16 * n << ld)
        return dict(bytes=nb + sum(longest.values()), flops=fl)
    if kind == "fold":
        m, k = case["m"], case["kappa"]
        return dict(bytes=m * 64 * (8 + 8 * k + 8 + 16) + 8 * k * 64 * 8, flops=2 * 8 * k * m * 64 + (8 + 4) * m * 64 * 6)
    if kind == "ring50":
        values = case["count"] << case["log_n"]
        return dict(bytes=3 * 8 * values, flops=values * (3 * (case["log_n"] - 1) + 5))
    ring_elements, limbs = case["columns"] * case["len_f162"] // 4, case["limbs"]
    out = case["columns"] * 648 * limbs * (4 + 2) + ring_elements * 648 * 4
    return dict(bytes=ring_elements * 96 + limbs * case["len_f162"] // 4 * 648 * 2 + out,
                flops=ring_elements * limbs * 648 * (2 + 10))


def exact(case, seed):
    """Every output is an exact residue or a byte: there is no error against 64-bit floating point to measure."""
    return None
