"""What a user of this library has it do, as cases to time: whole proofs, the commitment and opening of columns, transforms,
multi-scalar multiplications and the sumcheck rounds, each through the public Python entry points.

listed() gives the cases, draw() further ones of the same ranges; prepare() makes the inputs of a case on the GPU from a seed,
run() is one pass over them, work() what a pass cannot do without, tolerance() how far two correct results may differ."""
import hashlib
import math

import numpy as np
import torch

from project_b200 import KIND_FR, KIND_FR_MONT, KIND_G1, KIND_I64, KIND_U32, Backend, synthetic
from project_b200.flow import gpu_flow

# The BLS12-381 G1 generator, affine x || y, 2 x 48 bytes little-endian.
_GENERATOR = np.frombuffer(
    int("17f1d3a73197d7942695638c4fa9ac0fc3688c4f9774b905a14e3a3f171bac586c55e83ff97a1aeffb3af00adb22c6bb", 16).to_bytes(48, "little")
    + int("08b3f481e3aaa0f1a09e30ed741d8ae4fcf5e095d5d00af600db18cb2c04b3edd03cc744a2888ae40caa232946c5e7e1", 16).to_bytes(48, "little"),
    dtype=np.uint8,
)
_LIMB_PRODUCTS_FR, _LIMB_PRODUCTS_FP = 136, 300  # 32 x 32-bit products of one Montgomery multiplication (8 and 12 limbs)

_backend = None


def _context():
    """The one context a program keeps for its calls on a GPU."""
    global _backend
    if _backend is None:
        _backend = Backend(torch.cuda.current_device())
    return _backend


def listed():
    return [
        # A whole proof from host inputs at the size of a test graph: hundreds of short kernels and 20-odd read-backs, one after another.
        {"name": "proof_small", "op": "proof", "nodes": 1500, "directed_edges": 6000, "features": 64, "layers": 1, "heads": 2, "width": 8,
         "output_heads": 2, "classes": 3, "citation": False, "compact": False},
        # The mid-size configuration of the benchmark: many narrow heads, 1212 commitments in 69 barriers.
        {"name": "proof_mid", "op": "proof", "nodes": 19717, "directed_edges": 88648, "features": 500, "layers": 1, "heads": 8, "width": 8,
         "output_heads": 8, "classes": 3, "citation": False, "compact": False},
        # The 169k-node benchmark's model (wide heads, two hidden layers) on 1/32 of its graph, as the benchmark's host arm runs it.
        {"name": "proof_wide", "op": "proof", "nodes": 5291, "directed_edges": 36445, "features": 128, "layers": 2, "heads": 3, "width": 256,
         "output_heads": 1, "classes": 40, "citation": True, "compact": True},
        # The whole 169k-node citation graph with the narrow model of its published run (one hidden head of 8, 40 classes).
        {"name": "proof_large", "op": "proof", "nodes": 169343, "directed_edges": 1166243, "features": 128, "layers": 1, "heads": 1, "width": 8,
         "output_heads": 1, "classes": 40, "citation": True, "compact": True},
        # One commit barrier over node columns of the mid-size graph: a short call, bound by its dependent steps.
        {"name": "commit_node", "op": "commit", "log2n": 15, "length": 19717, "field": 8, "i64": 12, "u32": 4},
        # Opening of edge columns of the large graph at a fresh point and its rotation, weights included.
        {"name": "open_edge", "op": "open", "log2n": 22, "length": 2500733, "field": 12, "i64": 8, "u32": 4, "points": 2},
        # A batch of short transforms (per-column work of a small domain).
        {"name": "ntt_small", "op": "ntt", "log2n": 12, "batch": 4, "inverse": False, "coset": False, "canonical": True},
        # One long transform back from a coset.
        {"name": "ntt_large", "op": "ntt", "log2n": 22, "batch": 1, "inverse": True, "coset": True, "canonical": False},
        # Low-degree extension of one column, as a quotient needs it.
        {"name": "lde", "op": "lde", "log2n": 20, "log2_blowup": 1},
        # Commitment to one column against points met for the first time.
        {"name": "msm", "op": "msm", "log2n": 16, "table": False, "witness": False},
        # The same against the resident table of an SRS.
        {"name": "msm_table", "op": "msm", "log2n": 20, "table": True, "witness": False},
        # All rounds of a sumcheck, the challenges hashed from the round values on the host.
        {"name": "sumcheck", "op": "sumcheck", "log2n": 20, "canonical": False},
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    op = rng.choice(["proof", "proof", "proof", "commit", "open", "ntt", "ntt", "lde", "msm", "msm", "sumcheck"])
    if op == "proof":
        nodes = _log_uniform(rng, 300, 160000)
        citation = rng.random() < 0.5
        # the wider the model the smaller the graph: the products of the forward pass stay below those of the listed cases
        width = min(rng.choice([8, 8, 16, 24, 64, 256]), 8 if nodes > 20000 else 64 if nodes > 5000 else 256)
        heads = rng.randint(1, 1 if nodes > 60000 else 4 if width <= 64 else 2)
        layers = rng.randint(1, 1 if nodes > 20000 else 2)
        return {"op": "proof", "nodes": nodes, "directed_edges": int(nodes * rng.uniform(3.0, 7.0)), "features": rng.choice([50, 64, 128] if nodes > 20000 else [50, 64, 128, 500]),
                "layers": layers, "heads": heads, "width": width, "output_heads": rng.randint(1, 1 if nodes > 20000 else 4), "classes": rng.choice([3, 7, 40]),
                "citation": citation, "compact": nodes > 20000 or rng.random() < 0.5}
    if op == "commit":
        log2n = rng.randint(6, 20)
        return {"op": "commit", "log2n": log2n, "length": rng.randint((1 << log2n) // 2 + 1, 1 << log2n), "field": rng.randint(0, 12), "i64": rng.randint(0, 12),
                "u32": rng.randint(1, 5)}
    if op == "open":
        log2n = rng.randint(10, 22)
        length = rng.randint((1 << log2n) // 2 + 1, 1 << log2n)
        return {"op": "open", "log2n": log2n, "length": min(length, 2500000), "field": rng.randint(1, 12), "i64": rng.randint(0, 8), "u32": rng.randint(0, 4),
                "points": rng.randint(1, 2)}
    if op == "ntt":
        log2n = rng.randint(8, 22)
        batch = min(rng.choice([1, 1, 3, 4, 16, 64]), 1 << (22 - log2n))
        return {"op": "ntt", "log2n": log2n, "batch": batch, "inverse": rng.random() < 0.5, "coset": rng.random() < 0.5, "canonical": rng.random() < 0.5}
    if op == "lde":
        log2n = rng.randint(10, 20)
        return {"op": "lde", "log2n": log2n, "log2_blowup": rng.randint(1, min(3, 21 - log2n))}
    if op == "msm":
        return {"op": "msm", "log2n": rng.uniform(10.0, 20.0), "table": rng.random() < 0.5, "witness": rng.random() < 0.3}
    return {"op": "sumcheck", "log2n": rng.randint(10, 22), "canonical": rng.random() < 0.5}


class _State:
    """A case's inputs and outputs.  Device arrays are torch tensors the library works on in place."""

    def __init__(self, case):
        self.case = case
        self.flow = None
        self._buffers = []

    def own(self, buffer):
        self._buffers.append(buffer)
        return buffer

    def array(self, kind, tensor):
        """The library's view of a tensor, which lives as long as the state."""
        torch.cuda.current_stream().synchronize()  # the library works on a stream of its own
        buffer = self.own(_context().wrap(kind, tensor.shape[0], tensor.data_ptr()))
        buffer.tensor = tensor
        return buffer

    def __del__(self):
        try:
            if self.flow is not None:
                self.flow.close()
            for buffer in self._buffers:
                buffer.free()
        except Exception:
            pass  # the interpreter is going down


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _field(g, n):
    """n uniform-looking canonical field elements: four 64-bit words each, the top one below the modulus'."""
    t = torch.randint(-(1 << 63), (1 << 63) - 1, (n, 4), dtype=torch.int64, device="cuda", generator=g)
    t[:, 3] &= (1 << 62) - 1
    return t


def _empty(n):
    return torch.empty((n, 4), dtype=torch.int64, device="cuda")


def _witness(g, n, kind):
    """A quantised witness column: values of a few bits, signed for I64; a count or a selector for U32."""
    if kind == KIND_U32:
        return torch.randint(0, 1 << 12, (n,), dtype=torch.int32, device="cuda", generator=g)
    return torch.round(torch.randn(n, device="cuda", generator=g) * 48.0).to(torch.int64)


def _scalar(seed):
    """One canonical field element from a seed."""
    b = np.frombuffer(hashlib.sha256(b"scalar %d" % seed).digest(), dtype=np.uint8).copy()
    b[31] &= 0x3F
    return b


def _columns(s, g, rows):
    c = s.case
    kinds = [KIND_FR_MONT] * c["field"] + [KIND_I64] * c["i64"] + [KIND_U32] * c["u32"]
    return [s.array(k, _field(g, rows) if k == KIND_FR_MONT else _witness(g, rows, k)) for k in kinds]


def prepare(case, seed):
    s, op = _State(case), case["op"]
    if op == "proof":
        inputs = synthetic.make_inputs(
            seed=seed, nodes=case["nodes"], directed_edges=case["directed_edges"], feature_count=case["features"], hidden=[(case["heads"], case["width"])] * case["layers"],
            output_heads=case["output_heads"], class_count=case["classes"], power_law=True, symmetrize=case["citation"], feature_kind="gauss" if case["citation"] else "exp")
        s.flow = gpu_flow(torch.cuda.current_device(), inputs, _GENERATOR, compact_columns=case["compact"])
        return s
    be, g = _context(), _generator(seed)
    if op == "commit":
        s.cols = _columns(s, g, case["length"])
        s.weights = s.array(KIND_FR_MONT, _empty(1 << case["log2n"]))
        be.bary_weights(case["log2n"], _scalar(7), out=s.weights)  # the weights at tau belong to the key
    elif op == "open":
        s.cols = _columns(s, g, case["length"])
        s.point = _scalar(seed)
        s.weights = s.array(KIND_FR_MONT, _empty(1 << case["log2n"]))
    elif op == "ntt":
        n = case["batch"] << case["log2n"]
        s.vec = s.array(KIND_FR if case["canonical"] else KIND_FR_MONT, _field(g, n))
        s.out = s.array(KIND_FR_MONT, _empty(n))
        s.shift = _scalar(seed) if case["coset"] else None
    elif op == "lde":
        s.vec = s.array(KIND_FR_MONT, _field(g, 1 << case["log2n"]))
        s.out = s.array(KIND_FR_MONT, _empty(1 << (case["log2n"] + case["log2_blowup"])))
        s.shift = _scalar(seed)
    elif op == "msm":
        n = s.n = int(2 ** case["log2n"])
        if case["witness"]:  # a committed witness column, widened as the proof flow does it
            column = s.array(KIND_I64, _witness(g, n, KIND_I64))
            s.scalars = s.array(KIND_FR_MONT, _empty(n))
            be.linear_combination([column], np.eye(1, 32, dtype=np.uint8), n, n, out=s.scalars)
        else:
            s.scalars = s.array(KIND_FR, _field(g, n))
        s.points = s.own(be.g1_fixed_base_mul(_GENERATOR, s.array(KIND_FR, _field(g, n)), n))
        if case["table"]:
            s.table, s.window_bits = be.msm_precompute(s.points, n)
            s.own(s.table)
    else:
        n = 1 << case["log2n"]
        kind = KIND_FR if case["canonical"] else KIND_FR_MONT
        s.vec = s.array(kind, _field(g, n))
        s.halves = [s.array(kind, _empty(n // 2)), s.array(kind, _empty(max(1, n // 4)))]
    torch.cuda.synchronize()
    return s


def run(s):
    be, case, op = _context(), s.case, s.case["op"]
    if op == "proof":
        s.flow.prove()
        return s.flow.proof_bytes()
    if op == "commit":
        return be.commit_batch(s.cols, case["length"], case["log2n"], s.weights, _GENERATOR)
    if op == "open":
        be.bary_weights(case["log2n"], s.point, out=s.weights)
        return s.weights.tensor, be.eval_batch(s.cols, case["length"], case["log2n"], s.weights, (0, 1)[:case["points"]])
    if op == "ntt":
        return be.ntt(s.vec, case["log2n"], batch=case["batch"], inverse=case["inverse"], coset_shift=s.shift, out=s.out).tensor
    if op == "lde":
        return be.coset_lde(s.vec, case["log2n"], case["log2_blowup"], s.shift, out=s.out).tensor
    if op == "msm":
        return be.msm_precomputed(s.scalars, s.table, s.n, s.window_bits) if case["table"] else be.msm(s.scalars, s.points, s.n)
    table, rounds, transcript = s.vec, [], hashlib.sha256(b"sumcheck")
    for j in range(case["log2n"]):
        n = 1 << (case["log2n"] - j)
        rounds.append(be.sumcheck_round_sums(table, n))
        transcript.update(rounds[-1].tobytes())
        challenge = np.frombuffer(transcript.digest(), dtype=np.uint8).copy()
        challenge[31] &= 0x3F
        table = be.fold(table, n, challenge, out=s.halves[j % 2])
    return np.stack(rounds), table.download(count=1)


def _field_work(bytes_moved, multiplications):
    return {"bytes": float(bytes_moved), "flops": 2.0 * _LIMB_PRODUCTS_FR * multiplications}


def work(case):
    """Bytes: inputs read and outputs written once.  flops: two per 32 x 32-bit product of the field multiplications (and two
    per multiply-add of a proof's forward pass)."""
    op = case["op"]
    if op == "proof":
        nodes, edges = case["nodes"], case["directed_edges"] * (2 if case["citation"] else 1) + case["nodes"]
        width, heads, bytes_moved, madds, terms = case["features"], 0, 8.0 * case["nodes"] * case["features"] + 8.0 * edges, 0.0, 0.0
        for layer in range(case["layers"] + 1):
            k, w = (case["heads"], case["width"]) if layer < case["layers"] else (case["output_heads"], case["classes"])
            madds += k * w * (float(nodes) * width + edges)
            bytes_moved += k * (3 * 8.0 * nodes * w)  # the three quantised matrices of a head
            terms += k * 3.0 * nodes * w
            heads += k
            width = k * w
        # a head commits about 12 small-integer and 20 field-element edge columns, 5 and 10 node columns
        bytes_moved += heads * (edges * (12 * 8.0 + 20 * 32.0) + nodes * (5 * 8.0 + 10 * 32.0))
        terms += heads * 3.0 * (32.0 * edges + 15.0 * nodes)  # at tau, z and omega z: half a multiplication each, unreduced
        return {"bytes": bytes_moved, "flops": 2.0 * madds + 2.0 * 64.0 * terms}
    if op in ("commit", "open"):
        rows, columns = case["length"], case["field"] + case["i64"] + case["u32"]
        stored = rows * (32.0 * case["field"] + 8.0 * case["i64"] + 4.0 * case["u32"])
        if op == "commit":
            limbs = rows * (64.0 * case["field"] + 8.0 * (case["i64"] + case["u32"])) + columns * 700.0 * _LIMB_PRODUCTS_FP / 8
            return {"bytes": stored + 32.0 * rows + columns * 128.0, "flops": 2.0 * limbs}
        n = float(1 << case["log2n"])
        limbs = case["points"] * rows * (64.0 * case["field"] + 8.0 * (case["i64"] + case["u32"])) + 4.0 * n * _LIMB_PRODUCTS_FR
        return {"bytes": stored + 32.0 * n + case["points"] * columns * 32.0, "flops": 2.0 * limbs}
    if op == "ntt":
        n = float(case["batch"] << case["log2n"])
        return _field_work(64.0 * n, n * case["log2n"] / 2 + (n if case["inverse"] or case["coset"] or case["canonical"] else 0))
    if op == "lde":
        n, big = float(1 << case["log2n"]), float(1 << (case["log2n"] + case["log2_blowup"]))
        return _field_work(32.0 * (n + big), n * case["log2n"] / 2 + big * (case["log2n"] + case["log2_blowup"]) / 2 + n)
    if op == "msm":
        n = float(int(2 ** case["log2n"]))
        bits = 8 if case["witness"] else 255
        additions = n * math.ceil(bits / 16.0)  # one mixed addition of ten multiplications per point and 16-bit digit
        return {"bytes": 128.0 * n, "flops": 2.0 * _LIMB_PRODUCTS_FP * 10.0 * additions}
    n = float(1 << case["log2n"])
    return _field_work(32.0 * n, n)


def tolerance(case):
    """Field elements, curve points and proofs are exact: any correct implementation gives the same bytes."""
    return "exact"
