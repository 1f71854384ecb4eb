"""Workloads of the commitment path, through the package's public classes.

Each case is one call (or the few calls of one job) that a prover makes: a batch of
Poseidon2 permutations, a coset LDE, a Merkle commitment, a PCS commitment, a FRI commit
phase, a whole commit + FRI job, a batch of small traces under one plan.  Inputs are
uniform field elements, as witness columns and codewords are to the kernels; every output
is an exact integer modulo the field's prime.

`listed()` names the cases, `draw(rng)` gives one more of the same ranges, `prepare` makes
what a prover holds before the call, `run` is the call, `work` the bytes and operations it
cannot do without.
"""
import math

import numpy as np
import torch

import ziros_b200 as Z

BB_P = 0x78000001
SEED = 42            # Poseidon2 constants
ALPHA = (0x1234567, 0x2345678, 0x3456789, 0x456789A)
LARGEST = 1 << 31    # LDE cells (BabyBear) of the largest job


def listed():
    return [
        # A transcript's or a witness generator's permutations: one short launch.
        {"name": "perm_bb_1000", "kind": "perm", "field": "bb", "n": 1000},
        # The extension alone, as a quotient or preprocessed-column step asks for it.
        {"name": "lde_bb_2^20x64", "kind": "lde", "field": "bb", "log_h": 20, "width": 64, "blowup": 1,
         "bitrev": True},
        # The same in natural order on a width that no column chunk divides.
        {"name": "lde_bb_2^16x37_b2", "kind": "lde", "field": "bb", "log_h": 16, "width": 37, "blowup": 2,
         "bitrev": False},
        {"name": "lde_gl_2^20x64_b2", "kind": "lde", "field": "gl", "log_h": 20, "width": 64, "blowup": 2,
         "bitrev": True},
        # A small circuit's commitment: many short kernels.
        {"name": "pcs_bb_2^14x16", "kind": "pcs", "field": "bb", "p2": 16, "log_h": 14, "width": 16, "blowup": 1},
        # Goldilocks commitments with both hashers, a middle and a full-size one.
        {"name": "pcs_gl_w16_2^16x30", "kind": "pcs", "field": "gl", "p2": 16, "log_h": 16, "width": 30, "blowup": 1},
        {"name": "pcs_gl_w12_2^20x64_b2", "kind": "pcs", "field": "gl", "p2": 12, "log_h": 20, "width": 64,
         "blowup": 2},
        # Matrices of several heights in one tree (a multi-table proof), then two openings.
        {"name": "mmcs_bb_mixed", "kind": "mmcs", "field": "bb", "p2": 16,
         "shapes": "131072x30,131072x11,32768x67,1024x5", "opens": 2},
        # The FRI commit phase and its query answers on a codeword in device memory.
        {"name": "fri_2^22_q100", "kind": "fri", "log_n": 22, "log_final": 8, "queries": 100, "transcript": False},
        # A middle job from host memory with the Fiat-Shamir transcript.
        {"name": "job_host_2^17x200", "kind": "job", "host": True, "log_h": 17, "width": 200, "log_final": 8,
         "queries": 100, "transcript": True},
        # The full-size job: trace in device memory, LDE + Merkle + FRI.
        {"name": "job_bb_2^22x256", "kind": "job", "host": False, "log_h": 22, "width": 256, "log_final": 8,
         "queries": 100, "transcript": False},
        # Many small traces (one per shard or table) under one plan.
        {"name": "batch_64_small", "kind": "batch", "count": 64, "lo": 8, "hi": 14, "max_w": 64, "shape_seed": 3},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_h(rng, lo, hi, width, blowup, limit):
    top = hi
    while top > lo and (width << (top + blowup)) > limit:
        top -= 1
    return rng.randint(lo, top)


def draw(rng):
    kind = rng.choice(["perm", "lde", "lde", "pcs", "pcs", "mmcs", "fri", "job", "job", "batch"])
    field = rng.choice(["bb", "bb", "gl"])
    if kind == "perm":
        return {"kind": "perm", "field": field, "n": _log_uniform(rng, 100, 2000000)}
    if kind == "lde":
        width, blowup = _log_uniform(rng, 1, 300), rng.randint(1, 3)
        return {"kind": "lde", "field": field, "log_h": _log_h(rng, 6, 21, width, blowup, LARGEST >> 2), "width": width,
                "blowup": blowup, "bitrev": rng.random() < 0.7}
    if kind == "pcs":
        width, blowup = _log_uniform(rng, 1, 300), rng.randint(1, 3)
        p2 = rng.choice([12, 16]) if field == "gl" else 16
        limit = LARGEST >> 1 if field == "bb" else LARGEST >> 3
        return {"kind": "pcs", "field": field, "p2": p2, "log_h": _log_h(rng, 6, 21, width, blowup, limit),
                "width": width, "blowup": blowup}
    if kind == "mmcs":
        top = rng.randint(8, 18)
        hs, shapes = sorted({top, rng.randint(4, top), rng.randint(4, top)}, reverse=True), []
        for h in hs:
            for _ in range(rng.randint(1, 3)):
                shapes.append(f"{1 << h}x{_log_uniform(rng, 1, 150)}")
        p2 = rng.choice([12, 16]) if field == "gl" else 16
        return {"kind": "mmcs", "field": field, "p2": p2, "shapes": ",".join(shapes), "opens": rng.randint(1, 4)}
    if kind == "fri":
        log_n = rng.randint(10, 23)
        return {"kind": "fri", "log_n": log_n, "log_final": rng.randint(2, min(8, log_n - 1)),
                "queries": rng.randint(20, 120), "transcript": rng.random() < 0.5}
    if kind == "job":
        width, host = _log_uniform(rng, 8, 300), rng.random() < 0.3
        log_h = _log_h(rng, 8, 22, width, 1, LARGEST >> (4 if host else 1))
        return {"kind": "job", "host": host, "log_h": log_h, "width": width, "log_final": rng.randint(2, 8),
                "queries": rng.randint(20, 120), "transcript": rng.random() < 0.5}
    lo = rng.randint(6, 10)
    return {"kind": "batch", "count": rng.randint(8, 96), "lo": lo, "hi": rng.randint(lo + 1, 15),
            "max_w": rng.randint(8, 100), "shape_seed": rng.randint(0, 1 << 20)}


# ------------------------------------------------------------------------ preparation
def _field(case):
    return Z.GOLDILOCKS if case.get("field") == "gl" else Z.BABYBEAR


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1000003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _uniform(field, shape, g):
    """Canonical field elements: int32 words (BabyBear) or int64 words (Goldilocks)."""
    if field == Z.BABYBEAR:
        return torch.randint(0, BB_P, shape, dtype=torch.int32, device="cuda", generator=g)
    v = torch.randint(0, 0xFFFFFFFF, shape, dtype=torch.int64, device="cuda", generator=g)  # high word below 2^32 - 1
    v.bitwise_left_shift_(32)
    lo = torch.randint(-(1 << 31), 1 << 31, shape, dtype=torch.int32, device="cuda", generator=g)
    v.bitwise_or_(lo.to(torch.int64).bitwise_and_(0xFFFFFFFF))
    return v


def _mmcs_shapes(case):
    return [tuple(int(x) for x in s.split("x")) for s in case["shapes"].split(",")]


def _batch_shapes(case):
    r = np.random.default_rng(case["shape_seed"])
    return [(1 << int(r.integers(case["lo"], case["hi"] + 1)), int(r.integers(1, case["max_w"] + 1)))
            for _ in range(case["count"])]


def prepare(case, seed):
    kind, field, g = case["kind"], _field(case), _gen(seed)
    st = {"case": case, "field": field}
    if kind == "perm":
        st["rc"], st["ne"], st["ni"] = Z.round_constants(field, SEED)
        st["x"] = _uniform(field, (case["n"], 16), g)
        st["op"] = Z.CudaPoseidon2.new()
    elif kind == "lde":
        h, w = 1 << case["log_h"], case["width"]
        st["x"] = _uniform(field, (h, w), g)
        st["out"] = torch.empty((h << case["blowup"], w), dtype=st["x"].dtype, device="cuda")
        st["op"] = Z.CudaDft.new(field)
    elif kind == "pcs":
        st["x"] = _uniform(field, (1 << case["log_h"], case["width"]), g)
        st["op"] = Z.CudaTwoAdicPcs(field, SEED, case["blowup"], case["p2"])
    elif kind == "mmcs":
        st["x"] = [_uniform(field, s, g) for s in _mmcs_shapes(case)]
        st["op"] = Z.CudaMerkleTreeMmcs(field, SEED, case["p2"])
        top = max(s[0] for s in _mmcs_shapes(case))
        r = np.random.default_rng(seed)
        st["idx"] = [int(i) for i in r.integers(0, top, size=case["opens"])]
    elif kind == "fri":
        st["x"] = _uniform(field, (1 << case["log_n"], 4), g)
        st["op"] = Z.CudaFriProver(SEED, case["log_final"], case["queries"], challenge_seed=seed, query_seed=seed + 1,
                                   transcript=case["transcript"])
    elif kind == "job":
        x = _uniform(field, (1 << case["log_h"], case["width"]), g)
        st["x"] = x.cpu().pin_memory() if case["host"] else x
        st["op"] = Z.CudaTwoAdicPcs(field, SEED, 1)
        st["seeds"] = (seed, seed + 1)
    elif kind == "batch":
        shapes = _batch_shapes(case)
        st["x"] = [_uniform(field, s, g) for s in shapes]
        st["op"] = Z.BatchCommit(shapes, field=field, seed=SEED, log_blowup=1, autotune=False)
    torch.cuda.synchronize()
    return st


# -------------------------------------------------------------------------- the calls
def _proof(pf):
    return {"roots": pf.roots, "betas": pf.betas, "final": pf.final, "indices": pf.query_indices,
            "rows": pf.query_rows, "siblings": pf.query_siblings}


def run(state):
    case, kind, x, op = state["case"], state["case"]["kind"], state["x"], state["op"]
    if kind == "perm":
        y = x.clone()  # the permutation works in place
        op.batch_permute_dev(state["field"], y, state["rc"], state["ne"], state["ni"])
        return y
    if kind == "lde":
        op.coset_lde_batch_dev(x, case["blowup"], state["out"], bit_reverse_rows=case["bitrev"])
        return state["out"]
    if kind == "pcs":
        root, tree = op.commit_dev(x)
        return root
    if kind == "mmcs":
        root, tree = op.commit_dev(x)
        opened = [op.open_batch(i, tree) for i in state["idx"]]
        return {"root": root, "opened": opened}
    if kind == "fri":
        return _proof(op.commit_dev(x))
    if kind == "job":
        kw = dict(alpha=ALPHA, log_final=case["log_final"], num_queries=case["queries"],
                  challenge_seed=state["seeds"][0], query_seed=state["seeds"][1], transcript=case["transcript"])
        if case["host"]:
            root, _, pf = op.commit_fri_ptr(x.data_ptr(), x.shape[0], x.shape[1], **kw)
        else:
            root, _, pf = op.commit_fri_dev(x, **kw)
        return {"root": root, **_proof(pf)}
    stream = torch.cuda.current_stream().cuda_stream
    for i, t in enumerate(x):
        op.copy_in(i, t)
    op.run(stream)
    return op.roots(stream)


# ------------------------------------------------------------------------------- work
def _perm_muls(field, p2):
    """Products of one permutation: x^7 is four, and the Goldilocks diagonal one a lane."""
    if field == Z.BABYBEAR:
        return 4 * (8 * 16 + 13)
    return 4 * (8 * p2 + 22) + 22 * p2


def _sponge_perms(width):
    return (width + 7) // 8


def _lde_muls(log_h, width, blowup):
    """Half a product per butterfly level and element, inverse and forward transforms."""
    return width * (1 << log_h) * (log_h / 2 + (1 << blowup) * (log_h + 2) / 2)


def _commit(field, p2, log_h, width, blowup):
    es = 4 if field == Z.BABYBEAR else 8
    rows, out = 1 << (log_h + blowup), 8 if p2 == 16 else 4
    perms = rows * _sponge_perms(width) + rows - 1
    return {"bytes": es * (width * ((1 << log_h) + 2 * rows) + 2 * rows * out),
            "flops": _lde_muls(log_h, width, blowup) + perms * _perm_muls(field, p2)}


def _fri(log_n, log_final, queries):
    rows = sum(1 << (log_n - 1 - r) for r in range(log_n - log_final))
    perms = 2 * rows  # a leaf and (nearly) a compression for each sibling pair
    return {"bytes": 16 * ((1 << log_n) + 2 * rows) + 64 * rows + queries * 32 * log_n * log_n // 2,
            "flops": perms * _perm_muls(Z.BABYBEAR, 16) + 24 * rows}


def work(case):
    """Bytes of inputs and outputs once each; `flops` counts field products."""
    kind, field = case["kind"], _field(case)
    es = 4 if field == Z.BABYBEAR else 8
    if kind == "perm":
        return {"bytes": case["n"] * 16 * es * 2, "flops": case["n"] * _perm_muls(field, 16)}
    if kind == "lde":
        cells = case["width"] << case["log_h"]
        return {"bytes": es * (cells + (cells << case["blowup"])),
                "flops": _lde_muls(case["log_h"], case["width"], case["blowup"])}
    if kind == "pcs":
        return _commit(field, case["p2"], case["log_h"], case["width"], case["blowup"])
    if kind == "mmcs":
        by, fl, heights = 0, 0, {}
        for h, w in _mmcs_shapes(case):
            by += es * h * w
            heights[h] = heights.get(h, 0) + w
        top, out = max(heights), 8 if case["p2"] == 16 else 4
        perms = top - 1 + sum(h * (_sponge_perms(w) + (h != top)) for h, w in heights.items())
        return {"bytes": by + 2 * top * out * es, "flops": perms * _perm_muls(field, case["p2"])}
    if kind == "fri":
        return _fri(case["log_n"], case["log_final"], case["queries"])
    if kind == "job":
        a = _commit(field, 16, case["log_h"], case["width"], 1)
        b = _fri(case["log_h"] + 1, case["log_final"], case["queries"])
        reduce_muls = 4 * case["width"] << (case["log_h"] + 1)
        return {"bytes": a["bytes"] + b["bytes"], "flops": a["flops"] + b["flops"] + reduce_muls}
    tot = {"bytes": 0, "flops": 0}
    for h, w in _batch_shapes(case):
        c = _commit(field, 16, h.bit_length() - 1, w, 1)
        tot = {k: tot[k] + c[k] for k in tot}
    return tot


def exact(case, seed):
    """Every output is an integer that has to be equal, so no 64-bit value stands in for it."""
    return None
