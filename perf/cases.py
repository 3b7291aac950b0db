"""The work that the performance of this framework is judged on.

Each case is one kind of call a prover makes, at sizes from the smallest to the
largest that the repository's benchmark and tests use:

  commit        TwoAdicFriPcs.commit of device-resident traces (batched coset
                LDE + mixed-height Poseidon2 tree), the prover data released
                after it, as a prover does once a chunk is proven
  commit_read   the same, then the committed rows of every matrix read on its
                trace domain into device buffers (the quotient step's reads)
  commit_host   commit of traces in pinned host memory
  serve         many small commits in flight through CommitServer
  lde           Radix2DitParallel.coset_lde_batch_bitrev, device to device
  fri           the FRI commit phase of a device-resident EF4 codeword
  open          TwoAdicFriPcs.open of a resident commitment at zeta and zeta*w
  quotient      compute_quotient_values of one chip over resident LDEs

Inputs are uniform field elements in Montgomery form: traces, LDEs and
codewords of a prover are indistinguishable from these for every kernel here
(no path depends on the values).  All outputs are whole numbers (field
elements), so they are equal or wrong, and exact() has nothing to add.
"""
import random

import numpy as np
import torch

from pico_b200 import (CommitServer, GpuContext, Radix2DitParallel, TwoAdicDomain, TwoAdicFriPcs, fields,
                       new_challenger)
from pico_b200.quotient import ConstraintBuilder, compute_quotient_values

_CONTEXT = None


def _context():
    """One device context per process, as a prover keeps one."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = GpuContext(0)
    return _CONTEXT


def listed():
    return [
        # one tiny chip: launches, allocations and the host path are all of it
        dict(name="commit-tiny-bb", kind="commit", field="bb", blowup=1, mats=2, log_lo=5, log_hi=8, w_lo=5, w_hi=40,
             shape_seed=11, log_cells=0),
        # one mid-size trace: a single chip of a recursion program
        dict(name="commit-2^16x64-kb", kind="commit", field="kb", blowup=1, mats=1, log_lo=16, log_hi=16, w_lo=64,
             w_hi=64, shape_seed=1, log_cells=0),
        # a RISC-V shard: 32 chips of very different heights, 2^30 trace cells
        dict(name="commit-uneven-2^30-kb", kind="commit", field="kb", blowup=1, mats=32, log_lo=10, log_hi=22, w_lo=8,
             w_hi=400, shape_seed=15, log_cells=30),
        # a recursion batch: 48 BabyBear traces at blowup 4
        dict(name="commit-recursion-48-bb", kind="commit", field="bb", blowup=2, mats=48, log_lo=8, log_hi=20, w_lo=4,
             w_hi=600, shape_seed=3, log_cells=0),
        # a small shard whose committed rows the quotient step then reads
        dict(name="commit-read-2^24-kb", kind="commit_read", field="kb", blowup=1, mats=12, log_lo=8, log_hi=17,
             w_lo=3, w_hi=300, shape_seed=4, log_cells=24),
        # traces generated on the host: copies and compute overlap
        dict(name="commit-host-2^26-kb", kind="commit_host", field="kb", blowup=1, mats=10, log_lo=10, log_hi=19,
             w_lo=8, w_hi=400, shape_seed=5, log_cells=26),
        # proving service: requests of about 20 small traces, several in flight
        dict(name="serve-small-16-kb", kind="serve", field="kb", blowup=1, requests=16, mats=20, log_lo=8, log_hi=13,
             w_lo=8, w_hi=64, shape_seed=6),
        # one tall trace, extended only
        dict(name="lde-2^20x70-kb", kind="lde", field="kb", blowup=1, log_n=20, width=70),
        # one short wide trace, blowup 4
        dict(name="lde-2^11x333-bb", kind="lde", field="bb", blowup=2, log_n=11, width=333),
        # the FRI commit phase of the tallest codeword of a shard
        dict(name="fri-2^23-kb", kind="fri", field="kb", blowup=1, log_n=23),
        # opening a mid-size shard: 84 queries, 16 proof-of-work bits
        dict(name="open-uneven-2^26-kb", kind="open", field="kb", blowup=1, mats=16, log_lo=8, log_hi=19, w_lo=8,
             w_hi=400, shape_seed=7, log_cells=26),
        # a chip's constraints over its quotient domain
        dict(name="quotient-2^19-bb", kind="quotient", field="bb", blowup=1, log_n=19, width=33, degree=1),
    ]


def _log_int(rng, lo, hi):
    """An integer between lo and hi, uniform over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["commit", "commit", "commit", "commit_read", "commit_host", "serve", "lde", "lde", "fri",
                       "open", "quotient"])
    case = dict(kind=kind, field=rng.choice(["kb", "bb"]), blowup=rng.choice([1, 1, 2]))
    if kind in ("commit", "commit_read", "commit_host", "open"):
        log_lo = rng.randint(4, 10)
        case.update(mats=_log_int(rng, 1, 70), log_lo=log_lo, log_hi=rng.randint(log_lo + 1, 19), w_lo=rng.randint(1, 9),
                    w_hi=_log_int(rng, 10, 500), shape_seed=rng.randrange(1 << 20),
                    log_cells=rng.randint(14, 27 if kind != "commit_host" else 25))
    elif kind == "serve":
        log_lo = rng.randint(5, 9)
        case.update(requests=_log_int(rng, 2, 32), mats=_log_int(rng, 1, 40), log_lo=log_lo,
                    log_hi=rng.randint(log_lo, 13), w_lo=rng.randint(1, 9), w_hi=_log_int(rng, 10, 70),
                    shape_seed=rng.randrange(1 << 20))
    elif kind == "lde":
        log_n = rng.randint(3, 22)
        case.update(log_n=log_n, width=_log_int(rng, 1, max(2, min(600, 1 << (27 - log_n)))))
    elif kind == "fri":
        case.update(log_n=rng.randint(6, 22))
    else:
        case.update(log_n=rng.randint(6, 19), width=_log_int(rng, 8, 100), degree=1)
    return case


def _shapes(case, salt=0):
    """(log height, width) per matrix: log heights and widths uniform on their
    ranges; with log_cells, widths scaled so that the cells come to about
    2^log_cells."""
    rng = random.Random(case["shape_seed"] * 1000003 + salt)
    shapes = [(rng.randint(case["log_lo"], case["log_hi"]), rng.randint(case["w_lo"], case["w_hi"]))
              for _ in range(case["mats"])]
    if case.get("log_cells"):
        scale = 2.0 ** case["log_cells"] / sum(w << h for h, w in shapes)
        shapes = [(h, max(1, min(2000, round(w * scale)))) for h, w in shapes]
    return shapes


def _random(case, gen, *shape):
    """Uniform field elements (Montgomery-form words) on the GPU."""
    p = fields.P[fields.field_id(case["field"])]
    return torch.randint(0, p, shape, generator=gen, device="cuda", dtype=torch.int32)


def _word4(case, gen):
    return _random(case, gen, 4).cpu().numpy().view(np.uint32)


def _points(case, shapes, gen):
    """Every trace is opened at zeta and at zeta times its subgroup's generator."""
    f = fields.field_id(case["field"])
    zeta = _word4(case, gen)
    points = []
    for h, _ in shapes:
        w = fields.two_adic_generator(f, h)
        nxt = [fields.monty(f, fields.unmonty(f, int(v)) * w) for v in zeta]
        points.append(np.stack([zeta, np.array(nxt, dtype=np.uint32)]))
    return points


def _program(case):
    """A chip's constraints: products wired over the main columns, transitions,
    booleans, first and last row, and a running sum in a permutation column."""
    rng = random.Random(9)
    w = case["width"]
    b = ConstraintBuilder()

    def col(nxt=False):
        return b.main(rng.randrange(w), nxt)

    for _ in range(16):
        b.assert_zero(col() * col() - col())
    for _ in range(8):
        b.when_transition().assert_eq(col(True), col() + col())
    for _ in range(4):
        x = col()
        b.assert_zero(x * (x - 1))
    b.when_first_row().assert_eq(b.main(0), b.public(0))
    b.when_last_row().assert_eq(b.main(1), b.public(1))
    z, z_next = b.permutation(0), b.permutation(0, True)
    b.when_transition().assert_zero((z_next - z) * (b.challenge(0) + b.main(0) + b.challenge(1) * b.main(1)) - b.main(2))
    b.when_first_row().assert_zero(z - b.regional_cumulative_sum())
    return b.program(case["field"])


def prepare(case, seed):
    ctx = _context()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    state = dict(kind=kind, case=case)
    pcs = TwoAdicFriPcs(ctx, case["field"], case["blowup"])
    state["pcs"] = pcs
    if kind in ("commit", "commit_read", "commit_host", "open"):
        shapes = _shapes(case)
        traces = [_random(case, gen, 1 << h, w) for h, w in shapes]
        if kind == "commit_host":
            traces = [t.cpu().pin_memory().numpy().view(np.uint32) for t in traces]
        state["batch"] = [(TwoAdicDomain(h), t) for (h, _), t in zip(shapes, traces)]
        if kind == "commit_read":
            state["rows"] = [torch.empty_like(t) for t in traces]
        if kind == "open":
            torch.cuda.synchronize()
            _, data = pcs.commit(state.pop("batch"))
            state["rounds"] = [(data, _points(case, shapes, gen))]
    elif kind == "serve":
        state["server"] = CommitServer(ctx)
        state["requests"] = [[_random(case, gen, 1 << h, w) for h, w in _shapes(case, i)]
                             for i in range(case["requests"])]
    elif kind == "lde":
        state["dft"] = Radix2DitParallel(ctx, case["field"])
        state["mat"] = _random(case, gen, 1 << case["log_n"], case["width"])
        state["out"] = torch.empty((1 << (case["log_n"] + case["blowup"]), case["width"]), dtype=torch.int32,
                                   device="cuda")
        state["shift"] = fields.lde_shift(fields.field_id(case["field"]))
    elif kind == "fri":
        # a low-degree codeword, as the opening feeds it
        base = _random(case, gen, 1 << (case["log_n"] - case["blowup"]), 4)
        state["codeword"] = torch.empty((1 << case["log_n"], 4), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        Radix2DitParallel(ctx, case["field"]).coset_lde_batch_bitrev(
            base, case["blowup"], fields.lde_shift(fields.field_id(case["field"])), out=state["codeword"])
    elif kind == "quotient":
        n = 1 << case["log_n"]
        main, perm = _random(case, gen, n, case["width"]), _random(case, gen, n, 1, 4)
        torch.cuda.synchronize()
        _, data = pcs.commit([(TwoAdicDomain(case["log_n"]), main), (TwoAdicDomain(case["log_n"]), perm)])
        state.update(ctx=ctx, data=data, program=_program(case), public=_word4(case, gen)[:2],
                     challenges=np.stack([_word4(case, gen), _word4(case, gen)]), regional=_word4(case, gen),
                     alpha=_word4(case, gen),
                     out=torch.empty((n << case["degree"], 4), dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return state


def run(state):
    kind, case, pcs = state["kind"], state["case"], state["pcs"]
    if kind in ("commit", "commit_host"):
        root, data = pcs.commit(state["batch"])
        data.release()
        return root
    if kind == "commit_read":
        root, data = pcs.commit(state["batch"])
        for i, out in enumerate(state["rows"]):
            data.evaluations_on_domain(i, state["batch"][i][0].log_n, out=out)
        data.release()
        return {"root": root, "rows": state["rows"]}
    if kind == "serve":
        server = state["server"]
        requests = [server.submit(case["field"], traces, case["blowup"]) for traces in state["requests"]]
        roots = []
        for r in requests:
            root, data = r.wait()
            data.release()
            r.free()
            roots.append(root)
        return roots
    if kind == "lde":
        return state["dft"].coset_lde_batch_bitrev(state["mat"], case["blowup"], state["shift"], out=state["out"])
    if kind == "fri":
        res = pcs.fri_commit_phase(state["codeword"])
        return {"roots": res.roots, "betas": res.betas, "final": res.final_poly}
    if kind == "open":
        proof = pcs.open(state["rounds"], new_challenger())
        return {k: v for k, v in proof.items() if k != "stats"}
    return compute_quotient_values(state["ctx"], state["program"], case["log_n"], case["degree"], (state["data"], 0),
                                   permutation=(state["data"], 1), public_values=state["public"],
                                   perm_challenges=state["challenges"], regional_sum=state["regional"],
                                   alpha=state["alpha"], out=state["out"])


def exact(case, seed):
    """Every output is a field element: equal or wrong, with nothing in between."""
    return None


# Field products of one Poseidon2-16 permutation outside its linear layers'
# small constants: two per x^3 (KoalaBear, 148 S-boxes), four per x^7
# (BabyBear, 141).
_SBOX_PRODUCTS = {"kb": 148 * 2, "bb": 141 * 4}


def _commit_work(case, shapes):
    """Bytes: every trace read, every LDE and digest layer written once.  Products: the
    radix-2 butterflies of an inverse and 2^b forward transforms, and the S-boxes of the row and node hashes."""
    b = case["blowup"]
    cells = sum(w << h for h, w in shapes)
    top = max(h for h, _ in shapes) + b
    widths = {}
    for h, w in shapes:
        widths[h] = widths.get(h, 0) + w
    perms = (1 << top) - 1 + sum(((w + 7) // 8) << (h + b) for h, w in widths.items())
    perms += sum(1 << (h + b) for h in widths if h + b != top)
    butterflies = sum((w << h) * h // 2 for h, w in shapes) * (1 + (1 << b))
    return 4 * cells * (1 + (1 << b)) + (32 << (top + 1)), butterflies + perms * _SBOX_PRODUCTS[case["field"]]


def work(case):
    """Bytes read and written once, and field products (counted as flops), of one pass."""
    kind, b = case["kind"], case["blowup"]
    if kind in ("commit", "commit_host", "commit_read"):
        shapes = _shapes(case)
        nbytes, flops = _commit_work(case, shapes)
        if kind == "commit_read":
            nbytes += 8 * sum(w << h for h, w in shapes)
    elif kind == "serve":
        parts = [_commit_work(case, _shapes(case, i)) for i in range(case["requests"])]
        nbytes, flops = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "lde":
        cells = case["width"] << case["log_n"]
        nbytes, flops = 4 * cells * (1 + (1 << b)), cells * case["log_n"] // 2 * (1 + (1 << b)) + cells
    elif kind == "fri":
        # per round a leaf per two elements, its tree, and the fold: halving lengths
        n = 1 << case["log_n"]
        nbytes, flops = 16 * 2 * n + 2 * 32 * n, 2 * n * _SBOX_PRODUCTS[case["field"]] + n * 12
    elif kind == "open":
        # the low coset read for the values and once more for the reduction; the commit phase of the tallest height
        shapes = _shapes(case)
        cells = sum(w << h for h, w in shapes)
        n = 1 << (max(h for h, _ in shapes) + b)
        nbytes = 8 * cells + 16 * 2 * n + 2 * 32 * n
        flops = cells * 8 * 2 + 2 * n * _SBOX_PRODUCTS[case["field"]]
    else:
        points = 1 << (case["log_n"] + case["degree"])
        nbytes, flops = points * 4 * (case["width"] + 4 + 4), points * 200
    return {"bytes": nbytes, "flops": flops}
