"""The work that users of this framework have it do, as cases to be timed.

A case is a dict of plain values; ``kind`` names the call:

index     GroupIndexer.indices: positions -> column indices (a feature
          extraction on its own, from one self-play batch to a data set).
build     MatrixCSR.from_positions and the Jacobi diagonal: what every fit
          and every training run does first with new positions.
product   A x and A'y on a kept matrix: the two products of a caller's own
          solver or evaluation loop.
csr       The same on a matrix of the caller's own indices
          (MatrixCSR.from_indices), in the shapes of the reference's matrix
          benchmark (32 entries per row, rows / 16 columns).
fit       fit_weights on host positions and scores: FitWeights as the
          reference's training loop calls it (FP64, a fixed number of
          iterations), or a large data set in mixed precision to 1e-8.
stages    fit_weights_batched: the fits of several empty-count stages in one
          call, likewise.
train     Trainer.epoch: one epoch of the differentiable evaluator.
score     MultiStageScoreEstimator.eval: batch evaluation of positions with
          fitted weights.

Positions are random-play positions (generate_positions), targets come from
seeded weights plus noise (generate_targets), as in the repository's own
benchmark.  ``exact`` restates the indexers and the products in torch.
"""
import math

import numpy as np
import torch

import cassandra_b200 as cb
from cassandra_b200.evaluator import PatternEvaluator, Trainer

MASKS = {5: cb.PATTERNS_5, 8: cb.PATTERNS_8}


# --------------------------------------------------------------------------
# Cases
# --------------------------------------------------------------------------
def listed():
    return [
        # one self-play batch: a call whose launch and host work count
        {"name": "index_batch", "kind": "index", "masks": 5, "mode": "reference", "rows": 1000},
        # a data set in the unreduced layout
        {"name": "index_dataset", "kind": "index", "masks": 8, "mode": "expanded", "rows": 6_000_000},
        # from_positions as it stands: both layouts, the reference's columns
        {"name": "build_default", "kind": "build", "masks": 8, "mode": "reference", "layouts": "default",
         "rows": 1_000_003},
        # the layout that large mixed fits and training use
        {"name": "build_blocked", "kind": "build", "masks": 8, "mode": "expanded", "layouts": "blocked",
         "rows": 5_000_000},
        # the products of a large fit, FP32
        {"name": "product_large", "kind": "product", "masks": 8, "mode": "expanded", "rows": 10_000_000,
         "dtype": "float32"},
        # the products of a medium-sized fit, FP64, rows that fill no block
        {"name": "product_fp64", "kind": "product", "masks": 8, "mode": "reference", "rows": 1_500_001,
         "dtype": "float64"},
        # the reference's matrix benchmark at its largest size
        {"name": "csr_large", "kind": "csr", "rows": 2_000_000, "k": 32, "dtype": "float32"},
        # FitWeights with the defaults on one stage of a training loop
        {"name": "fit_default", "kind": "fit", "masks": 5, "mode": "reference", "precision": "fp64",
         "rows": 100_000, "tol": 0.0, "iterations": 10},
        # a large data set in mixed precision, solved to the end
        {"name": "fit_large", "kind": "fit", "masks": 8, "mode": "expanded", "precision": "mixed",
         "rows": 4_000_000, "tol": 1e-8, "iterations": 5000},
        # several stages of uneven size, solved to the end
        {"name": "stages", "kind": "stages", "masks": 8, "mode": "expanded", "precision": "mixed",
         "rows": 2_400_000, "problems": 8, "tol": 1e-8, "iterations": 20000},
        # one epoch of minibatch training
        {"name": "train_epoch", "kind": "train", "masks": 8, "mode": "expanded", "rows": 1_000_000, "batch": 65536},
        # scoring a data set with a fitted estimator
        {"name": "score_dataset", "kind": "score", "masks": 5, "rows": 3_000_000, "stage_size": 5},
    ]


def _spread(rng, lo, hi):
    """A size between lo and hi, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["index", "build", "product", "csr", "fit", "stages", "train", "score"])
    masks, mode = rng.choice([5, 8]), rng.choice(["reference", "expanded"])
    if kind == "index":
        return {"kind": kind, "masks": masks, "mode": mode, "rows": _spread(rng, 1000, 6_000_000)}
    if kind == "build":
        layouts = rng.choice(["default", "blocked"])
        return {"kind": kind, "masks": masks, "mode": mode, "layouts": layouts,
                "rows": _spread(rng, 20_000, 1_000_000 if layouts == "default" else 5_000_000)}
    if kind == "product":
        return {"kind": kind, "masks": masks, "mode": mode, "rows": _spread(rng, 20_000, 5_000_000),
                "dtype": rng.choice(["float32", "float64"])}
    if kind == "csr":
        return {"kind": kind, "rows": _spread(rng, 1000, 2_000_000), "k": 32,
                "dtype": rng.choice(["float32", "float64"])}
    if kind == "fit" and rng.random() < 0.5:
        return {"kind": kind, "masks": masks, "mode": mode, "precision": "fp64",
                "rows": _spread(rng, 20_000, 1_000_000), "tol": 0.0, "iterations": rng.randint(10, 30)}
    if kind == "fit":
        return {"kind": kind, "masks": masks, "mode": mode, "precision": "mixed",
                "rows": _spread(rng, 500_000, 4_000_000), "tol": 1e-8, "iterations": 5000}
    if kind == "stages" and rng.random() < 0.5:
        problems = rng.randint(10, 60)
        return {"kind": kind, "masks": masks, "mode": mode, "precision": "fp64",
                "rows": problems * _spread(rng, 10_000, 40_000), "problems": problems, "tol": 0.0, "iterations": 10}
    if kind == "stages":
        problems = rng.randint(3, 8)
        return {"kind": kind, "masks": masks, "mode": mode, "precision": "mixed",
                "rows": problems * _spread(rng, 300_000, 400_000), "problems": problems, "tol": 1e-8,
                "iterations": 20000}
    if kind == "train":
        return {"kind": kind, "masks": masks, "mode": mode, "rows": _spread(rng, 100_000, 1_000_000),
                "batch": 16384 * rng.choice([1, 2, 4])}
    return {"kind": kind, "masks": masks, "rows": _spread(rng, 1000, 3_000_000), "stage_size": rng.choice([1, 5, 10])}


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------
def _positions(seed, rows):
    return cb.generate_positions(seed, rows, 20, 40)


def _stage_sizes(seed, rows, problems):
    """Uneven stage sizes that add up to rows (log-uniform over a factor of 10)."""
    w = np.exp(np.random.RandomState(seed % (1 << 32)).uniform(0, math.log(10), problems))
    cut = np.floor(np.cumsum(w) / w.sum() * rows + 0.5).astype(np.int64)
    cut[-1] = rows
    return np.diff(cut, prepend=0)


def _targets(g, pos, seed):
    return cb.generate_targets(cb.MatrixCSR.from_positions(g, pos, "blocked"), seed)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _csr_indices(case, seed):
    cols = max(1, case["rows"] // 16)
    idx = torch.randint(cols, (case["rows"], case["k"]), generator=_gen(seed), device="cuda", dtype=torch.int32)
    return idx, cols


def _vectors(case, seed, cols):
    dt = getattr(torch, case["dtype"])
    g = _gen(seed + 1)
    return (torch.randn(cols, generator=g, device="cuda", dtype=dt),
            torch.randn(case["rows"], generator=g, device="cuda", dtype=dt))


def _score_weights(case, seed, cols):
    return torch.randn((cb.estimator_stages(case["stage_size"]), cols), generator=_gen(seed + 1), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "csr":
        idx, cols = _csr_indices(case, seed)
        x, y = _vectors(case, seed, cols)
        return {"kind": kind, "a": cb.MatrixCSR.from_indices(idx, cols), "x": x, "y": y}
    masks = MASKS[case["masks"]]
    pos = _positions(seed, case["rows"])
    if kind == "score":
        cols = cb.GroupIndexer(masks, "reference").index_space_size
        est = cb.MultiStageScoreEstimator(masks, case["stage_size"], _score_weights(case, seed, cols))
        return {"kind": kind, "est": est, "pos": pos}
    g = cb.GroupIndexer(masks, case["mode"])
    if kind == "index":
        return {"kind": kind, "g": g, "pos": pos}
    if kind == "build":
        return {"kind": kind, "g": g, "pos": pos,
                "layouts": None if case["layouts"] == "default" else case["layouts"]}
    if kind == "product":
        x, y = _vectors(case, seed, g.index_space_size)
        return {"kind": kind, "a": cb.MatrixCSR.from_positions(g, pos, "blocked"), "x": x, "y": y}
    b = _targets(g, pos, seed)
    if kind == "fit":
        return {"kind": kind, "masks": masks, "pos": pos.cpu().numpy().view(np.uint64),
                "scores": b.float().cpu().numpy(), "mode": case["mode"], "precision": case["precision"],
                "tol": case["tol"], "iterations": case["iterations"]}
    if kind == "stages":
        return {"kind": kind, "g": g, "pos": pos, "scores": b, "precision": case["precision"], "tol": case["tol"],
                "sizes": _stage_sizes(seed, case["rows"], case["problems"]), "iterations": case["iterations"]}
    return {"kind": kind, "trainer": Trainer(PatternEvaluator(masks, pos, case["mode"]), b, batch=case["batch"])}


def run(s):
    kind = s["kind"]
    if kind == "index":
        return s["g"].indices(s["pos"])
    if kind == "build":
        a = cb.MatrixCSR.from_positions(s["g"], s["pos"], s["layouts"])
        out = {"jacobi": cb.jacobi_preconditioner_of_ata(a)}
        if "rows" in a.layouts():
            out["col_ptr"], out["row_idx"] = a.transposed()
        return out
    if kind in ("product", "csr"):
        return {"ax": s["a"] @ s["x"], "aty": s["a"].rmatvec(s["y"])}
    if kind == "fit":
        return cb.fit_weights(s["masks"], s["pos"], s["scores"], mode=s["mode"], precision=s["precision"],
                              tol=s["tol"], max_iterations=s["iterations"])[0]
    if kind == "stages":
        w, _, _ = cb.fit_weights_batched(s["g"], s["pos"], s["scores"], s["sizes"], precision=s["precision"],
                                         tol=s["tol"], max_iterations=s["iterations"])
        return w.float()  # the estimators and their files hold FP32 weights
    if kind == "train":
        loss = s["trainer"].epoch()
        return {"loss": loss, "w": s["trainer"].model.weight.detach().clone()}
    return s["est"].eval(s["pos"])


# --------------------------------------------------------------------------
# What a pass cannot do without
# --------------------------------------------------------------------------
_NNZ = {(5, "reference"): 22, (8, "reference"): 34, (5, "expanded"): 40, (8, "expanded"): 64}
_COLS = {(5, "reference"): 105_543, (8, "reference"): 113_319, (5, "expanded"): 150_903, (8, "expanded"): 166_212}


def work(case):
    kind, n = case["kind"], case["rows"]
    if kind == "csr":
        es, cols = (4 if case["dtype"] == "float32" else 8), max(1, n // 16)
        return {"bytes": 2 * (4 * n * case["k"] + es * (n + cols)), "flops": 2 * n * case["k"]}
    key = (case["masks"], case.get("mode", "reference"))
    k, cols = _NNZ[key], _COLS[key]
    if kind == "index":
        return {"bytes": 16 * n + 4 * n * k, "flops": 0}
    if kind == "score":
        # the position and the score; the table entries are gathered through the caches
        return {"bytes": 20 * n, "flops": n * k}
    # one pass over the index stream in each direction (16-bit columns a
    # row's way, 32-bit column and row the other way)
    products = 6 * n * k
    if kind == "build":
        rows = 8 * n * k if case["layouts"] == "default" else 0
        return {"bytes": 16 * n + products + rows + 8 * cols, "flops": n * k}
    if kind == "product":
        es = 4 if case["dtype"] == "float32" else 8
        return {"bytes": products + 2 * es * (n + cols), "flops": 2 * n * k}
    if kind == "train":
        steps = -(-n // case["batch"])
        return {"bytes": products + 4 * n + 24 * cols * steps, "flops": 2 * n * k + 12 * cols * steps}
    # a solve to 1e-8 takes about 80 iterations at 4M rows and more with fewer
    problems, it = case.get("problems", 1), case["iterations"] if case["tol"] == 0 else 80
    es = 4 if case["precision"] == "mixed" else 8
    vec = 8 * es * cols * problems
    return {"bytes": 20 * n + products + it * (products + 2 * es * n + vec), "flops": it * (2 * n * k + 8 * cols * problems)}


# --------------------------------------------------------------------------
# The same in 64 bits, in plain torch
# --------------------------------------------------------------------------
# Board symmetries as maps of squares (bit b: x = b & 7, y = b >> 3).
_FLIP = {"C": lambda x, y: (7 - y, 7 - x), "D": lambda x, y: (y, x), "H": lambda x, y: (7 - x, y),
         "V": lambda x, y: (x, 7 - y)}
_LOWER_HALF, _STRICT_LOWER, _DIAGONAL = 0x00000000FFFFFFFF, 0x0080C0E0F0F8FCFE, 0x8040201008040201
_ALL = ["", "C", "D", "H", "V", "CH", "DH", "VH"]


def _moved(b, g):
    """The square that the flips g, applied in order, move b onto."""
    x, y = b & 7, b >> 3
    for f in g:
        x, y = _FLIP[f](x, y)
    return 8 * y + x


def _squares(mask):
    return [b for b in range(64) if mask >> b & 1]


def _flipped(mask, g):
    return sum(1 << _moved(b, g) for b in _squares(mask))


def _sources(mask, g):
    """The squares whose cells are the ternary digits of `mask` on the position flipped by g."""
    back = {_moved(b, g): b for b in range(64)}
    return [back[s] for s in _squares(mask)]


def _digits(cells, squares):
    out = torch.zeros(cells.shape[1], dtype=torch.int64, device=cells.device)
    for s in reversed(squares):
        out = out * 3 + cells[s]
    return out


def _pair(a, b, half):
    lo, hi = torch.minimum(a, b), torch.maximum(a, b)
    return lo * half + hi - lo * (lo + 1) // 2


def _orbit_table(mask, orbit, device):
    """Dense index of every configuration of `mask`: orbits numbered by their
    first member, player bits major and opponent bits minor."""
    sq = _squares(mask)
    n = len(sq)
    e = torch.arange(3 ** n, device=device)
    d = [e // 3 ** i % 3 for i in range(n)]
    cells = torch.zeros((64, 3 ** n), dtype=torch.int64, device=device)
    for i, s in enumerate(sq):
        cells[s] = d[i]
    first = None
    for g in orbit:
        src = _sources(mask, g)
        rank = sum(((cells[s] == 1).long() << (n + i)) + ((cells[s] == 2).long() << i) for i, s in enumerate(src))
        first = rank if first is None else torch.minimum(first, rank)
    return torch.unique(first, return_inverse=True)[1]


def _columns(masks, mode, pos):
    """The columns of every row, one int64 vector per slot, and their number."""
    cells = torch.empty((64, pos.shape[0]), dtype=torch.int8, device=pos.device)
    for b in range(64):
        cells[b] = ((pos[:, 0] >> b) & 1) + 2 * ((pos[:, 1] >> b) & 1)
    out, off = [], 0
    for m in masks:
        v, h, d, c = (_flipped(m, f) == m for f in "VHDC")
        if mode == "expanded" or not (v or h or d or c):
            out += [off + _digits(cells, _sources(m, g)) for g in _ALL]
            off += 3 ** len(_squares(m))
        elif (v and h) or (d and c):
            if v and h and d and c:
                orbit, inst = ["", "C", "D", "H", "V", "HC", "HD", "HV"], [""]
            elif v and h:
                orbit, inst = ["", "V", "H", "VH"], ["", "D"]
            else:
                orbit, inst = ["", "D", "C", "DC"], ["", "V"]
            table = _orbit_table(m, orbit, pos.device)
            out += [off + table[_digits(cells, _sources(m, g))] for g in inst]
            off += int(table.max()) + 1
        elif v or h:
            m = m if v else _flipped(m, "D")
            half = m & _LOWER_HALF
            hs = 3 ** len(_squares(half))
            out += [off + _pair(_digits(cells, _sources(half, g)), _digits(cells, _sources(half, g + "V")), hs)
                    for g in ("", "C", "D", "H")]
            off += hs * (hs + 1) // 2
        else:
            m = m if d else _flipped(m, "V")
            half, line = m & _STRICT_LOWER, m & _DIAGONAL
            hs, ds = 3 ** len(_squares(half)), 3 ** len(_squares(line))
            out += [off + _pair(_digits(cells, _sources(half, g)), _digits(cells, _sources(half, g + "D")), hs) * ds
                    + _digits(cells, _sources(line, g)) for g in ("", "C", "H", "V")]
            off += ds * hs * (hs + 1) // 2
    return out, off


def _ax(slots, x):
    y = torch.zeros(slots[0].numel(), dtype=torch.float64, device=x.device)
    for c in slots:
        y += x[c]
    return y


def _aty(slots, y, cols):
    x = torch.zeros(cols, dtype=torch.float64, device=y.device)
    for c in slots:
        x.index_add_(0, c, y)
    return x


def _diag(slots, cols):
    """diag(A'A): a row that holds a column m times adds m^2."""
    dg = torch.zeros(cols, dtype=torch.float64, device=slots[0].device)
    for c in slots:
        same = sum((c == other).double() for other in slots)
        dg.index_add_(0, c, same)
    return dg


def _pcg(slots, cols, b, iterations):
    """Jacobi-PCG on A'A x = A'b from x = 0."""
    d = 1 / _diag(slots, cols)
    d[~torch.isfinite(d)] = 1.0
    x = torch.zeros(cols, dtype=torch.float64, device=b.device)
    r = _aty(slots, b, cols)
    z = d * r
    p, rz = z.clone(), torch.dot(r, z)
    for _ in range(iterations):
        ap = _ax(slots, p)
        alpha = rz / torch.dot(ap, ap)
        x += alpha * p
        r -= alpha * _aty(slots, ap, cols)
        z = d * r
        rz, old = torch.dot(r, z), rz
        p = z + (rz / old) * p
    return x


def _epoch(slots, cols, target, batch, lr=1e-2, l2=1e-4, delta=4.0, betas=(0.9, 0.999), eps=1e-8):
    """The first epoch of Trainer's defaults from zero weights."""
    rows = target.numel()
    w, m, v = (torch.zeros(cols, dtype=torch.float64, device=target.device) for _ in range(3))
    starts = list(range(0, rows, batch))
    order = torch.randperm(len(starts), generator=torch.Generator().manual_seed(0)).tolist()
    total = 0.0
    for t, i in enumerate(order, 1):
        r0, r1 = starts[i], min(starts[i] + batch, rows)
        part = [c[r0:r1] for c in slots]
        d = _ax(part, w) - target[r0:r1]
        total += float(torch.where(d.abs() < delta, 0.5 * d * d, delta * (d.abs() - 0.5 * delta)).mean() + l2 * w.dot(w))
        g = _aty(part, d.clamp(-delta, delta) / (r1 - r0), cols) + 2 * l2 * w
        m = betas[0] * m + (1 - betas[0]) * g
        v = betas[1] * v + (1 - betas[1]) * g * g
        w = w - lr / (1 - betas[0] ** t) * m / (v.sqrt() / math.sqrt(1 - betas[1] ** t) + eps)
    return {"loss": total / len(starts), "w": w}


def exact(case, seed):
    kind = case["kind"]
    if kind == "index":
        return None  # whole numbers
    if case.get("tol", 0) > 0:
        return None  # where in the last decade a solve to a tolerance stops is no value of the inputs
    if kind == "csr":
        idx, cols = _csr_indices(case, seed)
        x, y = (t.double() for t in _vectors(case, seed, cols))
        slots = [idx[:, j].long() for j in range(case["k"])]
        return {"ax": _ax(slots, x), "aty": _aty(slots, y, cols)}
    masks = MASKS[case["masks"]]
    pos = _positions(seed, case["rows"])
    mode = case.get("mode", "reference")
    if kind == "score":
        slots, cols = _columns(masks, mode, pos)
        stage = sum(((pos[:, 0] | pos[:, 1]) >> b) & 1 for b in range(64))
        stage = (64 - stage) // case["stage_size"]
        w = _score_weights(case, seed, cols).double().reshape(-1)
        return _ax([stage * cols + c for c in slots], w)
    slots, cols = _columns(masks, mode, pos)
    if kind == "build":
        out = {"jacobi": 1 / _diag(slots, cols)}
        return out if case["layouts"] == "blocked" else out | {"col_ptr": None, "row_idx": None}
    if kind == "product":
        x, y = (t.double() for t in _vectors(case, seed, cols))
        return {"ax": _ax(slots, x), "aty": _aty(slots, y, cols)}
    b = _targets(cb.GroupIndexer(masks, mode), pos, seed)
    if kind == "fit":
        return _pcg(slots, cols, b, case["iterations"])
    if kind == "train":
        return _epoch(slots, cols, b, case["batch"])
    out, row = [], 0
    for n in _stage_sizes(seed, case["rows"], case["problems"]).tolist():
        out.append(_pcg([c[row:row + n] for c in slots], cols, b[row:row + n], case["iterations"]))
        row += n
    return torch.stack(out)
