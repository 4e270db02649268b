"""The work this package does for its users, as cases that can be timed and checked.

``listed()`` names the representative cases, ``draw(rng)`` gives more of the same
ranges, ``prepare``/``run`` make a case's inputs and take them once through the public
entry points, ``work`` counts what a pass cannot do without, and ``exact`` evaluates the
same quantity in float64 with plain torch.

Families (``op``):

* ``mul``, ``fma``, ``inplace``: the truncated free-tensor product of batches of pairs;
* ``exp``, ``fmexp``, ``log``, ``antipode``, ``adjoint``: the other dense operations;
* ``lie_exp`` (Lie coordinates -> signature) and ``log_lie`` (signature -> log-signature
  coordinates): the two directions between the Lie algebra and the group;
* ``sig`` / ``sig_grad``: batched signatures of streams, and their gradient;
* ``queries``: log-signatures of many intervals of one stream, from its dyadic cache.
"""
import math

import numpy as np
import torch

from roughpy_b200 import compute as rpc
from roughpy_b200 import signatures as sigs
from roughpy_b200 import streams

DTYPES = {"f32": torch.float32, "f64": torch.float64}
PAIR_OPS = ("mul", "fma", "inplace", "fmexp", "adjoint")
LIE_OPS = ("lie_exp", "log_lie")
MAX_WORDS = 1024 * 299593      # words of one operand of the largest listed product
MAX_LIE_TENSOR = 10000         # tensor size up to which Lie maps are drawn


def listed():
    return [
        # one pair of small tensors: what an interactive user or a per-step loop calls,
        # bound by the latency of one call
        {"name": "mul_pair_w3d4_f64", "op": "mul", "width": 3, "depth": 4, "batch": 1,
         "dtype": "f64"},
        # the free-tensor multiply-add sweep: wide and deep, the largest batch of all
        {"name": "fma_w8d6_f32", "op": "fma", "width": 8, "depth": 6, "batch": 1024,
         "dtype": "f32"},
        # the same sweep at its narrowest and deepest (time plus one channel)
        {"name": "fma_w2d12_f32", "op": "fma", "width": 2, "depth": 12, "batch": 1024,
         "dtype": "f32"},
        # products of an odd width and an odd batch in double precision
        {"name": "mul_w5d6_f64", "op": "mul", "width": 5, "depth": 6, "batch": 701,
         "dtype": "f64"},
        # running products updated in place (Chen's identity, one update of every row)
        {"name": "inplace_w4d7_f32", "op": "inplace", "width": 4, "depth": 7, "batch": 2000,
         "dtype": "f32"},
        # signatures of Lie elements (abelian pieces): embed, then exponentiate
        {"name": "lie_exp_w5d5_f32", "op": "lie_exp", "width": 5, "depth": 5, "batch": 4001,
         "dtype": "f32"},
        # log-signature coordinates of a batch of signatures: log, then project
        {"name": "log_lie_w6d5_f64", "op": "log_lie", "width": 6, "depth": 5, "batch": 4096,
         "dtype": "f64"},
        # the adjoint of left multiplication: the backward direction of a product
        {"name": "adjoint_w3d7_f64", "op": "adjoint", "width": 3, "depth": 7, "batch": 500,
         "dtype": "f64"},
        # a small batch of equal short streams in double precision
        {"name": "sig_w4d5_f64", "op": "sig", "width": 4, "depth": 5, "streams": 256,
         "min_len": 128, "max_len": 128, "dtype": "f64"},
        # the bulk workload: thousands of uneven streams in one launch
        {"name": "sig_w8d5_f32", "op": "sig", "width": 8, "depth": 5, "streams": 4096,
         "min_len": 16, "max_len": 4096, "dtype": "f32"},
        # a training step on signatures: forward and gradient of the increments
        {"name": "sig_grad_w5d6_f32", "op": "sig_grad", "width": 5, "depth": 6, "streams": 512,
         "min_len": 1024, "max_len": 1024, "dtype": "f32"},
        # many interval queries of one long stream with its dyadic cache built
        {"name": "queries_w6d5_f64", "op": "queries", "width": 6, "depth": 5, "log2_events": 16,
         "queries": 100000, "dtype": "f64"},
    ]


# ------------------------------------------------------------------ sizes
def level_starts(width, depth):
    db = [0]
    for k in range(depth + 1):
        db.append(db[-1] + width ** k)
    return db


def tensor_size(width, depth):
    return level_starts(width, depth)[-1]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: widths 2..10, small to large tensors, any batch."""
    op = rng.choice(("mul", "fma", "inplace", "exp", "fmexp", "log", "antipode", "adjoint",
                     "lie_exp", "log_lie", "sig", "sig_grad", "queries"))
    dtype = rng.choice(("f32", "f64"))
    if op in ("sig", "sig_grad"):
        width = rng.randint(2, 8)
        deepest = 8 if width <= 3 else 7 if width == 4 else 6
        if op == "sig_grad":
            while width ** (deepest - 2) > 992:
                deepest -= 1
        depth = rng.randint(2, deepest)
        size = tensor_size(width, depth)
        # total work at most that of the largest listed case of the family
        budget = (512 * 1024 * 19531) if op == "sig_grad" else (4096 * 2056 * 37449)
        budget //= 2 if dtype == "f64" else 1
        max_len = _log_uniform(rng, 16, 1024 if op == "sig_grad" else 4096)
        most = max(1, min(512 if op == "sig_grad" else 4096, budget // (size * max_len),
                          MAX_WORDS // size))
        n = _log_uniform(rng, 1, most)
        min_len = rng.choice((max_len, rng.randint(1, max_len)))
        return {"op": op, "width": width, "depth": depth, "streams": n, "min_len": min_len,
                "max_len": max_len, "dtype": dtype}
    if op == "queries":
        width = rng.randint(2, 6)
        depth = rng.choice([n for n in range(2, 13) if tensor_size(width, n) <= 9331])
        return {"op": op, "width": width, "depth": depth, "log2_events": rng.randint(8, 16),
                "queries": _log_uniform(rng, 1, 100000), "dtype": dtype}
    most = MAX_LIE_TENSOR if op in LIE_OPS else 299593
    width = rng.randint(2, 6 if op in LIE_OPS else 10)
    depth = rng.choice([n for n in range(2, 17) if 15 <= tensor_size(width, n) <= most
                        and (op not in LIE_OPS or n <= 10)] or [2])
    size = tensor_size(width, depth)
    # adjoint, exp, log: at most about the traffic of the largest listed case of their kind
    words = MAX_WORDS if op in ("mul", "fma", "inplace", "antipode") else MAX_WORDS // 8
    batch = _log_uniform(rng, 1, max(1, min(words // size, 65536)))
    return {"op": op, "width": width, "depth": depth, "batch": batch, "dtype": dtype}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _tensors(case, g, scalar, scale=1.0):
    """Rows with level-k coefficients N(0,1)/k! and the given scalar."""
    w, n = case["width"], case["depth"]
    db = level_starts(w, n)
    x = torch.randn(case["batch"], db[-1], dtype=DTYPES[case["dtype"]], device="cuda",
                    generator=g)
    for k in range(1, n + 1):
        x[:, db[k]:db[k + 1]] *= scale / math.factorial(k)
    x[:, 0] = scalar
    return x


def _lie_rows(case, g):
    """Lie coordinates of decaying size by degree."""
    degs = hall_set(case["width"], case["depth"])[2]
    x = torch.randn(case["batch"], len(degs), dtype=DTYPES[case["dtype"]], device="cuda",
                    generator=g)
    scale = [1.0 / math.factorial(k) for k in degs]
    return x * torch.tensor(scale, dtype=x.dtype, device="cuda")


def _offsets(case, seed):
    rng = np.random.default_rng(int(seed))
    lens = rng.integers(case["min_len"], case["max_len"] + 1, case["streams"])
    return np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)


def _increments(case, off, g):
    """Brownian increments N(0, 1/length) per channel."""
    lens = torch.from_numpy(np.diff(off)).cuda()
    scale = torch.repeat_interleave(lens.to(torch.float64).rsqrt(), lens)
    x = torch.randn(int(off[-1]), case["width"], dtype=torch.float64, device="cuda",
                    generator=g)
    return (x * scale[:, None]).to(DTYPES[case["dtype"]])


def _event_rows(case, seed):
    n = 1 << case["log2_events"]
    rng = np.random.default_rng(int(seed))
    rows = rng.standard_normal((n, case["width"])) * 2.0 ** (-case["log2_events"] / 2)
    a = rng.integers(0, n, case["queries"])
    b = rng.integers(0, n, case["queries"])
    lo, hi = np.minimum(a, b), np.maximum(a, b)
    hi = np.where(hi == lo, lo + 1, hi)
    return rows.astype(np.float32 if case["dtype"] == "f32" else np.float64), lo, hi


def inputs(case, seed):
    """The case's raw inputs, made from the seed alone."""
    g = _gen(seed)
    op = case["op"]
    if op in ("mul", "adjoint"):
        return _tensors(case, g, 1.0), _tensors(case, g, 1.0)
    if op == "fma":
        return _tensors(case, g, 1.0), _tensors(case, g, 1.0), _tensors(case, g, 1.0)
    if op == "inplace":
        # a step of a running product: a factor close to the unit
        return _tensors(case, g, 1.0), _tensors(case, g, 1.0, 0.01)
    if op == "fmexp":
        return _tensors(case, g, 1.0), _tensors(case, g, 0.0)
    if op == "exp":
        return (_tensors(case, g, 0.0),)
    if op in ("log", "log_lie", "antipode"):
        return (_tensors(case, g, 1.0),)
    if op == "lie_exp":
        return (_lie_rows(case, g),)
    if op in ("sig", "sig_grad"):
        off = _offsets(case, seed)
        inc = _increments(case, off, g)
        if op == "sig":
            return off, inc
        w = torch.randn(case["streams"], tensor_size(case["width"], case["depth"]),
                        dtype=inc.dtype, device="cuda", generator=g)
        return off, inc, w
    return _event_rows(case, seed)


def prepare(case, seed):
    """What a user's program holds before the call: inputs, bases, plans, streams."""
    op, x = case["op"], inputs(case, seed)
    state = {"op": op}
    if op in ("sig", "sig_grad"):
        state["plan"] = sigs.SignaturePlan(x[0], case["width"], case["depth"],
                                           "f32c" if case["dtype"] == "f32" else "f64")
        state["inc"] = x[1]
        if op == "sig_grad":
            state["inc"].requires_grad_(True)
            state["weights"] = x[2]
        return state
    if op == "queries":
        rows, lo, hi = x
        n = 1 << case["log2_events"]
        state["stream"] = streams.LieIncrementStream.from_increments(
            rows, indices=np.arange(n) / n, width=case["width"], depth=case["depth"],
            resolution=case["log2_events"])
        state["infs"], state["sups"] = lo / n, hi / n
        # the first batch of queries builds the stream's device cache, as in a program
        # that goes on querying it
        k = min(case["queries"], 1024)
        state["stream"].log_signature_batch(state["infs"][:k], state["sups"][:k])
        return state
    basis = rpc.TensorBasis(case["width"], case["depth"])
    if op in LIE_OPS:
        state["lie_basis"] = rpc.LieBasis(case["width"], case["depth"])
        state["tensor_basis"] = basis
        # the maps belong to the basis and are made once
        if op == "lie_exp":
            state["x"] = rpc.Lie(x[0], state["lie_basis"])
            state["lie_basis"].get_l2t_matrix(np.float64)
        else:
            state["x"] = rpc.FreeTensor(x[0], basis)
            state["lie_basis"].get_t2l_matrix(np.float64)
        return state
    state["args"] = [rpc.FreeTensor(t, basis) for t in x]
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    op = state["op"]
    if op == "sig":
        return state["plan"].run(state["inc"])
    if op == "sig_grad":
        sig = sigs.signature_with_grad(state["inc"], state["plan"])
        (grad,) = torch.autograd.grad(sig, state["inc"], state["weights"])
        return sig.detach(), grad
    if op == "queries":
        return state["stream"].log_signature_batch(state["infs"], state["sups"])
    if op == "lie_exp":
        return rpc.ft_exp(rpc.lie_to_tensor(state["x"], state["tensor_basis"])).data
    if op == "log_lie":
        return rpc.tensor_to_lie(rpc.ft_log(state["x"]), state["lie_basis"]).data
    args = state["args"]
    if op == "mul":
        return rpc.ft_mul(*args).data
    if op == "fma":
        rpc.ft_fma(*args)
        return args[0].data
    if op == "inplace":
        rpc.ft_inplace_mul(*args)
        return args[0].data
    if op == "exp":
        return rpc.ft_exp(args[0]).data
    if op == "fmexp":
        return rpc.ft_fmexp(*args).data
    if op == "log":
        return rpc.ft_log(args[0]).data
    if op == "antipode":
        return rpc.antipode(args[0]).data
    return rpc.ft_adjoint_left_mul(*args).data


# ------------------------------------------------------------------ what a pass needs
def work(case):
    w, n, op = case["width"], case["depth"], case["op"]
    es = 4 if case["dtype"] == "f32" else 8
    size = tensor_size(w, n)
    product = sum(2.0 * (k + 1) * w ** k for k in range(n + 1))
    step = sum(2.0 * (k + 1) * w ** k for k in range(1, n + 1))     # one Chen step
    if op in ("sig", "sig_grad"):
        # the expected number of rows; every word's Horner chain is shared by the words
        # below it, so a step costs about one multiply-add a word
        rows = case["streams"] * (case["min_len"] + case["max_len"]) / 2
        per_row = 2.0 * sum(w ** k for k in range(1, n + 1)) * w / (w - 1)
        io = es * (rows * w + case["streams"] * size)
        if op == "sig":
            return {"bytes": io, "flops": rows * per_row}
        return {"bytes": 2 * io + es * case["streams"] * size, "flops": 3 * rows * per_row}
    if op == "queries":
        # each query: the two ends of its range, a logarithm and a projection
        lie = len(hall_set(w, n)[2])
        q = case["queries"]
        return {"bytes": q * (2.0 * es * size + 8.0 * lie), "flops": q * 2.0 * product}
    b = case["batch"]
    if op in LIE_OPS:
        lie = len(hall_set(w, n)[2])
        return {"bytes": float(b * es * (size + lie)), "flops": b * product}
    # log needs as many series steps as levels, but only the last reaches the top level
    passes = {"mul": 3, "fma": 4, "inplace": 3, "exp": 2, "fmexp": 3, "log": 2, "antipode": 2,
              "adjoint": 3}[op]
    flops = {"antipode": 0.0, "exp": step, "log": step, "adjoint": product}.get(op, product)
    return {"bytes": float(b * size * es * passes), "flops": b * flops}


# ------------------------------------------------------------------ float64 in plain torch
def _levels(x, w, n):
    db = level_starts(w, n)
    return [x[:, db[k]:db[k + 1]] for k in range(n + 1)]


def _mul64(a, b, w, n, out=None):
    """out (zeros by default) += a (x) b, rows of dense tensors in float64."""
    if out is None:
        out = torch.zeros_like(a)
    la, lb, lo = _levels(a, w, n), _levels(b, w, n), _levels(out, w, n)
    rows = a.shape[0]
    for k in range(n + 1):
        for p in range(k + 1):
            lo[k].view(rows, w ** p, w ** (k - p)).addcmul_(la[p].unsqueeze(2),
                                                            lb[k - p].unsqueeze(1))
    return out


def _exp64(x, w, n, mult=None):
    """mult (x) exp(x) by Horner's rule; the scalar of x is ignored."""
    x = x.clone()
    x[:, 0] = 0
    if mult is None:
        mult = torch.zeros_like(x)
        mult[:, 0] = 1
    r = mult.clone()
    for k in range(n, 0, -1):
        r = _mul64(r, x / k, w, n, mult.clone())
    return r


def _log64(x, w, n):
    x = x.clone()
    x[:, 0] = 0
    r = torch.zeros_like(x)
    for k in range(n, 0, -1):
        r[:, 0] += (1.0 if k % 2 else -1.0) / k
        r = _mul64(r, x, w, n)
    return r


def _antipode64(x, w, n):
    out = torch.empty_like(x)
    for k, (src, dst) in enumerate(zip(_levels(x, w, n), _levels(out, w, n))):
        t = src.reshape([x.shape[0]] + [w] * k)
        t = t.permute([0] + list(range(k, 0, -1))).reshape(x.shape[0], -1)
        dst.copy_(-t if k % 2 else t)
    return out


def _adjoint64(op, arg, w, n):
    out = torch.zeros_like(arg)
    lop, larg, lout = _levels(op, w, n), _levels(arg, w, n), _levels(out, w, n)
    for k in range(n + 1):
        for q in range(n - k + 1):
            a = larg[k + q].reshape(arg.shape[0], w ** q, w ** k)
            lout[k] += torch.bmm(lop[q].reshape(arg.shape[0], 1, -1), a).squeeze(1)
    return out


def _by_rows(f, rows, size):
    """f(a, b) over row ranges of at most 2**26 words."""
    step = max(1, (1 << 26) // size)
    return torch.cat([f(i, min(i + step, rows)) for i in range(0, rows, step)])


_HALL = {}


def hall_set(width, depth):
    """(left, right, degrees) of the Hall basis in the package's order; key 0 is null."""
    if (width, depth) not in _HALL:
        left, right, deg = [0] + [0] * width, [0] + list(range(1, width + 1)), [0] + [1] * width
        begin = [0, 1, width + 1]
        for d in range(2, depth + 1):
            for e in range(1, d // 2 + 1):
                for i in range(begin[e], begin[e + 1]):
                    for j in range(max(i + 1, begin[d - e]), begin[d - e + 1]):
                        if left[j] <= i:
                            left.append(i)
                            right.append(j)
                            deg.append(d)
            begin.append(len(left))
        _HALL[width, depth] = (left, right, deg[1:])
    return _HALL[width, depth]


_MAPS = {}


def _l2t64(width, depth):
    """Per degree k: the [n_k, width**k] matrix of the Hall elements as tensors."""
    if (width, depth) not in _MAPS:
        left, right, deg = hall_set(width, depth)
        out, begin, key = [None], [0, 1], 1
        for k in range(1, depth + 1):
            begin.append(begin[k] + deg.count(k))
            m = torch.zeros(deg.count(k), width ** k, dtype=torch.float64)
            for r in range(m.shape[0]):
                if k == 1:
                    m[r, r] = 1
                else:
                    i, j = left[key], right[key]
                    di, dj = deg[i - 1], deg[j - 1]
                    a, b = out[di][i - begin[di]], out[dj][j - begin[dj]]
                    m[r] = torch.outer(a, b).reshape(-1) - torch.outer(b, a).reshape(-1)
                key += 1
            out.append(m)
        _MAPS[width, depth] = [m.cuda() if m is not None else None for m in out]
    return _MAPS[width, depth]


def _lie_to_tensor64(x, w, n):
    maps = _l2t64(w, n)
    parts, at = [torch.zeros(x.shape[0], 1, dtype=torch.float64, device=x.device)], 0
    for k in range(1, n + 1):
        parts.append(x[:, at:at + maps[k].shape[0]] @ maps[k])
        at += maps[k].shape[0]
    return torch.cat(parts, 1)


def _bracket64(x, w, k):
    """Right-normed bracketing of words, as a map of degree-k tensors."""
    if k == 1:
        return x
    z = _bracket64(x.reshape(-1, w ** (k - 1)), w, k - 1).reshape(-1, w, w ** (k - 1))
    return z.reshape(x.shape[0], -1) - z.transpose(1, 2).reshape(x.shape[0], -1)


def _tensor_to_lie64(x, w, n):
    maps, parts = _l2t64(w, n), []
    for k, level in enumerate(_levels(x, w, n)):
        if k == 0 or maps[k].shape[0] == 0:
            continue
        m = maps[k]
        r = _bracket64(level.contiguous(), w, k) / k
        chol = torch.linalg.cholesky(m @ m.T)
        parts.append(torch.cholesky_solve(m @ r.T, chol).T)
    return torch.cat(parts, 1)


def _chen_step64(state, x, w, n):
    """One step state <- state (x) exp(x) on lists of levels, differentiable."""
    out = list(state)
    for k in range(n, 0, -1):
        acc = x / k
        for i in range(1, k):
            acc = state[i] + acc
            acc = (acc.unsqueeze(2) * (x / (k - i)).unsqueeze(1)).reshape(x.shape[0], -1)
        out[k] = state[k] + acc
    return out


def _signature64(inc, off, w, n):
    """Signatures of all streams, stepping the streams that are still running together."""
    lens = np.diff(off)
    order = np.argsort(-lens, kind="stable")
    first = torch.from_numpy(off[:-1][order].copy()).cuda()
    size = tensor_size(w, n)
    s = torch.zeros(len(lens), size, dtype=torch.float64, device="cuda")
    s[:, 0] = 1
    levels = [torch.zeros(len(lens), w ** k, dtype=torch.float64, device="cuda")
              for k in range(n + 1)]
    running = np.searchsorted(-lens[order], -np.arange(1, int(lens.max()) + 1), side="right")
    for t, m in enumerate(running):
        m = int(m)
        x = inc[first[:m] + t]
        xs = [None] + [x / q for q in range(1, n + 1)]
        for k in range(n, 0, -1):
            acc = xs[k]
            for i in range(1, k):
                acc = acc + levels[i][:m]
                if i < k - 1:
                    acc = (acc.unsqueeze(2) * xs[k - i].unsqueeze(1)).reshape(m, -1)
            if k == 1:
                levels[1][:m] += x
            else:
                levels[k][:m].view(m, w ** (k - 1), w).addcmul_(acc.unsqueeze(2), x.unsqueeze(1))
    out = torch.empty(len(lens), size, dtype=torch.float64, device="cuda")
    levels[0][:] = 1
    out[torch.from_numpy(order).cuda()] = torch.cat(levels, 1)
    return out


def _signature_grad64(inc, off, weights, w, n):
    """(signature, gradient of <weights, signature>) by autograd with checkpoints."""
    from torch.utils.checkpoint import checkpoint
    lens = np.diff(off)
    longest = int(lens.max())
    # shorter streams end in zero steps, which change nothing
    pos = np.minimum(off[:-1, None] + np.arange(longest)[None], max(int(off[-1]) - 1, 0))
    live = torch.from_numpy(np.arange(longest)[None] < lens[:, None]).cuda()
    inc = inc.detach().requires_grad_(True)
    rows = inc[torch.from_numpy(pos).cuda()] * live[..., None]

    def segment(block, *state):
        state = list(state)
        for t in range(block.shape[1]):
            state = _chen_step64(state, block[:, t], w, n)
        return tuple(state)

    state = [torch.ones(len(lens), 1, dtype=torch.float64, device="cuda")]
    state += [torch.zeros(len(lens), w ** k, dtype=torch.float64, device="cuda")
              for k in range(1, n + 1)]
    step = max(1, min(32, (1 << 34) // max(1, 4 * len(lens) * tensor_size(w, n) * 8)))
    for t in range(0, longest, step):
        state = list(checkpoint(segment, rows[:, t:t + step], *state, use_reentrant=False))
    sig = torch.cat(state, 1)
    (grad,) = torch.autograd.grad(sig, inc, weights)
    return sig.detach(), grad


def _queries64(case, seed):
    w, n = case["width"], case["depth"]
    rows, lo, hi = _event_rows(case, seed)
    size, events = tensor_size(w, n), rows.shape[0]
    x = torch.zeros(events, size, dtype=torch.float64, device="cuda")
    x[:, 1:w + 1] = torch.from_numpy(rows).cuda().double()
    x = _by_rows(lambda a, b: _exp64(x[a:b], w, n), events, size)
    # prefix products in log2(events) rounds
    s = 1
    while s < events:
        tail = _by_rows(lambda a, b: _mul64(x[a:b], x[a + s:b + s], w, n), events - s, size)
        x[s:] = tail
        del tail
        s *= 2
    unit = torch.zeros(1, size, dtype=torch.float64, device="cuda")
    unit[0, 0] = 1
    x = torch.cat([unit, x])
    lo, hi = torch.from_numpy(lo).cuda(), torch.from_numpy(hi).cuda()

    def part(a, b):
        s = _mul64(_antipode64(x[lo[a:b]], w, n), x[hi[a:b]], w, n)
        return _tensor_to_lie64(_log64(s, w, n), w, n)
    return _by_rows(part, len(lo), size)


def exact(case, seed):
    """The value of ``run`` for these inputs in float64."""
    w, n, op = case["width"], case["depth"], case["op"]
    if op == "queries":
        return _queries64(case, seed)
    if op == "sig":
        off, inc = inputs(case, seed)
        return _signature64(inc.double(), off, w, n)
    if op == "sig_grad":
        off, inc, weights = inputs(case, seed)
        return _signature_grad64(inc.double(), off, weights.double(), w, n)
    x = inputs(case, seed)
    f = {"mul": lambda a, b: _mul64(a, b, w, n),
         "fma": lambda c, a, b: _mul64(a, b, w, n, c.clone()),
         "inplace": lambda a, b: _mul64(a, b, w, n),
         "exp": lambda a: _exp64(a, w, n),
         "fmexp": lambda m, a: _exp64(a, w, n, m),
         "log": lambda a: _log64(a, w, n),
         "antipode": lambda a: _antipode64(a, w, n),
         "adjoint": lambda o, a: _adjoint64(o, a, w, n),
         "lie_exp": lambda a: _exp64(_lie_to_tensor64(a, w, n), w, n),
         "log_lie": lambda a: _tensor_to_lie64(_log64(a, w, n), w, n)}[op]
    return _by_rows(lambda a, b: f(*(t[a:b].double() for t in x)), x[0].shape[0],
                    tensor_size(w, n))
