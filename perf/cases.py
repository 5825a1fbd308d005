"""The work that is timed: what a program that uses this package has it do.

Four kinds of calls, all through the package's public entry points on device
buffers (the resident forms that a solver loop, a server or a Krylov method
keeps):

* ``product``  -- ``hssA * B`` (``DeviceHss.matmul_device``), FP64, one to 64
  columns, also with the adjoint (``trans``);
* ``ldiv``     -- ``hssA \\ B``: factorization and solve in one call
  (``UlvFactor.factsolve_device``), plain FP64 or FP32 refined to 1e-10;
* ``solve``    -- a solve with a factorization that is already there
  (``UlvFactor.solve_device``);
* ``batch``    -- the same for a forest of independent matrices of mixed
  sizes (``refactor`` + ``solve_batch_device``);
* ``sample``   -- the products A Omega and A^T Omega of randomized compression
  (``sample``);
* ``compress`` -- ``randcompress_adaptive`` of a kernel matrix, and a
  64-column product with the result.

Sizes are those of the package's own configurations and tests: n up to 65536,
leafsize 64 / 128 / 256, ranks 4 to 48.  Matrices have the synthetic form of
``synthetic_hss`` (dense leaf blocks shifted by 4 I, orthonormal nested bases,
couplings of norm about one); with ``vary`` every node has ranks of its own, as
compression gives them, and U and V sides differ.  The shape of a case comes from
the case alone, all values from the seed.
"""
import math

import numpy as np
import torch

import __graft_entry__

pkg = __graft_entry__.load_package()

GRAPHS = 4      # HSS_OPT_GRAPHS: launch sequences replayed as CUDA graphs
SHIFT, COUPLING = 4.0, 0.5


def listed():
    return [
        # an operator of a few hundred unknowns inside an iterative method: launch latency
        dict(name="product_small", op="product", n=512, ls=64, k=16, r=1, vary=False, trans=False),
        # the matvec workload: one vector, the largest matrix
        dict(name="product_vector", op="product", n=65536, ls=128, k=32, r=1, vary=False, trans=False),
        # an adjoint product, odd sizes and ranks of compression, a few columns
        dict(name="product_ragged_adjoint", op="product", n=10007, ls=64, k=20, r=7, vary=True, trans=True),
        # the matvec workload with a block of columns (block Krylov, sampling an operator)
        dict(name="product_block", op="product", n=65536, ls=128, k=32, r=32, vary=False, trans=False),
        # a small system solved once, plain FP64 (the default of hssA \ b)
        dict(name="ldiv_small", op="ldiv", n=1200, ls=64, k=16, r=2, vary=False, prec="fp64", graphs=False),
        # the largest system in plain FP64
        dict(name="ldiv_fp64", op="ldiv", n=65536, ls=128, k=32, r=32, vary=False, prec="fp64", graphs=True),
        # the precision workload: the largest system, FP32 factors refined to 1e-10
        dict(name="ldiv_mixed", op="ldiv", n=65536, ls=128, k=32, r=32, vary=False, prec="fp32", graphs=True),
        # large leaves, odd size, ranks of compression, few right-hand sides
        dict(name="ldiv_wide_leaves", op="ldiv", n=20011, ls=256, k=40, r=5, vary=True, prec="fp32", graphs=False),
        # a request against a resident factorization (the serving form)
        dict(name="solve_resident", op="solve", n=16384, ls=128, k=32, r=4, vary=False, prec="fp32", graphs=False),
        # many independent systems of mixed sizes in one forest (the batching form)
        dict(name="batch_mixed", op="batch", count=48, sizes=2, rmax=16, prec="fp32", graphs=True),
        # the sample products of randomized compression, both directions
        dict(name="sample_both", op="sample", n=8192, r=30, prec="fp64"),
        # a kernel matrix compressed, and used for one block product
        dict(name="compress_apply", op="compress", n=16384, ls=128, r=64, prec="fp64"),
    ]


def draw(rng):
    op = rng.choice(["product", "product", "product", "ldiv", "ldiv", "ldiv", "solve", "batch", "sample", "compress"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    if op == "batch":
        return dict(op=op, count=log(8, 48), sizes=rng.randrange(1 << 20), rmax=log(1, 16),
                    prec=rng.choice(["fp32", "fp32", "fp64"]), graphs=rng.random() < 0.5)
    if op == "sample":
        return dict(op=op, n=log(700, 8192), r=log(8, 70), prec=rng.choice(["fp64", "fp64", "df"]))
    if op == "compress":
        return dict(op=op, n=log(1500, 12000), ls=rng.choice([64, 100, 128]), r=log(4, 64),
                    prec=rng.choice(["fp64", "fp64", "df"]))
    ls = rng.choice([64, 128, 128, rng.randrange(40, 129), 256])
    n = log(256, 65536 if ls <= 128 else 20011)
    if rng.random() < 0.4:
        n = max(256, n // 128 * 128)
    k = rng.choice([8, 16, 32, rng.randrange(4, 49)])
    case = dict(op=op, n=n, ls=ls, k=min(k, ls // 2), r=log(1, 64 if op == "product" else 32), vary=rng.random() < 0.5)
    if op == "product":
        case["trans"] = rng.random() < 0.3
    else:
        case["prec"] = rng.choice(["fp32", "fp64"])
        case["graphs"] = rng.random() < 0.5
    return case


# ---- matrices ---------------------------------------------------------------------


def _shapes(n, ls, k, vary):
    """The tree as nested lists: [size, ku, kv, left, right], 0 ranks at the root."""
    pick = np.random.default_rng([n, ls, k])

    def build(m, root):
        kids = [] if m <= ls else [build((m + 1) // 2, False), build(m // 2, False)]
        tops = [min(k, m)] * 2 if not kids else [min(k, kids[0][q] + kids[1][q]) for q in (1, 2)]
        ku, kv = (0, 0) if root else tops
        if vary and not root:
            ku, kv = (int(pick.integers(max(1, (t + 1) // 2), t + 1)) for t in (ku, kv))
        return [m, ku, kv] + (kids or [None, None])

    return build(n, True)


def _walk(t):
    yield t
    if t[3]:
        yield from _walk(t[3])
        yield from _walk(t[4])


def _values(shape, seed):
    """Block values for every node: leaves (D, U, V), branches (B12, B21, R, W)."""
    rng = np.random.default_rng(seed)
    nodes = list(_walk(shape))
    values = {}
    wanted = {}
    for i, t in enumerate(nodes):
        if t[3] is None:
            wanted.setdefault((t[0], t[0]), []).append((i, "D"))
        rows_u, rows_v = (t[0], t[0]) if t[3] is None else (t[3][1] + t[4][1], t[3][2] + t[4][2])
        if t[1]:
            wanted.setdefault((rows_u, t[1], "q"), []).append((i, "U"))
            wanted.setdefault((rows_v, t[2], "q"), []).append((i, "V"))
        if t[3]:
            wanted.setdefault((t[3][1], t[4][2]), []).append((i, "B12"))
            wanted.setdefault((t[4][1], t[3][2]), []).append((i, "B21"))
    for key, at in wanted.items():
        x = rng.standard_normal((len(at),) + key[:2])
        if len(key) == 3:       # orthonormal columns
            x = torch.linalg.qr(torch.from_numpy(x)).Q.numpy()
        for (i, what), b in zip(at, x):
            if what == "D":
                b = b / math.sqrt(key[0]) + SHIFT * np.eye(key[0])
            elif what[0] == "B":
                b = b * (COUPLING / math.sqrt(max(key)))
            values[i, what] = b
    return nodes, values


def _tree(shape, seed):
    """The package's ``HssMatrix`` of a shape."""
    nodes, val = _values(shape, seed)
    at = {id(t): i for i, t in enumerate(nodes)}
    H = pkg.HssMatrix

    def build(t, root):
        i = at[id(t)]
        if t[3] is None:
            return H.leaf(val[i, "D"], rootnode=True) if root else H.leaf(val[i, "D"], val[i, "U"], val[i, "V"])
        a, b = build(t[3], False), build(t[4], False)
        if root:
            return H.branch(a, b, val[i, "B12"], val[i, "B21"], rootnode=True)
        ku, kv, U, V = t[3][1], t[3][2], val[i, "U"], val[i, "V"]
        return H.branch(a, b, val[i, "B12"], val[i, "B21"], U[:ku], V[:kv], U[ku:], V[kv:], rootnode=False)

    return build(shape, True)


def _kernel(n, seed):
    """1 / (x_i - x_j) with a unit diagonal on jittered points of [-1, 1], as the row-major tensor of A."""
    jitter = torch.from_numpy(np.random.default_rng(seed).uniform(-0.2, 0.2, n)).cuda()
    x = torch.linspace(-1.0, 1.0, n, dtype=torch.float64, device="cuda") + jitter * (2.0 / n)
    A = (x[:, None] - x[None, :]).reciprocal_()
    A.diagonal().fill_(1.0)
    return A


def _columns(seed, r, n):
    """n x r, column-major on the device: a tensor of r rows."""
    return torch.from_numpy(np.random.default_rng(np.append(seed, 1)).standard_normal((r, n))).cuda()


def _forest(case):
    """(n, leafsize, k, r) of every matrix of a batch, as the batching workload draws them."""
    rng = np.random.default_rng(case["sizes"])
    out = []
    for _ in range(case["count"]):
        n = int(rng.integers(1024 // 128, 8192 // 128 + 1)) * 128
        ls, k = int(rng.choice([64, 128, 256])), int(rng.integers(8, 49))
        out.append((n, ls, min(k, ls // 2), int(rng.integers(1, case["rmax"] + 1))))
    return out


# ---- the measured interface ---------------------------------------------------------


def prepare(case, seed):
    op = case["op"]
    state = dict(op=op, stream=torch.cuda.current_stream())
    if op == "sample":
        # the matrix is stored by columns, as the package keeps it
        state.update(A=pkg.DenseDevice(_kernel(case["n"], seed)), X=_columns(seed, case["r"], case["n"]),
                     df=int(case["prec"] == "df"))
        return state
    if op == "compress":
        n = case["n"]
        cl = pkg.bisection_cluster(n, case["ls"])
        state.update(A=pkg.DenseDevice(_kernel(n, seed)), cl=cl, X=_columns(seed, case["r"], n), n=n, seed=seed,
                     prec=case["prec"])
        state["Y"] = torch.empty_like(state["X"])
        return state
    if op != "product":
        pkg._lib.check(pkg._lib.load().hss_set_option(GRAPHS, int(case["graphs"])))
        if case["graphs"]:      # graphs are replayed on a stream of the program's own
            state["stream"] = torch.cuda.Stream()
    if op == "batch":
        trees = [_tree(_shapes(n, ls, k, False), [seed, i]) for i, (n, ls, k, _r) in enumerate(_forest(case))]
        state["ns"] = [f[0] for f in _forest(case)]
        state["rs"] = [f[3] for f in _forest(case)]
        state["dev"] = pkg.DeviceHss.from_trees(trees)
        state["B"] = [_columns([seed, i], r, n) for i, (n, r) in enumerate(zip(state["ns"], state["rs"]))]
        state["X"] = [torch.empty_like(b) for b in state["B"]]
    else:
        state.update(n=case["n"], r=case["r"], trans=case.get("trans", False))
        state["dev"] = pkg.DeviceHss(_tree(_shapes(case["n"], case["ls"], case["k"], case["vary"]), seed))
        state["B"] = _columns(seed, case["r"], case["n"])
        state["X"] = torch.empty_like(state["B"])
    torch.cuda.synchronize()
    if op != "product":
        state["F"] = state["dev"].ulvfactor(case["prec"], stream=state["stream"])
    return state


def run(s):
    op, st = s["op"], s["stream"]
    if op == "product":
        s["dev"].matmul_device(s["B"], s["n"], s["r"], s["X"], s["n"], stream=st, trans=s["trans"])
        return s["X"]
    if op == "ldiv":
        s["F"].factsolve_device(s["B"], s["n"], s["r"], s["X"], s["n"], maxit=20, stream=st)
        return s["X"]
    if op == "solve":
        s["F"].solve_device(s["B"], s["n"], s["r"], s["X"], s["n"], maxit=20, stream=st)
        return s["X"]
    if op == "batch":
        s["F"].refactor(stream=st)
        s["F"].solve_batch_device(s["B"], s["ns"], s["rs"], s["X"], s["ns"], maxit=20, stream=st)
        return s["X"]
    if op == "sample":
        lib = pkg._lib.load()
        if s["df"]:
            lib.hss_set_option(pkg.compression.HSS_OPT_SAMPLE_DF, 1)
        out = [pkg.sample(s["A"], s["X"], stream=st), pkg.sample(s["A"], s["X"], trans=True, stream=st)]
        if s["df"]:
            lib.hss_set_option(pkg.compression.HSS_OPT_SAMPLE_DF, 0)
        return out
    hss = pkg.randcompress_adaptive(s["A"], s["cl"], s["cl"], kest=10, atol=1e-9, rtol=1e-9, noversampling=10,
                                    stepsize=20, rng=np.random.default_rng(s["seed"]), device=True,
                                    sample_precision=s["prec"])
    hss.matmul_device(s["X"], s["n"], s["X"].shape[0], s["Y"], s["n"], stream=st)
    return s["Y"]


def _entries(shape):
    total = 0
    for t in _walk(shape):
        m, ku, kv, a, b = t
        if a is None:
            total += m * m + m * (ku + kv)
        else:
            total += a[1] * b[2] + b[1] * a[2] + (a[1] + b[1]) * ku + (a[2] + b[2]) * kv
    return total


def _ulv_flops(shape):
    """Operations of the factorization, and of a solve per right-hand side."""
    fac = sol = 0.0

    def visit(t, root):
        nonlocal fac, sol
        m, ku, kv, a, b = t
        if a is not None:
            ra, rb = visit(a, False), visit(b, False)
            m = ra + rb
            # T = U B, the off-diagonal blocks, and the merged bases
            fac += 2.0 * (ra * a[1] * b[2] + rb * b[1] * a[2] + ra * b[2] * rb + rb * a[2] * ra)
            fac += 2.0 * (ra * a[1] + rb * b[1]) * ku + 2.0 * (ra * a[2] + rb * b[2]) * kv
            sol += 2.0 * (ra * (a[1] + b[2]) + rb * (b[1] + a[2]))
        if root:
            fac += 2.0 / 3.0 * m ** 3
            sol += 2.0 * m * m
            return 0
        e = m - ku          # rows eliminated
        if e <= 0:
            return m
        fac += 2.0 * m * ku * ku + 4.0 * m * m * ku          # QL of U, applied to D
        fac += 2.0 * e * e * m + 4.0 * m * e * (ku + kv)     # LQ of the top rows, applied below and to V
        sol += 4.0 * m * (ku + e) + e * e + 2.0 * e * (ku + kv)
        return ku

    visit(shape, True)
    return fac, sol


def work(case):
    op = case["op"]
    if op == "sample":
        n, r = case["n"], case["r"]
        return {"bytes": 8.0 * (n * n + 3 * n * r), "flops": 4.0 * n * n * r}
    if op == "compress":
        # 20 sample columns, two rounds with 20 test columns each, both directions
        n, r = case["n"], case["r"]
        return {"bytes": 8.0 * (n * n + 2 * n * r), "flops": 4.0 * n * n * 60}
    one = (_forest(case) if op == "batch" else [(case["n"], case["ls"], case["k"], case["r"])])
    total = {"bytes": 0.0, "flops": 0.0}
    for n, ls, k, r in one:
        shape = _shapes(n, ls, k, case.get("vary", False))
        size = _entries(shape)
        total["bytes"] += 8.0 * (size + 2 * n * r)
        if op == "product":
            total["flops"] += 2.0 * size * r
            continue
        fac, sol = _ulv_flops(shape)
        total["flops"] += sol * r + (0.0 if op == "solve" else fac)
        if case["prec"] == "fp32":      # a refined solve: two passes, two residuals
            total["flops"] += (4.0 * size + sol) * r
    return total


# ---- the same in plain 64-bit torch ----------------------------------------------------


def _to_gpu(shape, seed):
    nodes, val = _values(shape, seed)
    return {id(t): i for i, t in enumerate(nodes)}, {key: torch.from_numpy(v).cuda() for key, v in val.items()}


def _plain_product(shape, seed, B, trans):
    """A B (or A^T B) by the two sweeps over the tree; B is n x r."""
    at, val = _to_gpu(shape, seed)
    U, V = ("V", "U") if trans else ("U", "V")
    get = lambda t, what: val[at[id(t)], what]  # noqa: E731
    out = torch.empty_like(B)
    z, places = {}, {}

    def up(t, row0, root):
        places[id(t)] = row0
        if t[3] is None:
            x = B[row0:row0 + t[0]]
        else:
            x = torch.cat([up(t[3], row0, False), up(t[4], row0 + t[3][0], False)])
        if not root:
            z[id(t)] = get(t, V).T @ x
            return z[id(t)]

    def down(t, f):
        if t[3] is None:
            D = get(t, "D")
            row0 = places[id(t)]
            y = (D.T if trans else D) @ B[row0:row0 + t[0]]
            out[row0:row0 + t[0]] = y if f is None else y + get(t, U) @ f
            return
        B12, B21 = (get(t, "B21").T, get(t, "B12").T) if trans else (get(t, "B12"), get(t, "B21"))
        g1, g2 = B12 @ z[id(t[4])], B21 @ z[id(t[3])]
        if f is not None:
            both = get(t, U) @ f
            g1, g2 = g1 + both[:g1.shape[0]], g2 + both[g1.shape[0]:]
        down(t[3], g1)
        down(t[4], g2)

    up(shape, 0, True)
    down(shape, None)
    return out


def _plain_solve(shape, seed, b):
    """A^-1 b by block elimination over the tree; b is n x r.

    With f a node's incoming coefficients (its rows of A x = b read A_node x +
    U f = b), every node keeps z = V^T A_node^-1 b and G = V^T A_node^-1 U."""
    at, val = _to_gpu(shape, seed)
    get = lambda t, what: val[at[id(t)], what]  # noqa: E731
    kept, out = {}, torch.empty_like(b)

    def up(t, row0, root):
        if t[3] is None:
            rhs = b[row0:row0 + t[0]]
            if not root:
                rhs = torch.cat([rhs, get(t, "U")], dim=1)
            s = torch.linalg.solve(get(t, "D"), rhs)
            kept[id(t)] = (row0, s)
        else:
            (z1, G1), (z2, G2) = up(t[3], row0, False), up(t[4], row0 + t[3][0], False)
            kv1, kv2 = z1.shape[0], z2.shape[0]
            M = torch.eye(kv1 + kv2, dtype=b.dtype, device=b.device)
            M[:kv1, kv1:] = G1 @ get(t, "B12")
            M[kv1:, :kv1] = G2 @ get(t, "B21")
            rhs = torch.cat([z1, z2])
            if not root:
                R = get(t, "U")
                rhs = torch.cat([rhs, torch.cat([G1 @ R[:t[3][1]], G2 @ R[t[3][1]:]])], dim=1)
            s = torch.linalg.solve(M, rhs)
            kept[id(t)] = (kv1, s)
        if not root:
            g = get(t, "V").T @ s
            return g[:, :b.shape[1]], g[:, b.shape[1]:]

    def down(t, f):
        first, s = kept[id(t)]
        r = b.shape[1]
        x = s[:, :r] if f is None else s[:, :r] - s[:, r:] @ f
        if t[3] is None:
            out[first:first + t[0]] = x
            return
        f1, f2 = get(t, "B12") @ x[first:], get(t, "B21") @ x[:first]
        if f is not None:
            both = get(t, "U") @ f
            f1, f2 = f1 + both[:t[3][1]], f2 + both[t[3][1]:]
        down(t[3], f1)
        down(t[4], f2)

    up(shape, 0, True)
    down(shape, None)
    return out


def exact(case, seed):
    op = case["op"]
    if op in ("sample", "compress"):
        A = _kernel(case["n"], seed)
        X = _columns(seed, case["r"], case["n"]).T
        y = (A @ X).T.contiguous()
        return y if op == "compress" else [y, (A.T @ X).T.contiguous()]
    if op == "batch":
        out = []
        for i, (n, ls, k, r) in enumerate(_forest(case)):
            out.append(_plain_solve(_shapes(n, ls, k, False), [seed, i], _columns([seed, i], r, n).T).T.contiguous())
        return out
    shape = _shapes(case["n"], case["ls"], case["k"], case["vary"])
    B = _columns(seed, case["r"], case["n"]).T
    if op == "product":
        return _plain_product(shape, seed, B, case["trans"]).T.contiguous()
    return _plain_solve(shape, seed, B).T.contiguous()
