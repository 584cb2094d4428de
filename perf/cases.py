"""The work that users of this library have it do, as cases to measure.

Each case is one call sequence of a user's program through the public Python
API (the same C ABI calls as the C++ API makes): an H^2 matvec, a
preconditioner solve, building and factoring a preconditioner, building an
operator, a GMRES solve on resident systems, or the whole step (build, factor,
solve).  Sizes, kernels, ranks and tolerances are those of the repository's
tests, bench and serving loop.

Vectors on the device are (nrhs, n) row-major tensors, i.e. the library's
column-major n x nrhs with ld = n.
"""
import functools
import math

import numpy as np
import torch

import mxc_b200 as m
from mxc_b200 import _lib as L
from mxc_b200.serving import gaussian_mixture_points, unit_sphere_points

LEAF = 256
TOL = 1e-10  # GMRES tolerance of the bench and the serving loop


def _case(name, do, n, nrhs, **more):
    c = {
        "name": name,
        "do": do,  # matvec | precond | factor | operator | solve | step
        "n": n,
        "nrhs": nrhs,
        "points": "cube",  # cube | mixture | sphere | mesh (the reference's golden-angle sphere)
        "kernel": "laplace",  # laplace | yukawa | helmholtz (complex vectors)
        "singularity": 1e-4,  # diagonal 1/s: dominates the fill that the factorization drops
        "theta": 2.0,
        "eps": 1e-8,  # operator accuracy
        "op_samples": 4000,  # far bodies beyond the nearest three levels (operator sketch); 0: every far body
        "rank": 128,  # of the preconditioner
        "samples": 4000,  # far samples per box of the preconditioner
        "precision": "fp32",  # of the preconditioner: fp64 | fp32 | bf16 (bf16 substitution blocks)
        "matrix_free": False,  # operator blocks evaluated inside the matvec
        "graph": False,  # the solve as one captured graph
        "host": False,  # host arrays (the reference's in-place calls) instead of device arrays
    }
    c.update(more)
    return c


def listed():
    return [
        # The smallest call: one product of the 2048-body test and smoke size on a host vector.
        _case("matvec_host_2048_r1", "matvec", 2048, 1, eps=1e-10, op_samples=0, host=True),
        # An ordinary product of a stored operator with a full batch of right-hand sides (every Arnoldi step is one).
        _case("matvec_65536_r16", "matvec", 65536, 16),
        # The same where the blocks do not fit or are not worth storing: evaluated inside the product.
        _case("matvec_mf_131072_r16", "matvec", 131072, 16, matrix_free=True),
        # The smallest preconditioner solve, on a host vector.
        _case("precond_fp64_host_2048_r1", "precond", 2048, 1, rank=100, samples=2000, precision="fp64", host=True),
        # The mixed mode's preconditioner solve at a large size (every Arnoldi step is one).
        _case("precond_fp32_131072_r16", "precond", 131072, 16),
        # The scale-up configuration's preconditioner solve, smaller and ragged: sphere, Yukawa, bf16 blocks.
        _case("precond_bf16_60001_r8", "precond", 60001, 8, points="sphere", kernel="yukawa", singularity=1e-6,
              theta=3.0, rank=160, samples=6000, precision="bf16"),
        # A preconditioner for a new geometry: built, factored and applied once.
        _case("factor_fp32_65536", "factor", 65536, 16),
        # The README's and lorasp's FP64 run (N = 20000, rank 100, 2000 samples): leaves of 312 or 313 bodies.
        _case("factor_fp64_20000", "factor", 20000, 1, rank=100, samples=2000, precision="fp64"),
        # An operator for a new geometry, and its first product.
        _case("operator_20000", "operator", 20000, 1, op_samples=0),
        # One batch of the serving loop on a resident system: host arrays, captured solve, rank 100.
        _case("solve_8192_r16", "solve", 8192, 16, rank=100, graph=True, host=True),
        # The bench's step (build, factor and solve on a resident operator) at half its size, so that three
        # operators fit the card.
        _case("step_131072_r16", "step", 131072, 16),
        # The reference's default kernel and geometry (complex Helmholtz on a sphere mesh), the bench's 8 columns.
        _case("step_helmholtz_4096_r8", "step", 4096, 8, points="mesh", kernel="helmholtz", singularity=0.1,
              theta=1.0, eps=1e-10, op_samples=0, rank=50, samples=0),
    ]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n | 1 if rng.random() < 0.5 else n


def draw(rng):
    do = rng.choice(["matvec", "matvec", "precond", "precond", "factor", "factor", "operator", "solve", "step", "step",
                     "helmholtz"])
    if do == "helmholtz":  # ranks barely compress at its upper levels: few sizes fit the box limit
        c = _case("", "step", _size(rng, 1500, 4096), rng.randint(1, 8), points="mesh", kernel="helmholtz",
                  singularity=0.1, theta=1.0, eps=1e-10, op_samples=0, rank=50, samples=0,
                  precision=rng.choice(["fp32", "fp64"]))
        del c["name"]
        return c
    top = {"matvec": 100000, "precond": 131072, "factor": 65536, "operator": 20000, "solve": 32768, "step": 65536}[do]
    c = _case("", do, _size(rng, 2048, top), 1 if do == "operator" else rng.choice([1, 2, 4, 5, 8, 12, 16]))
    del c["name"]
    c["points"] = rng.choice(["cube", "cube", "mixture"])
    if c["points"] == "mixture":
        c["singularity"] = 1e-6  # row sums of the narrow clusters reach 1e6
    c["rank"] = rng.choice([64, 100, 128])
    c["samples"] = rng.choice([2000, 4000])
    c["matrix_free"] = do in ("matvec", "solve", "step") and rng.random() < 0.4
    if not c["matrix_free"] and c["nrhs"] == 16 and rng.random() < 0.25:
        c["nrhs"] = 20  # above the streaming applies' 16 columns; matrix-free products end there
    c["graph"] = do == "solve" and rng.random() < 0.5
    c["host"] = c["n"] <= 16384 and rng.random() < 0.5
    if do == "precond":
        c["precision"] = rng.choice(["fp64", "fp32", "fp32", "bf16"])
    elif do in ("factor", "solve", "step"):
        c["precision"] = rng.choice(["fp64", "fp32", "fp32"])
    return c


# ---------------------------------------------------------------- inputs


def _kernel(case):
    s = case["singularity"]
    return {"laplace": m.Laplace3D(s), "yukawa": m.Yukawa3D(s, 1.0), "helmholtz": m.Helmholtz3D(1.0, s)}[case["kernel"]]


def _geometry(case, seed):
    """Bodies in tree order, and the tree."""
    n, kind = case["n"], case["points"]
    levels = m.levels_for(n, LEAF)
    if kind == "mixture":
        b = gaussian_mixture_points(n, 32, seed)
        levels = max(levels, math.ceil(math.log2(n / LEAF)))  # leaves of 32 to 256 bodies
        return b, m.build_tree(b, levels, 32, LEAF)
    if kind == "cube":
        b = np.random.default_rng(seed).random((n, 3))
    elif kind == "sphere":
        b = unit_sphere_points(n, seed)
    else:  # the mesh is fixed: only its radius moves with the seed
        b = m.mesh_sphere(n, math.sqrt(n / (4.0 * math.pi)) * (1.0 + 0.01 * np.random.default_rng(seed).random()))
    return b, m.build_tree(b, levels)


def _vectors(case, seed):
    """nrhs columns, uniform in [0, 1) as the reference's, as rows."""
    rng = np.random.default_rng(seed + 7919)
    x = rng.random((case["nrhs"], case["n"]))
    return x + 1j * rng.random(x.shape) if case["kernel"] == "helmholtz" else x


def _operator(case, h, b, tree):
    h.set_option(L.OPT_SAMPLING, L.SAMPLING_SKETCH)
    h.set_option(L.OPT_MATRIX_FREE, int(case["matrix_free"]))
    A = m.H2MatrixSolver(h, _kernel(case), case["eps"], case["rank"], 0, tree, case["theta"], b,
                         samples=case["op_samples"], precision=L.FP64)
    h.set_option(L.OPT_SAMPLING, L.SAMPLING_STRIDED)
    h.set_option(L.OPT_MATRIX_FREE, 0)
    return A


def _preconditioner(case, h, b, tree):
    h.set_option(L.OPT_PRECOND_BF16, int(case["precision"] == "bf16"))
    M = m.H2MatrixSolver(h, _kernel(case), 0.0, case["rank"], 0, tree, case["theta"], b, samples=case["samples"],
                         precision=L.FP64 if case["precision"] == "fp64" else L.FP32)
    M.factorizeM()
    return M


def prepare(case, seed):
    b, tree = _geometry(case, seed)
    h = m.Handle(0)
    s = {"case": case, "h": h, "bodies": b, "tree": tree}
    do = case["do"]
    if do in ("matvec", "solve", "step"):
        s["A"] = _operator(case, h, b, tree)
    if do in ("precond", "solve"):
        s["M"] = _preconditioner(case, h, b, tree)
    h.trim()  # construction scratch, as the serving loop does
    x = _vectors(case, seed)
    if do in ("solve", "step"):  # B = K x_true
        x = np.ascontiguousarray(m.dense_matvec(h, _kernel(case), b, x.T).T)
    if case["host"]:
        s["in"] = np.asfortranarray(x.T)
    else:
        s["in"] = torch.from_numpy(x).cuda()
        s["x"] = torch.empty_like(s["in"])
        torch.cuda.synchronize()
    if case["graph"]:
        h.set_option(L.OPT_GRAPH_SOLVE, 1)
    return s


# ---------------------------------------------------------------- one pass


def _apply(s, solver, method):
    """X <- op(X) in place on a copy of the input, by host or device arrays."""
    if s["case"]["host"]:
        x = s["in"].copy(order="F")
        (solver.matVecMul if method == "matvec" else solver.solvePrecondition)(x)
        return x
    x = s["x"]
    x.copy_(s["in"])
    torch.cuda.current_stream().synchronize()  # the library works on its own stream
    getattr(solver, method + "_device")(x.data_ptr(), s["case"]["nrhs"], _ld(s))
    s["h"].synchronize()
    return x


def _ld(s):
    return s["case"]["n"] * (2 if s["case"]["kernel"] == "helmholtz" else 1)


def _solve(s, M):
    if s["case"]["host"]:
        x = np.zeros_like(s["in"])
        s["A"].solveGMRES(TOL, M, x, s["in"], 10, 50, early_exit=True)
        return x
    x = s["x"]
    x.zero_()
    torch.cuda.current_stream().synchronize()
    s["A"].gmres_device(M, TOL, x.data_ptr(), s["in"].data_ptr(), s["case"]["nrhs"], _ld(s), 10, 50, True)
    return x


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "matvec":
        return _apply(state, state["A"], "matvec")
    if do == "precond":
        return _apply(state, state["M"], "precondition")
    if do == "solve":
        return _solve(state, state["M"])
    if do == "operator":
        A = _operator(case, state["h"], state["bodies"], state["tree"])
        y = _apply(state, A, "matvec")
        A.close()
        return y
    M = _preconditioner(case, state["h"], state["bodies"], state["tree"])
    x = _apply(state, M, "precondition") if do == "factor" else _solve(state, M)
    M.close()
    return x


# ---------------------------------------------------------------- what a pass cannot do without


@functools.lru_cache(maxsize=64)
def _pairs(n, points, theta):
    """Leaf size, near pairs and far pairs per level of such a tree (unordered pairs halve them)."""
    b, tree = _geometry({"n": n, "points": points}, 0)
    near, far = m.pair_csr("N", tree, theta)[0], m.pair_csr("F", tree, theta)[0]
    at = [(1 << l) - 1 for l in range(tree.levels + 2)]
    return (n / (1 << tree.levels), [int(near[at[l + 1]] - near[at[l]]) for l in range(tree.levels + 1)],
            [int(far[at[l + 1]] - far[at[l]]) for l in range(tree.levels + 1)])


def _work_matvec(case, leaf, near, far):
    # Operator ranks are about 150 at these accuracies.  K is symmetric: a pair's block is read once.
    w = 2 if case["kernel"] == "helmholtz" else 1
    r, leaf, nodes = 150.0 * w, leaf * w, [1 << l for l in range(len(near))]
    has = [any(far[: l + 1]) for l in range(len(near))]
    blocks = near[-1] * leaf * leaf + sum(far) * r * r
    bases = sum(nodes[l] * min(leaf if l == len(near) - 1 else 2 * r, 4 * r) * r for l in range(len(near)) if has[l])
    nr = case["nrhs"]
    flops = 2.0 * nr * (blocks + 2 * bases) + (10.0 * blocks if case["matrix_free"] else 0.0)
    stored = 3.0 * case["n"] + bases if case["matrix_free"] else 0.5 * (near[-1] + nodes[-1]) * leaf * leaf \
        + 0.5 * sum(far) * r * r + bases
    return 8.0 * stored + 16.0 * w * case["n"] * nr, flops


def _levels_of_m(case, leaf, near):
    """(boxes, near pairs, box size M, rank) per level of the fixed-rank preconditioner."""
    w = 2 if case["kernel"] == "helmholtz" else 1
    out, size = [], leaf * w
    for l in range(len(near) - 1, -1, -1):
        r = min(size, case["rank"] * w) if l else 0
        out.append((1 << l, near[l], size, r))
        size = 2.0 * r
    return out


def _work_precond(case, leaf, near):
    e = {"fp64": 8.0, "fp32": 4.0, "bf16": 2.0}[case["precision"]]
    w = 2 if case["kernel"] == "helmholtz" else 1
    elems = sum(2.0 * b * M * M + 2.0 * p * r * (M - r) for b, p, M, r in _levels_of_m(case, leaf, near))
    return e * elems + 16.0 * w * case["n"] * case["nrhs"], 2.0 * case["nrhs"] * elems


def _work_factor(case, leaf, near):
    e = 8.0 if case["precision"] == "fp64" else 4.0
    samples = float(case["samples"] or case["n"])
    elems = flops = 0.0
    for b, p, M, r in _levels_of_m(case, leaf, near):
        q, off = M - r, p - b
        elems += 2.0 * b * M * M + p * M * M
        if r:  # samples' Gram matrix or QR, interpolation, orthogonal completion
            flops += b * (samples * M * M + 2.0 * M * M * r + 4.0 * M * M * r)
        flops += b * (4.0 * M ** 3 + 2.0 / 3.0 * q ** 3 + 2.0 * q * q * M + 2.0 * q * M * r + 2.0 * r * r * q)
        flops += off * (2.0 * M ** 3 + 2.0 * M * (r * M + q * r) + 6.0 * r * r * q)
    return e * elems + 24.0 * case["n"], flops


def work(case):
    leaf, near, far = _pairs(case["n"], case["points"], case["theta"])
    do = case["do"]
    if do == "matvec":
        b, f = _work_matvec(case, leaf, near, far)
    elif do == "precond":
        b, f = _work_precond(case, leaf, near)
    elif do == "factor":
        b, f = (x + y for x, y in zip(_work_factor(case, leaf, near), _work_precond(case, leaf, near)))
    elif do == "operator":
        # Far-field sketch (box size squared times its far list), pivoted QR, blocks written, one product.
        b, f = _work_matvec(case, leaf, near, far)
        f += (1 << (len(near) - 1)) * 2.0 * leaf * leaf * (case["op_samples"] or case["n"]) * 2.0
    else:
        # Products and preconditioner solves of the fewest steps such a solve takes (about 8 and 12).
        mv, pc = _work_matvec(case, leaf, near, far), _work_precond(case, leaf, near)
        b, f = 8 * mv[0] + 12 * pc[0], 8 * mv[1] + 12 * pc[1]
        if do == "step":
            fb, ff = _work_factor(case, leaf, near)
            b, f = b + fb, f + ff
    return {"bytes": b, "flops": f}


def tolerance(case):
    """About four times what was measured (2-norm, largest) over the listed and 14 drawn cases."""
    if case["do"] in ("matvec", "operator"):
        # Against the dense product, which any operator of this accuracy is as far from: up to 1e-8, 2.5e-6 at eps 1e-8.
        return {"rel": 4.0 * case["eps"], "max": 1e3 * case["eps"]}
    if case["do"] in ("solve", "step"):
        # Against the known solution, at the operator's accuracy: up to 2.2e-7, 6.7e-5 at eps 1e-8 (contractions in
        # another order on the same operator: up to 1.4e-9).
        return {"rel": 100.0 * case["eps"], "max": 3e4 * case["eps"]}
    # Against contractions in FP32 sums and bases by another factorization: fp64 up to 1.6e-7, 6.9e-6; fp32 up to
    # 4.3e-5, 3.4e-3; bf16 up to 9.4e-4, 1.9e-2.
    return {"fp64": {"rel": 7e-7, "max": 3e-5}, "fp32": {"rel": 2e-4, "max": 1.4e-2},
            "bf16": {"rel": 4e-3, "max": 8e-2}}[case["precision"]]


# ---------------------------------------------------------------- what it comes to in 64 bits


def _dense(case, b, x):
    """K x by dense FP64 products of row chunks (real kernels)."""
    p = torch.from_numpy(b).cuda()
    x = torch.from_numpy(x).cuda()
    y = torch.empty_like(x)
    n, step = case["n"], max(1, (1 << 27) // case["n"])
    for i in range(0, n, step):
        d = torch.zeros(min(step, n - i), n, dtype=torch.float64, device="cuda")
        for k in range(3):
            d += (p[i:i + step, k, None] - p[None, :, k]) ** 2
        d.sqrt_()
        v = torch.exp(-d).div_(d) if case["kernel"] == "yukawa" else 1.0 / d
        v[d == 0] = 1.0 / case["singularity"]
        y[:, i:i + step] = (v @ x.T).T
    return y.cpu().numpy()


def exact(case, seed):
    """The dense product that an operator approximates, or the known solution of a solve.  A fixed-rank
    preconditioner is defined by its own construction: there is no such value for its solve."""
    if case["do"] in ("precond", "factor"):
        return None
    x = _vectors(case, seed)
    if case["do"] in ("matvec", "operator"):
        x = _dense(case, _geometry(case, seed)[0], x)
    return np.asfortranarray(x.T) if case["host"] else torch.from_numpy(np.ascontiguousarray(x))
