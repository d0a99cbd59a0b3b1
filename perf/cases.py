"""The calls that a user of this framework makes, as cases to be timed.

Every case goes through a public entry point: the Python module's functions
with host arrays, or the C ABI's device entry points with device buffers.

  call      compute_sparse_{eri,erida}_gausslet_integrals: enumeration, tables
            and values in one Python call (host arrays out)
  values    gli_b200_sparse_values_dev: the values of a class list that is kept
            on the device (the whole list, or one rank's range of it)
  nuclear   gli_b200_nuclear_batch_dev: nuclear matrices of one geometry, or of
            a batch of geometries, each on its own grid
  project   SparseERI.project: the ERI tensor in an orbital basis
  apply     SparseERI.apply: the ERI tensor applied to two-particle states
  kinetic   gli_b200_kinetic_matrix_noalloc: the dense kinetic matrix

Coefficients are the G10 gausslet set with a relative noise of 1e-3 from the
seed (a coefficient set of another fit); geometries, orbitals and states are
drawn from the seed.
"""
import ctypes as C
import math

import numpy as np
import torch

import gausslectronitegrate_b200 as gli
from gausslectronitegrate_b200 import _abi
from gausslectronitegrate_b200.workloads import dense_rows_in_sparse, sym_grid

G10 = np.load("tests/golden/reference_fixtures.npz")["g10"]
FORMS = {"fp64": _abi.GLI_FORM_FP64, "mixed": _abi.GLI_FORM_MIXED}
KINDS = {"erida": _abi.GLI_KIND_ERIDA, "eri": _abi.GLI_KIND_ERI}
# classes of the complete lists, by (kind, points per axis)
ERI_CLASSES = {3: 1027, 5: 138187, 7: 3571977}


def listed():
    return [
        # the smallest whole call: a minimal-grid ERI tensor, all latency
        dict(name="eri3_call", do="call", kind="eri", edge=3, form="fp64", tol=1e-16),
        # an ordinary whole call: the diagonal approximation on a 33^3 grid
        dict(name="erida33_call", do="call", kind="erida", edge=33, form="fp64", tol=1e-16),
        # the largest diagonal-approximation grid, in both forms
        dict(name="erida129_fp64", do="values", kind="erida", edge=129, form="fp64", tol=1e-16, lo=0.0, hi=1.0),
        dict(name="erida129_mixed", do="values", kind="erida", edge=129, form="mixed", tol=1e-16, lo=0.0, hi=1.0),
        # the headline workload: every ERI class of the 7^3 grid, in both forms
        dict(name="eri7_fp64", do="values", kind="eri", edge=7, form="fp64", tol=1e-16, lo=0.0, hi=1.0),
        dict(name="eri7_mixed", do="values", kind="eri", edge=7, form="mixed", tol=1e-16, lo=0.0, hi=1.0),
        # one molecule on a ragged box
        dict(name="nuclear_one", do="nuclear", grids="13x16x11", nuclei=5, form="fp64", tol=1e-8),
        # a batch of geometries on grids from 8^3 to 24^3
        dict(name="nuclear_batch", do="nuclear",
             grids="24x24x24 8x8x8 21x21x21 11x11x11 18x18x18 13x13x13 16x16x16 9x9x9", nuclei=6, form="fp64",
             tol=1e-8),
        # 32 orbitals on the 6^3 points inside the 7^3 class list
        dict(name="project_eri6", do="project", edge=7, dense="6x6x6", states=32, tol=1e-16),
        # 20 orbitals on all of the 7^3 points
        dict(name="project_eri7", do="project", edge=7, dense="7x7x7", states=20, tol=1e-16),
        # the tensor applied to a few two-particle states (an iterative solver's step)
        dict(name="apply_eri5", do="apply", edge=5, states=4, tol=1e-16),
        # the one-particle matrix of a large grid
        dict(name="kinetic24", do="kinetic", grid="24x24x24"),
    ]


def draw(rng):
    do = rng.choice(["call", "values", "values", "values", "nuclear", "nuclear", "project", "apply", "kinetic"])
    tol = 10.0 ** rng.uniform(-16, -5)
    form = rng.choice(["fp64", "mixed"])
    odd_edge = lambda lo, hi: 2 * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2 - 0.5)) + 1  # noqa: E731
    if do == "call":
        if rng.random() < 0.5:
            return dict(do=do, kind="eri", edge=rng.choice([3, 5]), form=form, tol=tol)
        return dict(do=do, kind="erida", edge=odd_edge(3, 65), form=form, tol=tol)
    if do == "values":
        # a whole list, or the contiguous range of one rank of several
        ranks = rng.choice([1, 1, 2, 3, 5, 8])
        r = rng.randrange(ranks)
        part = dict(lo=r / ranks, hi=(r + 1) / ranks)
        if rng.random() < 0.5:
            return dict(do=do, kind="eri", edge=rng.choice([3, 5, 7, 7]), form=form, tol=tol, **part)
        return dict(do=do, kind="erida", edge=min(129, odd_edge(9, 129)), form=form, tol=tol, **part)
    if do == "nuclear":
        count, grids, entries = rng.choice([1, 1, 2, 4, 7]), [], 0
        cubes = rng.random() < 0.5
        for _ in range(count):
            n = [rng.randint(6, 24) for _ in range(3)]
            n = [n[0]] * 3 if cubes else n
            entries += (n[0] * n[1] * n[2]) ** 2
            if grids and entries > 3.3e8:
                break
            grids.append("%dx%dx%d" % tuple(n))
        return dict(do=do, grids=" ".join(grids), nuclei=rng.randint(1, 9), form=form, tol=10.0 ** rng.uniform(-12, -5))
    if do == "project":
        edge = rng.choice([3, 5, 7])
        n = [rng.randint(max(1, edge - 3), edge) for _ in range(3)]
        return dict(do=do, edge=edge, dense="%dx%dx%d" % tuple(n), states=rng.randint(3, 20 if edge == 7 else 32), tol=tol)
    if do == "apply":
        return dict(do=do, edge=rng.choice([3, 5, 5]), states=rng.randint(1, 4), tol=tol)
    while True:
        n = [rng.randint(5, 40) for _ in range(3)]
        if n[0] * n[1] * n[2] <= 24 ** 3:
            return dict(do=do, grid="%dx%dx%d" % tuple(n))


# ---------------------------------------------------------------------------
# inputs

def _box(text):
    return [int(v) for v in text.split("x")]


def _centred(n):
    return [(-(k // 2), k) for k in n]


def _coeffs(seed):
    h = (G10.size - 1) // 2
    noise = 1e-3 * np.random.default_rng(seed).standard_normal(h + 1)
    return np.ascontiguousarray(G10 * (1.0 + np.concatenate([noise[:0:-1], noise])))


def _gdata(b):
    g = _abi.GaussletData()
    g.coefficients = b.ctypes.data_as(_abi.dptr)
    g.indices.num = b.size
    g.indices.istart = -(b.size - 1) // 2
    return g


def _grid(spec):
    g = _abi.Grid()
    for a in range(3):
        g.coord_range[a].istart, g.coord_range[a].num = spec[a]
    return g


def _check(rc):
    if rc != 0:
        raise RuntimeError(gli.lib().gli_b200_last_error_message().decode())


def _class_list(kind, spec):
    """The grid's class list as a device tensor."""
    L, d, n = gli.lib(), C.c_void_p(), C.c_int64()
    _check(L.gli_b200_enumerate_dev(KINDS[kind], C.byref(_grid(spec)), C.byref(d), C.byref(n), None))

    class Raw:
        __cuda_array_interface__ = {"data": (d.value, False), "shape": (n.value,), "typestr": "<i8", "version": 2}
    idx = torch.as_tensor(Raw(), device="cuda").clone()
    torch.cuda.synchronize()
    _check(L.gli_b200_free_dev(d, None))
    return idx


def _range(case, n):
    return int(round(case["lo"] * n)), int(round(case["hi"] * n))


def _nuclei(case, seed):
    """Nuclei of every instance: positions in the middle of its box, charges 1 to 8."""
    rng = np.random.default_rng(seed + 1)
    out = []
    for text in case["grids"].split():
        spec = _centred(_box(text))
        pos = np.stack([s + (n - 1) * (0.5 + 0.25 * rng.uniform(-1, 1, case["nuclei"])) for s, n in spec], axis=1)
        out.append((spec, pos, rng.integers(1, 9, case["nuclei"])))
    return out


def _basis(case, seed):
    """Orthonormal orbitals on the dense sub-grid, zero on the other points."""
    n, sparse = _box(case["dense"]), sym_grid(case["edge"])
    dense = [(-(case["edge"] // 2), k) for k in n]
    rows = dense_rows_in_sparse(sparse, dense)
    m = case["states"]
    a = np.random.default_rng(seed + 2).standard_normal((rows.size, m))
    q = np.linalg.qr(a)[0] if m <= rows.size else a / math.sqrt(rows.size)
    full = np.zeros((case["edge"] ** 3, m))
    full[rows] = q
    return full


def _states(case, seed):
    v = np.random.default_rng(seed + 3).standard_normal((case["edge"] ** 6, case["states"]))
    return v / np.linalg.norm(v, axis=0)


def prepare(case, seed):
    b = _coeffs(seed)
    st = dict(case=case, b=b, g=_gdata(b), L=gli.lib())
    do = case["do"]
    if do == "call":
        st["spec"] = sym_grid(case["edge"])
    elif do == "values":
        spec = sym_grid(case["edge"])
        idx = _class_list(case["kind"], spec)
        lo, hi = _range(case, idx.numel())
        st.update(grid=_grid(spec), idx=idx[lo:hi].clone(), out=torch.empty(hi - lo, dtype=torch.float64, device="cuda"))
    elif do == "nuclear":
        inst = _nuclei(case, seed)
        n = len(inst)
        arr = (_abi.Nucleus * (n * case["nuclei"]))()
        outs = []
        for k, (spec, pos, q) in enumerate(inst):
            for j in range(case["nuclei"]):
                arr[k * case["nuclei"] + j].pos[:] = [float(v) for v in pos[j]]
                arr[k * case["nuclei"] + j].charge = int(q[j])
            N = spec[0][1] * spec[1][1] * spec[2][1]
            outs.append(torch.empty((N, N), dtype=torch.float64, device="cuda"))
        st.update(n=n, grids=(_abi.Grid * n)(*[_grid(s) for s, _, _ in inst]), nuclei=arr, outs=outs,
                  offsets=np.arange(n + 1, dtype=np.int64) * case["nuclei"],
                  ptrs=(C.c_void_p * n)(*[o.data_ptr() for o in outs]))
    elif do in ("project", "apply"):
        st["eri"] = gli.compute_sparse_eri_gausslet_integrals(b, sym_grid(case["edge"]), case["tol"])
        st["x"] = _basis(case, seed) if do == "project" else _states(case, seed)
    else:
        spec = _centred(_box(case["grid"]))
        N = spec[0][1] * spec[1][1] * spec[2][1]
        st.update(grid=_grid(spec), db=torch.tensor(b, device="cuda"),
                  out=torch.empty((N, N), dtype=torch.float64, device="cuda"))
    return st


def run(st):
    case, L = st["case"], st["L"]
    do = case["do"]
    if do == "call":
        fn = getattr(gli, f"compute_sparse_{case['kind']}_gausslet_integrals")
        s = fn(st["b"], st["spec"], case["tol"], form=case["form"])
        return {"indices": s.indices, "values": s.values}
    if do == "values":
        _check(L.gli_b200_sparse_values_dev(KINDS[case["kind"]], st["g"].coefficients, st["b"].size, C.byref(st["grid"]),
                                            C.c_void_p(st["idx"].data_ptr()), st["idx"].numel(), case["tol"],
                                            FORMS[case["form"]], C.c_void_p(st["out"].data_ptr()), None))
        return st["out"]
    if do == "nuclear":
        _check(L.gli_b200_nuclear_batch_dev(C.byref(st["g"]), st["n"], st["grids"], st["offsets"].ctypes.data_as(_abi.lptr),
                                            st["nuclei"], case["tol"], FORMS[case["form"]], st["ptrs"], None))
        return st["outs"]
    if do == "project":
        return st["eri"].project(st["x"])
    if do == "apply":
        return st["eri"].apply(st["x"])
    _check(L.gli_b200_kinetic_matrix_noalloc(C.c_void_p(st["db"].data_ptr()), st["b"].size, C.byref(st["grid"]),
                                             C.c_void_p(st["out"].data_ptr()), None))
    return st["out"]


# ---------------------------------------------------------------------------
# work that a pass cannot do without

def _classes(kind, edge):
    if kind == "eri":
        return ERI_CLASSES[edge]
    e = edge - 1  # displacements |dx| >= |dy| >= |dz| up to the grid's length
    return (e + 1) * (e + 2) * (e + 3) // 6


def _value_flops(kind, edge, classes):
    """The separable lattice sums over the weights' supports, shared by the classes of equal axis keys."""
    half = 80 if kind == "erida" else 104
    keys = edge if kind == "erida" else (edge * (edge + 1) // 2) * (2 * edge - 1) // 3
    U = (3 if kind == "erida" else 6) * (edge - 1) + half + 1
    band = min(U, 2 * half + 1)
    return 2.0 * (keys * (U * U / 4.0) * band + keys * keys / 2.0 * U * band + min(classes, keys ** 3 / 6) * band)


def work(case):
    do = case["do"]
    if do in ("call", "values"):
        n = _classes(case["kind"], case["edge"])
        if do == "values":
            lo, hi = _range(case, n)
            n = max(1, hi - lo)
        return {"bytes": 16.0 * n, "flops": _value_flops(case["kind"], case["edge"], n)}
    if do == "nuclear":
        by, fl = 0.0, 0.0
        for text in case["grids"].split():
            n = _box(text)
            U, k = [6 * (v - 1) + 99 for v in n], [v * (v + 1) // 2 for v in n]
            by += 8.0 * (n[0] * n[1] * n[2]) ** 2
            fl += 2.0 * 99 * (k[2] * U[0] * U[1] + k[2] * k[1] * U[0] + k[0] * k[1] * k[2])
            fl += 10.0 * case["nuclei"] * U[0] * U[1] * U[2]
        return {"bytes": by, "flops": fl}
    m = ERI_CLASSES[case["edge"]] if "edge" in case else 0
    if do == "project":
        n, M = _box(case["dense"]), case["states"]
        N, pairs = n[0] * n[1] * n[2], math.prod(v * (v + 1) // 2 for v in n)
        # per distinct coordinate pair: half of a symmetric N x N matrix times the orbitals, then
        # onto the orbital pairs; then the second pair of indices
        return {"bytes": 16.0 * m + 8.0 * case["edge"] ** 3 * M + 8.0 * M ** 4,
                "flops": 1.0 * pairs * N * N * M + 1.0 * pairs * N * M * M + 0.5 * pairs * M ** 4}
    if do == "apply":
        N = case["edge"] ** 3
        return {"bytes": 16.0 * m + 16.0 * N * N * case["states"], "flops": 2.0 * N ** 4 * case["states"]}
    n = _box(case["grid"])
    return {"bytes": 8.0 * (n[0] * n[1] * n[2]) ** 2, "flops": 0.0}


# ---------------------------------------------------------------------------
# the same in 64 bits, from the defining sums (torch, no code of this repository)

def _factors(b, L, tol=None):
    """F_s[m]: Gaussian-pair factors of coordinate difference s at offset m (sixths of a unit)."""
    nb = b.size
    i = np.arange(nb)
    F = np.zeros((L, 2 * nb - 1))
    for s in range(L):
        M = math.sqrt(math.pi) / 3 * np.outer(b, b) * np.exp(-(0.5 * (3 * s + i[:, None] - i[None, :])) ** 2)
        flip = M[:, ::-1]
        for m in range(2 * nb - 1):
            F[s, m] = np.trace(flip, offset=nb - 1 - m)
    if tol is not None:
        F[np.abs(F) <= tol] = 0.0
    return F


def _lattice(kind, b, L, tol):
    """Folded weights W[key][u] and the Coulomb table's parameters."""
    nb = b.size
    if kind == "erida":
        P = [2 * math.pi / 9 * np.convolve(b, b[::-1])]
        keys = [(0, 3 * d) for d in range(L)]
        half = nb - 1
    else:
        F = _factors(b, L)
        P = [np.convolve(F[lo], F[hi][::-1]) for hi in range(L) for lo in range(hi + 1)]
        keys = [(p, 3 * c) for p in range(len(P)) for c in range(2 * L - 1)]
        half = 2 * nb - 2
    P = np.array(P)
    P[np.abs(P) <= tol] = 0.0
    pos = np.arange(-half, half + 1)
    used = np.abs(pos)[np.any(P != 0, axis=0)]
    U = max(c for _, c in keys) + (int(used.max()) if used.size else 0) + 1
    W = np.zeros((len(keys), U))
    for k, (p, c) in enumerate(keys):
        u = np.abs(pos + c)
        ok = (P[p] != 0) & (u < U)
        np.add.at(W[k], u[ok], P[p][ok])
    return torch.tensor(W, device="cuda"), U


def _key_values(kind, b, L, tol):
    """V[kx][ky][kz]: the integral of three axis keys."""
    W, U = _lattice(kind, b, L, tol)
    n = torch.arange(3 * (U - 1) ** 2 + 1, device="cuda", dtype=torch.float64)
    r = torch.sqrt(n)
    r[0] = 1.0
    T = torch.erf(r * 0.35355339059327376220) * 6.0 / r if kind == "eri" else torch.erf(r * 0.5) * 3.0 / r
    T[0] = 3.0 * math.sqrt(2.0 / math.pi) if kind == "eri" else 3.0 / math.sqrt(math.pi)
    u = torch.arange(U, device="cuda")
    H = torch.empty((W.shape[0], U, U), dtype=torch.float64, device="cuda")  # [key][u][v]
    for v in range(U):
        H[:, :, v] = W @ T[u[:, None] ** 2 + u[None, :] ** 2 + v * v].T
    H2 = torch.matmul(H, W.T)                        # [key a][u][key b]
    return torch.matmul(H2.transpose(1, 2), W.T)      # [key a][key b][key c]


def _points(spec):
    ax = [torch.arange(s, s + n, device="cuda") for s, n in spec]
    return torch.stack([g.reshape(-1) for g in torch.meshgrid(*ax, indexing="ij")], dim=1)


def _eri_key(d1, s1, d2, s2, L):
    lo, hi = torch.minimum(d1, d2), torch.maximum(d1, d2)
    return (hi * (hi + 1) // 2 + lo) * (2 * L - 1) + (s1 - s2).abs()


def _exact_values(kind, b, L, tol, idx):
    V, p = _key_values(kind, b, L, tol), _points(sym_grid(L))
    N = p.shape[0]
    out = torch.empty(idx.numel(), dtype=torch.float64, device="cuda")
    for c in range(0, idx.numel(), 1 << 20):
        x = idx[c:c + (1 << 20)]
        if kind == "erida":
            k = (p[x // N] - p[x % N]).abs()
        else:
            i, j, m, n = p[x // N ** 3], p[x // N ** 2 % N], p[x // N % N], p[x % N]
            k = _eri_key((i - j).abs(), i + j, (m - n).abs(), m + n, L)
        out[c:c + (1 << 20)] = V[k[:, 0], k[:, 1], k[:, 2]]
    return out


def _exact_nuclear(b, spec, pos, q, tol):
    F = _factors(b, max(n for _, n in spec), tol)
    nz = np.nonzero(np.any(F != 0, axis=0))[0] - (b.size - 1)
    h = int(np.abs(nz).max())
    W, ax, key = [], [], []
    for s, n in spec:
        U = 6 * (n - 1) + 2 * h + 1
        w = np.zeros((n * (n + 1) // 2, U))
        tri = np.zeros((n, n), dtype=np.int64)
        for hi in range(n):
            for lo in range(hi + 1):
                k = hi * (hi + 1) // 2 + lo
                tri[lo, hi] = tri[hi, lo] = k
                w[k, 3 * (lo + hi):3 * (lo + hi) + 2 * h + 1] = F[hi - lo, b.size - 1 - h:b.size + h]
        W.append(torch.tensor(w, device="cuda"))
        ax.append(torch.arange(6 * s - h, 6 * s - h + U, device="cuda", dtype=torch.float64) / 6.0)
        key.append(torch.tensor(tri, device="cuda"))
    phi = torch.zeros([a.numel() for a in ax], dtype=torch.float64, device="cuda")
    for k in range(len(q)):
        r = torch.sqrt((ax[0] - pos[k][0])[:, None, None] ** 2 + (ax[1] - pos[k][1])[None, :, None] ** 2 +
                       (ax[2] - pos[k][2])[None, None, :] ** 2)
        phi += float(q[k]) * torch.where(r > 0, torch.erf(3.0 * r) / r, 6.0 / math.sqrt(math.pi))
    V = torch.einsum("uvt,kt->uvk", phi, W[2])
    V = torch.einsum("uvk,jv->ujk", V, W[1])
    V = torch.einsum("ujk,iu->ijk", V, W[0])
    nx, ny, nzz = (n for _, n in spec)
    V = V[key[0][:, None, None, :, None, None], key[1][None, :, None, None, :, None], key[2][None, None, :, None, None, :]]
    return V.reshape(nx * ny * nzz, nx * ny * nzz)


def _pair_classes(spec):
    """Of every ordered point pair: the class of equal per-axis |difference| and sum, and the classes' fields."""
    p = _points(spec)
    d, s = (p[:, None] - p[None, :]).abs(), p[:, None] + p[None, :]
    f = torch.stack([d, s], dim=-1).reshape(-1, 6)
    cls, inv = torch.unique(f, dim=0, return_inverse=True)
    return cls.reshape(-1, 3, 2), inv


def _exact_pair_rows(V, cls, c, L):
    a = cls[c][:, None]
    k = [_eri_key(a[..., x, 0], a[..., x, 1], cls[None, :, x, 0], cls[None, :, x, 1], L) for x in range(3)]
    return V[k[0], k[1], k[2]]


def exact(case, seed):
    do, b = case["do"], _coeffs(seed)
    if do == "call":
        idx = _class_list(case["kind"], sym_grid(case["edge"]))
        return {"indices": None, "values": _exact_values(case["kind"], b, case["edge"], case["tol"], idx).cpu().numpy()}
    if do == "values":
        idx = _class_list(case["kind"], sym_grid(case["edge"]))
        lo, hi = _range(case, idx.numel())
        return _exact_values(case["kind"], b, case["edge"], case["tol"], idx[lo:hi])
    if do == "nuclear":
        return [_exact_nuclear(b, spec, pos, q, case["tol"]) for spec, pos, q in _nuclei(case, seed)]
    if do == "project":
        L, M = case["edge"], case["states"]
        V = _key_values("eri", b, L, case["tol"])
        dense = [(-(L // 2), k) for k in _box(case["dense"])]
        B = torch.tensor(_basis(case, seed)[dense_rows_in_sparse(sym_grid(L), dense)], device="cuda")
        cls, inv = _pair_classes(dense)
        D = torch.zeros((cls.shape[0], M * M), dtype=torch.float64, device="cuda")
        D.index_add_(0, inv, (B[:, None, :, None] * B[None, :, None, :]).reshape(-1, M * M))
        E = torch.zeros((M * M, M * M), dtype=torch.float64, device="cuda")
        for c in range(0, cls.shape[0], 512):
            E += D[c:c + 512].T @ (_exact_pair_rows(V, cls, slice(c, c + 512), L) @ D)
        return E.reshape(M, M, M, M).cpu().numpy()
    if do == "apply":
        L, N = case["edge"], case["edge"] ** 3
        V = _key_values("eri", b, L, case["tol"])
        cls, inv = _pair_classes(sym_grid(L))
        x = torch.tensor(_states(case, seed), device="cuda").reshape(N, N, -1)     # [j][l][s]
        Vc = torch.cat([_exact_pair_rows(V, cls, slice(c, c + 256), L) for c in range(0, cls.shape[0], 256)])
        inv = inv.reshape(N, N)
        out = torch.zeros((N, N, x.shape[2]), dtype=torch.float64, device="cuda")
        for i in range(N):
            for j in range(N):
                out[i] += Vc[inv[i, j]][inv] @ x[j]
        return out.reshape(N * N, -1).cpu().numpy()
    spec = _centred(_box(case["grid"]))
    i = np.arange(b.size)
    K, I = [], [torch.eye(n, dtype=torch.float64, device="cuda") for _, n in spec]
    for _, n in spec:
        d = 3 * np.arange(n)[:, None, None] + i[None, :, None] - i[None, None, :]
        g = 1.5 * math.sqrt(math.pi) * (1 - 0.5 * d ** 2) * np.exp(-0.25 * d ** 2)
        k1 = torch.tensor(0.5 * np.einsum("i,j,sij->s", b, b, g), device="cuda")
        t = torch.arange(n, device="cuda")
        K.append(k1[(t[:, None] - t[None, :]).abs()])
    kron = lambda a, c, d: torch.kron(torch.kron(a, c), d)  # noqa: E731
    return kron(K[0], I[1], I[2]) + kron(I[0], K[1], I[2]) + kron(I[0], I[1], K[2])
