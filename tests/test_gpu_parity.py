"""GPU parity against the oracle: bit-exact sparsity pattern and pair set, FP64 values within
rounding, deterministic runs. All calls go through the C ABI (libnlfem_gpu.so)."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp

from conftest import conf2d, conf3d, square_mesh, cube_mesh, labeled_mesh, rel_errors, same_pattern

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-12   # relative Frobenius / max-entry error of the FP64 path (summation order only)


@pytest.fixture(scope="module")
def nl():
    from nlfem_gb300 import nlfem, _lib
    lib = _lib.load()
    if lib.nlfem_device_count() == 0:
        pytest.fail("no CUDA device visible: the GPU library cannot run")
    return nlfem


@pytest.fixture(scope="module")
def orc():
    from oracle import oracle
    return oracle


def _cases_retri(rng, n):
    out = []
    for i in range(n):
        T = rng.uniform(-1, 1, 6)
        delta = rng.uniform(0.05, 1.5)
        mode = i % 4
        if mode == 0:
            x = rng.uniform(-1.5, 1.5, 2)
        elif mode == 1:   # center near a vertex
            k = rng.integers(3)
            x = T[2 * k: 2 * k + 2] + rng.normal(0, 1e-3, 2)
        elif mode == 2:   # ball tangent-ish to an edge
            k = rng.integers(3)
            p, q = T[2 * k: 2 * k + 2], T[(2 * k + 2) % 6: (2 * k + 2) % 6 + 2]
            m = 0.5 * (p + q)
            nrm = np.array([q[1] - p[1], p[0] - q[0]])
            nrm /= np.linalg.norm(nrm)
            x = m + nrm * delta * (1 + rng.normal(0, 1e-9))
        else:            # vertex exactly on the sphere
            k = rng.integers(3)
            ang = rng.uniform(0, 2 * np.pi)
            x = T[2 * k: 2 * k + 2] + delta * np.array([np.cos(ang), np.sin(ang)])
        out.append((x, T, delta * delta, int(rng.integers(2))))
    return out


def test_retriangulate_bitexact(nl, orc):
    rng = np.random.Generator(np.random.PCG64(7))
    cases = _cases_retri(rng, 4000)
    for caps in (0, 1):
        sub = [c for c in cases if c[3] == caps]
        X = np.array([c[0] for c in sub]); T = np.array([c[1] for c in sub])
        sq = np.array([c[2] for c in sub])
        for j in range(len(sub)):
            cnt, out = nl.retriangulate_batch(X[j:j + 1], T[j:j + 1], sq[j], caps)
            n, tri = orc.retriangulate_sq(X[j], T[j], sq[j], caps)
            assert cnt[0] == n
            np.testing.assert_array_equal(out[0, :n], tri)


def test_debug_hooks(nl, orc):
    T = np.array([0.1, 0.2, 0.9, 0.1, 0.3, 0.8])
    x = np.array([0.4, 0.35])
    p = nl.py_toRef(T, x)
    np.testing.assert_allclose(nl.py_toPhys(T, p), x, rtol=0, atol=1e-15)
    A = np.array([2.0, 1.0, 1.0, 3.0]); b = np.array([1.0, 2.0])
    np.testing.assert_allclose(nl.py_solve2x2(A, b), np.linalg.solve(A.reshape(2, 2), b), rtol=1e-15)
    n, lst = nl.py_retriangulate(np.array([0.3, 0.3]), T, 0.2, 1)
    m, tri = orc.retriangulate(np.array([0.3, 0.3]), T, 0.2, 1)
    assert n == m
    np.testing.assert_array_equal(lst[: 6 * n], tri.ravel())


KC = {"function": "constant", "horizon": 0.1, "outputdim": 1}


def test_pair_list_config1(nl, orc):
    m = square_mesh(32, 0.1)
    ref = orc.assemble(m, KC, conf2d(), want_pairs=True)
    got = nl.pair_list(m, KC, conf2d())
    rp = ref["pairs"][np.lexsort((ref["pairs"][:, 1], ref["pairs"][:, 0]))]
    np.testing.assert_array_equal(got, rp)


def test_config1_constant_fp64(nl, orc):
    m = square_mesh(32, 0.1)
    A = nl.stiffnessMatrix(m, KC, conf2d())
    B = orc.assemble(m, KC, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)


def test_jittered_parabola_fp64(nl, orc):
    m = square_mesh(20, 0.15, jitter=0.2, seed=4)
    k = {"function": "parabola", "horizon": 0.15, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf2d())
    B = orc.assemble(m, k, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)


def test_no_caps_and_full_search(nl, orc):
    m = square_mesh(8, 0.1, jitter=0.1, seed=2)
    c = conf2d(caps=0)
    A = nl.stiffnessMatrix(m, KC, c); B = orc.assemble(m, KC, c)["A"]
    assert same_pattern(A, B) and rel_errors(A, B)[0] < FP64_TOL
    c = conf2d(); c["is_fullConnectedComponentSearch"] = 1
    A = nl.stiffnessMatrix(m, KC, c); B = orc.assemble(m, KC, c)["A"]
    assert same_pattern(A, B) and rel_errors(A, B)[0] < FP64_TOL


def test_label_zero_bridges(nl, orc):
    m = square_mesh(14, 0.1, jitter=0.1, seed=5)
    lab = m["elementLabels"].copy()
    lab[40:60] = 0
    from nlfem_gb300.meshes import mesh_dict
    m2 = mesh_dict(m["vertices"], m["elements"], lab)
    A = nl.stiffnessMatrix(m2, KC, conf2d()); B = orc.assemble(m2, KC, conf2d())["A"]
    assert same_pattern(A, B) and rel_errors(A, B)[0] < FP64_TOL


@pytest.mark.parametrize("kern", ["constant", "parabola"])
def test_label_zero_bridges_mixed(nl, orc, kern):
    """Mixed path on a mesh with label-0 elements (searched through, never paired), with the
    constant kernel's closed forms and the general kernel."""
    m = square_mesh(16, 0.12, jitter=0.2, seed=7)
    lab = m["elementLabels"].copy()
    lab[60:90] = 0
    from nlfem_gb300.meshes import mesh_dict
    m2 = mesh_dict(m["vertices"], m["elements"], lab)
    k = {"function": kern, "horizon": 0.12, "outputdim": 1}
    A = nl.stiffnessMatrix(m2, k, conf2d(precision="mixed")); B = orc.assemble(m2, k, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


def test_mixed_no_caps(nl, orc):
    m = square_mesh(18, 0.1, jitter=0.2, seed=11)
    A = nl.stiffnessMatrix(m, KC, conf2d(caps=0, precision="mixed")); B = orc.assemble(m, KC, conf2d(caps=0))["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_domain_decomposition_weights(nl, orc, prec):
    """Domain decomposition (Cassemble.cpp:649-657): every pair's blocks weighted by 1 / the number
    of subdomains its elements share. Two subdomains overlap in a strip wider than the ball, so
    every interacting pair shares one; the first 20 elements lie in both (chk_Mesh, checks.cpp:74-84,
    requires them to share one pairwise)."""
    m = square_mesh(14, 0.1, jitter=0.1, seed=8)
    x = m["vertices"][m["elements"]].mean(axis=1)[:, 0]
    rows = [[0, 1] if e < 20 else ([0] if xi < 0.3 else ([1] if xi > 0.7 else [0, 1])) for e, xi in enumerate(x)]
    indptr = np.cumsum([0] + [len(r) for r in rows])
    Z = sp.csr_matrix((np.ones(indptr[-1]), np.concatenate(rows), indptr), shape=(len(rows), 2))
    m["nZeta"] = 2
    m["ZetaIndicator"] = Z
    A = nl.stiffnessMatrix(m, KC, conf2d(precision=prec))
    B = orc.assemble(m, KC, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    tol = FP64_TOL if prec == "fp64" else MIX_TOL
    assert fro < tol and mx < tol, (fro, mx)
    m0 = dict(m)
    m0["nZeta"] = 0
    B0 = orc.assemble(m0, KC, conf2d())["A"]
    assert abs(B - B0).max() > 1e-3 * abs(B0).max()   # the weights change the matrix


def test_pair_blocks_match_oracle(nl, orc):
    m = square_mesh(16, 0.1, jitter=0.2, seed=9)
    k = {"function": "parabola", "horizon": 0.1, "outputdim": 1}
    pairs = orc.assemble(m, k, conf2d(), want_pairs=True)["pairs"]
    rng = np.random.Generator(np.random.PCG64(3))
    sel = pairs[rng.choice(len(pairs), 500, replace=False)]
    g, gr = nl.pair_blocks(m, k, conf2d(), sel)
    o, orr = orc.pair_blocks(m, k, conf2d(), sel)
    np.testing.assert_array_equal(gr != 0, orr != 0)
    np.testing.assert_allclose(g, o, rtol=1e-12, atol=1e-12 * np.abs(o).max())


LABEL_KERNELS = ["labeled", "notch", "labeledNotch", "labeledValve", "constantTruncated"]


_labeled_mesh = labeled_mesh


@pytest.mark.parametrize("name,method", [(k, "retriangulate") for k in LABEL_KERNELS] + [("labeledValve", "baryCenter"), ("notch", "baryCenter")])
def test_label_kernels_fp64(nl, orc, name, method):
    """Label- and position-dependent kernels (model.cpp:30-42, 67-114) on the FP64 path."""
    m = _labeled_mesh()
    k = {"function": name, "horizon": 0.1, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf2d(method=method))
    B = orc.assemble(m, k, conf2d(method=method))["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    if name != "constantTruncated":   # the kernel matters: not the constant kernel's matrix
        C = orc.assemble(m, KC, conf2d(method=method))["A"]
        assert abs(B - C).max() > 1e-3 * abs(C).max()


def test_label_kernel_pair_blocks(nl, orc):
    m = _labeled_mesh(10, 6)
    k = {"function": "labeled", "horizon": 0.1, "outputdim": 1}
    pairs = orc.assemble(m, k, conf2d(), want_pairs=True)["pairs"]
    g, gr = nl.pair_blocks(m, k, conf2d(), pairs)
    o, orr = orc.pair_blocks(m, k, conf2d(), pairs)
    np.testing.assert_array_equal(gr != 0, orr != 0)
    np.testing.assert_allclose(g, o, rtol=1e-12, atol=1e-12 * np.abs(o).max())


def test_label_kernel_errors(nl):
    from nlfem_gb300._lib import NlfemError
    k = {"function": "labeled", "horizon": 0.1, "outputdim": 1}
    m = square_mesh(8, 0.1, jitter=0.1, seed=1)
    m["elementLabels"] = np.where(m["elementLabels"] > 0, 2, -1)   # 10 * 2 - 1 = 19: the reference aborts
    with pytest.raises(NlfemError, match="outside its domain"):
        nl.stiffnessMatrix(m, k, conf2d())
    with pytest.raises(NlfemError, match="fp64 path only"):
        nl.stiffnessMatrix(_labeled_mesh(8), k, conf2d(precision="mixed"))
    # the session still works after the error
    m = _labeled_mesh(8)
    assert nl.stiffnessMatrix(m, k, conf2d()).nnz > 0


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_tangent_sphere_polygons(nl, orc, prec):
    """Unjittered grid with h = 0.15 and delta = 0.1: element centroids lie at distance delta from
    grid lines, the sphere touches edges up to rounding, and some polygons would need more than 9
    points. Both sides keep the first 9."""
    m = square_mesh(8, 0.1)
    A = nl.stiffnessMatrix(m, KC, conf2d(precision=prec))
    B = orc.assemble(m, KC, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    tol = FP64_TOL if prec == "fp64" else 1e-6
    assert fro < tol and mx < tol, (fro, mx)


FURTHER_RULES = ["retriangulate_unsymm", "subSetBall", "averageBall", "baryCenterRT", "noTruncation"]


@pytest.mark.parametrize("method", FURTHER_RULES)
def test_further_rules_fp64(nl, orc, method):
    """retriangulate_unsymm, subSetBall, averageBall, baryCenterRT and noTruncation
    (integration.cpp:290-343, 542-704, 1021-1095, 1155-1249) on the FP64 path: assembled
    matrices, and the blocks and interaction flags of single pairs."""
    n = 6 if method == "noTruncation" else 14   # noTruncation pairs every element with every other
    m = square_mesh(n, 0.1, jitter=0.15, seed=12)
    conf = conf2d(method=method)
    for name in ("constant", "parabola"):
        k = {"function": name, "horizon": 0.1, "outputdim": 1}
        A = nl.stiffnessMatrix(m, k, conf)
        r = orc.assemble(m, k, conf, want_pairs=True)
        B = r["A"]
        assert same_pattern(A, B)
        fro, mx = rel_errors(A, B)
        assert fro < FP64_TOL and mx < FP64_TOL, (name, fro, mx)
    rng = np.random.Generator(np.random.PCG64(5))
    sel = r["pairs"][rng.choice(len(r["pairs"]), min(400, len(r["pairs"])), replace=False)]
    g, gr = nl.pair_blocks(m, k, conf, sel)
    o, orr = orc.pair_blocks(m, k, conf, sel)
    np.testing.assert_array_equal(gr != 0, orr != 0)
    np.testing.assert_allclose(g, o, rtol=1e-12, atol=1e-12 * np.abs(o).max())


def test_further_rules_with_label_kernel(nl, orc):
    m = _labeled_mesh(12, 7)
    k = {"function": "labeledValve", "horizon": 0.1, "outputdim": 1}
    for method in ("retriangulate_unsymm", "averageBall", "baryCenterRT"):
        A = nl.stiffnessMatrix(m, k, conf2d(method=method))
        B = orc.assemble(m, k, conf2d(method=method))["A"]
        assert same_pattern(A, B)
        fro, mx = rel_errors(A, B)
        assert fro < FP64_TOL and mx < FP64_TOL, (method, fro, mx)


def test_further_rules_mixed_precision_refused(nl):
    from nlfem_gb300._lib import NlfemError
    with pytest.raises(NlfemError, match="fp64 path only"):
        nl.stiffnessMatrix(square_mesh(6, 0.1), KC, conf2d(method="subSetBall", precision="mixed"))


def _conf_dg(method="retriangulate", precision="fp64"):
    c = conf2d(method=method, precision=precision)
    c["ansatz"] = "DG"
    return c


@pytest.mark.parametrize("kname,method", [("constant", "retriangulate"), ("parabola", "retriangulate"),
                                          ("constant", "baryCenter"), ("labeledValve", "retriangulate"),
                                          ("constant", "averageBall")])
def test_dg_matches_oracle(nl, orc, kname, method):
    """The DG ansatz (element DOFs dV e + a, every row kept; Cassemble.cpp:580-585, 637-642) on
    the FP64 path, and its sum over vertex copies against the CG assembly."""
    m = _labeled_mesh(10, 14) if kname.startswith("labeled") else square_mesh(10, 0.1, jitter=0.15, seed=14)
    k = {"function": kname, "horizon": 0.1, "outputdim": 1}
    A = nl.stiffnessMatrix(dict(m), k, _conf_dg(method))
    B = orc.assemble(m, k, _conf_dg(method))["A"]
    nE, nV = m["elements"].shape[0], m["vertices"].shape[0]
    assert A.shape == (3 * nE, 3 * nE)
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    C = nl.stiffnessMatrix(dict(m), k, conf2d(method=method))
    P = sp.csr_matrix((np.ones(3 * nE), (np.arange(3 * nE), m["elements"].ravel())), shape=(3 * nE, nV))
    S = (P.T @ A @ P).toarray()
    S[m["vertexLabels"] <= 0] = 0
    assert np.abs(S - C.toarray()).max() <= 1e-12 * abs(C).max()


@pytest.mark.parametrize("close,kname", [("weakSingular", "fractional"), ("weakSingular", "linearPrototypeMicroelastic")])
def test_dg_singular_kernels(nl, orc, close, kname):
    """DG with a singular kernel: the close pairs (sharing a vertex) take the weakSingular Duffy rule
    (the reference refuses the fractional rule for DG, checks.cpp:105-107), found on the vertex
    table while the rows are element DOFs (Cassemble.cpp:580-585, integration.cpp:82-185); against
    the oracle, and summed over the vertex copies against the CG assembly."""
    m = square_mesh(8, 0.2, jitter=0.1, seed=16)
    s = 0.4 if kname == "fractional" else -0.5
    k = {"function": kname, "horizon": 0.2, "outputdim": 1, "fractional_s": s}
    c = _conf_dg()
    c["closeElements"] = close
    c["quadrature"]["tensorGaussDegree"] = 3
    A = nl.stiffnessMatrix(dict(m), k, c)
    B = orc.assemble(m, k, c)["A"]
    nE, nV = m["elements"].shape[0], m["vertices"].shape[0]
    assert A.shape == (3 * nE, 3 * nE)
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < 1e-11 and mx < 1e-11, (fro, mx)
    cc = dict(c, ansatz="CG")
    C = nl.stiffnessMatrix(dict(m), k, cc)
    P = sp.csr_matrix((np.ones(3 * nE), (np.arange(3 * nE), m["elements"].ravel())), shape=(3 * nE, nV))
    S = (P.T @ A @ P).toarray()
    S[m["vertexLabels"] <= 0] = 0
    assert np.abs(S - C.toarray()).max() <= 1e-11 * abs(C).max()


def test_dg_load_vector(nl, orc):
    m = square_mesh(12, 0.1, jitter=0.2, seed=15)
    f = nl.loadVector(dict(m), {"function": "linear"}, _conf_dg())
    g = orc.assemble(m, None, _conf_dg(), compute="forcing", load={"function": "linear"})["f"]
    assert f.shape == (3 * m["elements"].shape[0],)
    np.testing.assert_allclose(f, g, rtol=1e-13, atol=1e-15 * np.abs(g).max())


def test_dg_session_reassembly_and_cache(nl, orc):
    """A DG session assembles again on its mesh (the row space goes back to the vertices for the
    pair search), and a CG call after a DG call on the same sizes is unchanged."""
    m = square_mesh(10, 0.1, jitter=0.1, seed=16)
    C0 = nl.stiffnessMatrix(dict(m), KC, conf2d())
    s = nl.Session([(dict(m), KC, _conf_dg())])
    s.assemble()
    A1 = s.download(0)
    s.assemble()
    A2 = s.download(0)
    assert same_pattern(A1, A2) and np.array_equal(A1.data, A2.data)
    B = orc.assemble(m, KC, _conf_dg())["A"]
    fro, mx = rel_errors(A1, B)
    assert fro < FP64_TOL and mx < FP64_TOL
    nl.stiffnessMatrix(dict(m), KC, _conf_dg())
    C1 = nl.stiffnessMatrix(dict(m), KC, conf2d())
    assert same_pattern(C0, C1) and np.array_equal(C0.data, C1.data)
    with pytest.raises(Exception, match="CG sessions only"):
        s.solve(0, np.zeros(m["vertices"].shape[0]), np.zeros(m["vertices"].shape[0]))


def test_dg_refusals(nl):
    from nlfem_gb300._lib import NlfemError
    m = square_mesh(6, 0.1)
    with pytest.raises(NlfemError, match="fp64 path only"):
        nl.stiffnessMatrix(dict(m), KC, _conf_dg(precision="mixed"))
    with pytest.raises(NlfemError, match="one at a time"):
        nl.stiffnessMatrix_batch([(dict(m), KC, _conf_dg()), (dict(m), KC, _conf_dg())])


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_linear_prototype_kernel(nl, orc, prec):
    """linearPrototypeMicroelastic (model.cpp:116-124), singular (Cassemble.cpp:89-94), with the
    fractional close-pair rule: the oracle's values, and bit for bit the fractional kernel at
    s = -1/2, whose formula it is."""
    m = square_mesh(10, 0.1, jitter=0.15, seed=9)
    kp = {"function": "linearPrototypeMicroelastic", "horizon": 0.1, "outputdim": 1, "fractional_s": -0.5}
    kf = {"function": "fractional", "horizon": 0.1, "outputdim": 1, "fractional_s": -0.5}
    A = nl.stiffnessMatrix(dict(m), kp, conf2d(rule="16", close="fractional", deg=3, precision=prec))
    B = orc.assemble(m, kp, conf2d(rule="16", close="fractional", deg=3))["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    tol = FP64_TOL if prec == "fp64" else MIX_TOL
    assert fro < tol and mx < tol, (fro, mx)
    F = nl.stiffnessMatrix(dict(m), kf, conf2d(rule="16", close="fractional", deg=3, precision=prec))
    assert same_pattern(A, F) and np.array_equal(A.data, F.data)


def test_weak_singular_close_rule(nl, orc):
    """The weakSingular close rule (integration.cpp:82-185) with the weakly singular kernel
    linearPrototypeMicroelastic: the oracle's matrix and close-pair blocks, and the matrix of the
    fractional close rule, which for this kernel is the same sum."""
    from nlfem_gb300._lib import NlfemError
    m = square_mesh(10, 0.1, jitter=0.15, seed=9)
    kp = {"function": "linearPrototypeMicroelastic", "horizon": 0.1, "outputdim": 1, "fractional_s": -0.5}
    cw = conf2d(rule="16", close="weakSingular", deg=3)
    A = nl.stiffnessMatrix(dict(m), kp, cw)
    B = orc.assemble(m, kp, cw)["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    F = nl.stiffnessMatrix(dict(m), kp, conf2d(rule="16", close="fractional", deg=3))
    assert abs(A - F).max() <= 1e-12 * abs(F).max()
    T = m["elements"]
    pairs = [(e, f) for e in (3, 40, 77) for f in range(T.shape[0]) if set(T[e]) & set(T[f])]
    g, _ = nl.pair_blocks(m, kp, cw, np.array(pairs), close=True)
    o, _ = orc.pair_blocks(m, kp, cw, np.array(pairs), method="weakSingular")
    np.testing.assert_allclose(g, o, rtol=1e-12, atol=1e-12 * np.abs(o).max())
    # the mixed path: FP32 Duffy rule (weakSingular form) for the close pairs, within the mixed bound
    Am = nl.stiffnessMatrix(dict(m), kp, conf2d(rule="16", close="weakSingular", deg=3, precision="mixed"))
    assert same_pattern(Am, B)
    fro, mx = rel_errors(Am, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)
    with pytest.raises(NlfemError, match="fractional close rule only"):
        nl.stiffnessMatrix(dict(m), kp, conf2d(rule="16", close="weakSingular", deg=3, precision="fp64-onesided"))


@pytest.mark.parametrize("name", ["config1", "tangent", "parabola20", "frac12", "cube5", "labeled10", "average10",
                                  "exact8", "dg10", "weak10", "field8"])
def test_gpu_matches_committed_fixtures(nl, name):
    """The FP64 path against the committed oracle fixtures (tests/golden/oracle_cases.npz, made by
    tests/golden/make_oracle_golden.py): bit-exact pattern, values within rounding."""
    import importlib.util
    import os
    gdir = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
    spec = importlib.util.spec_from_file_location("make_oracle_golden", os.path.join(gdir, "make_oracle_golden.py"))
    mg = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mg)
    fx = np.load(os.path.join(gdir, "oracle_cases.npz"))
    _, kernel, conf, load = mg.cases()[name]
    # the stored mesh: the fixture's own inputs, whatever numpy this host runs
    mesh = {k: fx[f"{name}.{k}"] for k in ("elements", "elementLabels", "vertices", "vertexLabels")}
    indptr = fx[f"{name}.indptr"]
    K = indptr.size - 1
    B = sp.csr_matrix((fx[f"{name}.data"], fx[f"{name}.indices"], indptr), shape=(K, K))
    A = nl.stiffnessMatrix(dict(mesh), kernel, conf)
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    tol = 1e-11 if name == "frac12" else FP64_TOL
    assert fro < tol and mx < tol, (fro, mx)
    if load is not None:
        f = nl.loadVector(dict(mesh, outdim=int(kernel.get("outputdim", 1))), load, conf)
        g = fx[f"{name}.f"]
        np.testing.assert_allclose(f, g, rtol=1e-13, atol=1e-15 * np.abs(g).max())


def test_load_vector(nl, orc):
    m = square_mesh(24, 0.1, jitter=0.2, seed=8)
    f = nl.loadVector(m, {"function": "linear"}, conf2d())
    g = orc.assemble(m, None, conf2d(), compute="forcing", load={"function": "linear"})["f"]
    np.testing.assert_allclose(f, g, rtol=1e-13, atol=1e-15 * np.abs(g).max())


def test_fractional_close_pairs(nl, orc):
    m = square_mesh(12, 0.2)
    k = {"function": "fractional", "horizon": 0.2, "outputdim": 1, "fractional_s": 0.4}
    c = conf2d(rule="16", close="fractional", deg=3)
    A = nl.stiffnessMatrix(m, k, c)
    B = orc.assemble(m, k, c)["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < 1e-11 and mx < 1e-11, (fro, mx)


def test_fractional_close_blocks(nl, orc):
    m = square_mesh(6, 0.2, jitter=0.2, seed=1)
    k = {"function": "fractional", "horizon": 0.2, "outputdim": 1, "fractional_s": 0.4}
    c = conf2d(rule="16", close="fractional", deg=4)
    e = m["elements"]
    pairs = [(i, i) for i in range(0, 60, 7)]
    for a in range(0, 60, 5):
        for b in range(e.shape[0]):
            if a != b and len(set(e[a]) & set(e[b])) in (1, 2):
                pairs.append((a, b))
    pairs = np.array(pairs)
    g, _ = nl.pair_blocks(m, k, c, pairs, close=True)
    o, _ = orc.pair_blocks(m, k, c, pairs, method="fractional")
    np.testing.assert_allclose(g, o, rtol=1e-11, atol=1e-12 * np.abs(o).max())


def test_3d_barycenter(nl, orc):
    m = cube_mesh(5, 0.1, jitter=0.15, seed=2)
    k = {"function": "constant3D", "horizon": 0.3, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf3d())
    B = orc.assemble(m, k, conf3d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    f = nl.loadVector(m, {"function": "linear3D"}, conf3d())
    g = orc.assemble(m, None, conf3d(), compute="forcing", load={"function": "linear3D"})["f"]
    np.testing.assert_allclose(f, g, rtol=1e-13, atol=1e-15 * np.abs(g).max())


def test_batch_equals_single(nl):
    probs = []
    for i, (n, d, kn) in enumerate([(10, 0.1, "constant"), (14, 0.13, "parabola"), (8, 0.2, "constant")]):
        probs.append((square_mesh(n, d, jitter=0.2, seed=i), {"function": kn, "horizon": d, "outputdim": 1}, conf2d()))
    As = nl.stiffnessMatrix_batch(probs)
    for (m, k, c), A in zip(probs, As):
        B = nl.stiffnessMatrix(m, k, c)
        assert same_pattern(A, B)
        assert abs(A - B).max() == 0


def test_deterministic_runs(nl):
    m = square_mesh(24, 0.1, jitter=0.2, seed=6)
    k = {"function": "parabola", "horizon": 0.1, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf2d())
    B = nl.stiffnessMatrix(m, k, conf2d())
    assert same_pattern(A, B)
    assert np.array_equal(A.data, B.data)


def test_par_assemble_file_protocol(nl, tmp_path):
    from nlfem_gb300 import _lib
    lib = _lib.load()
    m = square_mesh(10, 0.1)
    c = conf2d()
    A = nl.stiffnessMatrix(m, KC, c)
    el = np.ascontiguousarray(m["elements"].ravel(), np.int64)
    elab = np.ascontiguousarray(m["elementLabels"], np.int64)
    ve = np.ascontiguousarray(m["vertices"].ravel(), np.float64)
    vlab = np.ascontiguousarray(m["vertexLabels"], np.int64)
    P = np.ascontiguousarray(c["quadrature"]["outer"]["points"].ravel()); w = c["quadrature"]["outer"]["weights"]
    dp, lp = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_long)
    D = lambda a: a.ctypes.data_as(dp)
    L = lambda a: a.ctypes.data_as(lp)
    nE, nV = m["elements"].shape[0], m["vertices"].shape[0]
    path = str(tmp_path / "spAd").encode()
    r = lib.nlfem_par_assemble(b"system", path, b"", int((vlab > 0).sum()), nV, L(el), L(elab), D(ve), L(vlab),
                               nE, int((elab > 0).sum()), nV, int((vlab > 0).sum()), D(P), len(w), D(w),
                               D(P), len(w), D(w), ctypes.c_double(0.1 ** 2), 0, 0, b"constant", b"",
                               b"retriangulate", b"retriangulate", 1, 2, 1, None, None, ctypes.c_long(0),
                               None, 0, None, ctypes.c_double(0.0), ctypes.c_double(-1.0), 0, 0)
    assert r == 0, lib.nlfem_last_error()
    B = nl.read_arma_spMat(tmp_path / "spAd")
    assert same_pattern(A, B) and abs(A - B).max() == 0


# ---------------------------------------------------------------- mixed precision
MIX_TOL = 1e-6   # relative Frobenius / max-entry error of the mixed path against the FP64 oracle


def test_certified_geometry_small_triangles(nl, orc):
    """Mesh regime: triangles of size ~delta/20 straddling the sphere, incl. near-tangent edges
    and vertices close to it. Certified FP32 cases must match the exact polygon exactly."""
    rng = np.random.Generator(np.random.PCG64(23))
    delta = 0.1
    n = 60000
    ang = rng.uniform(0, 2 * np.pi, n)
    rad = delta + rng.normal(0, 0.004, n)
    rad[::5] = delta + rng.normal(0, 1e-6, n)[::5]          # vertex near the sphere
    c = np.stack([rad * np.cos(ang), rad * np.sin(ang)], 1)
    h = delta / 20 * rng.uniform(0.5, 1.5, n)
    th = rng.uniform(0, 2 * np.pi, (n, 3))
    T = np.zeros((n, 6))
    T[:, 0:2] = c
    T[:, 2:4] = c + h[:, None] * np.stack([np.cos(th[:, 1]), np.sin(th[:, 1])], 1)
    T[:, 4:6] = c + h[:, None] * np.stack([np.cos(th[:, 2]), np.sin(th[:, 2])], 1)
    T[1::7, 2:4] = T[1::7, 0:2] + (T[1::7, 0:2] / np.linalg.norm(T[1::7, 0:2], axis=1)[:, None])[:, ::-1] * [1, -1] * h[1::7, None]
    x0 = np.array([0.3, -0.2])
    X = np.tile(x0, (n, 1))
    T = T + np.tile(x0, 3)
    for caps in (1, 0):
        cnt, amb, pts = nl.retriangulate_certified_batch(X, T, delta ** 2, caps)
        namb = 0
        for j in range(n):
            if amb[j]:
                namb += 1
                continue
            m, tri = orc.retriangulate_sq(X[j], T[j], delta ** 2, caps)
            exact_pts = 0 if m == 0 else m + 2
            got = cnt[j] if cnt[j] >= 3 else 0
            assert got == exact_pts, (caps, j, cnt[j], m)
            if m:
                R = np.concatenate([tri[0, :1], tri[:, 1], tri[-1:, 2]], axis=0) - X[j]
                # positions: FP32 accuracy, looser along near-tangent edges (values only)
                np.testing.assert_allclose(pts[j, :exact_pts], R, atol=1e-3 * delta)
        # about a third of the cases are built on a decision boundary
        assert namb < 0.45 * n


def test_certified_geometry_mesh_regime(nl, orc):
    """Outer points of mesh elements against the elements near their ball boundary (the cases the
    assembly meets): certified FP32 results equal the exact polygon counts; few fall back."""
    from nlfem_gb300 import meshes, quadrules
    v, e, l = meshes.regular_square(64, 0.1, jitter=0.2, seed=3)
    P, w = quadrules.dunavant7()
    rng = np.random.Generator(np.random.PCG64(4))
    E = v[e]
    bary = E.mean(axis=1)
    X, T = [], []
    for a in rng.choice(len(e), 60, replace=False):
        xs = E[a][0] + (E[a][1] - E[a][0]) * P[:, :1] + (E[a][2] - E[a][0]) * P[:, 1:2]
        d = np.linalg.norm(bary - bary[a], axis=1)
        cand = np.where(np.abs(d - 0.1) < 0.04)[0]
        for x in xs:
            X.append(np.repeat(x[None], len(cand), 0)); T.append(E[cand].reshape(-1, 6))
    X = np.concatenate(X); T = np.concatenate(T)
    cnt, amb, pts = nl.retriangulate_certified_batch(X, T, 0.01, 1)
    ex, _ = nl.retriangulate_batch(X, T, 0.01, 1)
    ok = amb == 0
    got = np.where(cnt >= 3, cnt - 2, 0)
    np.testing.assert_array_equal(got[ok], ex[ok])
    assert (~ok).sum() < 0.01 * (ex > 0).sum()


def test_certified_geometry_never_disagrees(nl, orc):
    """Where the FP32 geometry does not flag a decision as ambiguous, it reproduces the exact
    polygon point count and its points to FP32 accuracy. Half of the cases are built to sit on a
    decision boundary (tangent edges, vertices on the sphere); random cases rarely do."""
    rng = np.random.Generator(np.random.PCG64(17))
    cases = _cases_retri(rng, 4000)
    amb_random = 0
    for j, (x, T, sq, caps) in enumerate(cases):
        c, a, pts = nl.retriangulate_certified_batch(x[None], T[None], sq, caps)
        n, tri = orc.retriangulate_sq(x, T, sq, caps)
        if a[0]:
            amb_random += (j % 4 == 0)
            continue
        exact_pts = 0 if n == 0 else n + 2
        got = c[0] if c[0] >= 3 else 0
        assert got == exact_pts, (j, c[0], n)
        if n:
            R = np.concatenate([tri[0, :1], tri[:, 1], tri[-1:, 2]], axis=0) - x
            np.testing.assert_allclose(pts[0, :exact_pts], R, atol=1e-3 * np.sqrt(sq) + 1e-6)
    assert amb_random < 0.05 * len(cases) / 4


@pytest.mark.parametrize("n,delta,kern,jit", [(32, 0.1, "constant", 0.0), (24, 0.12, "parabola", 0.2),
                                              (20, 0.15, "constant", 0.2)])
def test_mixed_matches_oracle(nl, orc, n, delta, kern, jit):
    m = square_mesh(n, delta, jitter=jit, seed=n)
    k = {"function": kern, "horizon": delta, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf2d(precision="mixed"))
    B = orc.assemble(m, k, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


def test_mixed_batch_mixed_kernels(nl, orc):
    """A batch mixing constant (closed-form inner sums) and parabola problems equals the single
    assemblies, and each problem matches the oracle."""
    probs = []
    for i, (n, d, kn) in enumerate([(10, 0.1, "constant"), (14, 0.13, "parabola"), (8, 0.2, "constant")]):
        probs.append((square_mesh(n, d, jitter=0.2, seed=i), {"function": kn, "horizon": d, "outputdim": 1},
                      conf2d(precision="mixed")))
    As = nl.stiffnessMatrix_batch(probs)
    for (m, k, c), A in zip(probs, As):
        B = nl.stiffnessMatrix(m, k, c)
        assert same_pattern(A, B)
        assert abs(A - B).max() <= 1e-12 * abs(B).max()
        R = orc.assemble(m, k, conf2d())["A"]
        assert same_pattern(A, R)
        fro, mx = rel_errors(A, R)
        assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


def test_mixed_batch_three_kernel_classes(nl, orc):
    """Constant, parabola and fractional (Duffy close pairs) problems in one batch: one pass
    launch per kernel class, each matrix equal to its single assembly."""
    c = conf2d(rule="16", close="fractional", deg=3, precision="mixed")
    probs = [(square_mesh(10, 0.2, jitter=0.1, seed=21), {"function": "constant", "horizon": 0.2, "outputdim": 1}, c),
             (square_mesh(9, 0.2, jitter=0.1, seed=22), {"function": "fractional", "horizon": 0.2, "outputdim": 1,
                                                          "fractional_s": 0.4}, c),
             (square_mesh(8, 0.2, jitter=0.1, seed=23), {"function": "parabola", "horizon": 0.2, "outputdim": 1}, c)]
    As = nl.stiffnessMatrix_batch(probs)
    for (m, k, cc), A in zip(probs, As):
        B = nl.stiffnessMatrix(m, k, cc)
        assert same_pattern(A, B)
        assert abs(A - B).max() <= 1e-12 * abs(B).max()
        R = orc.assemble(m, k, conf2d(rule="16", close="fractional", deg=3))["A"]
        assert same_pattern(A, R)
        fro, mx = rel_errors(A, R)
        assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


def test_one_shot_capacity_hints_overflow(nl, orc):
    """One-shot calls reuse the previous call's pattern sizes as scratch capacities when the mesh
    has the same counts. A second mesh with the same counts and a larger ball overflows them; the
    recount must give the exact pattern and values."""
    m = square_mesh(16, 0.1, jitter=0.2, seed=31)
    k1 = {"function": "constant", "horizon": 0.1, "outputdim": 1}
    nl.stiffnessMatrix(m, k1, conf2d(precision="mixed"))
    m2 = square_mesh(16, 0.1, jitter=0.1, seed=32)   # same counts
    k2 = {"function": "constant", "horizon": 0.25, "outputdim": 1}
    A = nl.stiffnessMatrix(m2, k2, conf2d(precision="mixed"))
    B = orc.assemble(m2, k2, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)
    A1 = nl.stiffnessMatrix(m, k1, conf2d(precision="mixed"))   # and back to the smaller one
    B1 = orc.assemble(m, k1, conf2d())["A"]
    assert same_pattern(A1, B1)


@pytest.mark.parametrize("case", ["2d", "2d_J", "3d", "dg"])
def test_evaluate_mass_matches_oracle(nl, orc, case):
    """par_evaluateMass on the GPU (deterministic fixed-point sums) against the oracle's
    sequential restatement."""
    from types import SimpleNamespace
    from nlfem_gb300 import quadrules
    rng = np.random.Generator(np.random.PCG64(7))
    if case == "3d":
        m = cube_mesh(5, 0.1, jitter=0.1, seed=2)
        P, w = quadrules.keast11()
    else:
        m = square_mesh(12, 0.1, jitter=0.2, seed=5)
        P, w = quadrules.dunavant7()
    nE, dV = m["elements"].shape
    dg = case == "dg"
    K = dV * nE if dg else m["vertices"].shape[0]
    ud = rng.standard_normal(K)
    J = nE // 2 if case == "2d_J" else nE
    mesh = SimpleNamespace(elements=m["elements"], elementLabels=m["elementLabels"], vertices=m["vertices"],
                           vertexLabels=m["vertexLabels"], dim=m["vertices"].shape[1], nE_Omega=J,
                           is_DiscontinuousGalerkin=dg, K=K)
    vd = nl.evaluateMass(mesh, ud, P, w)
    ref = orc.evaluate_mass(m, ud, P, w, J=J, is_dg=dg)
    assert np.abs(vd - ref).max() <= 1e-13 * np.abs(ref).max()
    assert np.array_equal(vd, nl.evaluateMass(mesh, ud, P, w))   # deterministic


def test_mixed_pair_list_exact(nl, orc):
    m = square_mesh(24, 0.13, jitter=0.2, seed=3)
    k = {"function": "constant", "horizon": 0.13, "outputdim": 1}
    ref = orc.assemble(m, k, conf2d(), want_pairs=True)
    got = nl.pair_list(m, k, conf2d(precision="mixed"))
    rp = ref["pairs"][np.lexsort((ref["pairs"][:, 1], ref["pairs"][:, 0]))]
    np.testing.assert_array_equal(got, rp)


def test_mixed_fractional(nl, orc):
    m = square_mesh(12, 0.2, jitter=0.1, seed=5)
    k = {"function": "fractional", "horizon": 0.2, "outputdim": 1, "fractional_s": 0.4}
    A = nl.stiffnessMatrix(m, k, conf2d(rule="16", close="fractional", deg=3, precision="mixed"))
    B = orc.assemble(m, k, conf2d(rule="16", close="fractional", deg=3))["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


def test_mixed_3d(nl, orc):
    m = cube_mesh(5, 0.1, jitter=0.15, seed=2)
    k = {"function": "constant3D", "horizon": 0.3, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf3d(precision="mixed"))
    B = orc.assemble(m, k, conf3d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


def test_mixed_deterministic(nl):
    m = square_mesh(28, 0.1, jitter=0.2, seed=6)
    k = {"function": "parabola", "horizon": 0.1, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf2d(precision="mixed"))
    B = nl.stiffnessMatrix(m, k, conf2d(precision="mixed"))
    assert same_pattern(A, B) and np.array_equal(A.data, B.data)


def test_mixed_pattern_equals_fp64_at_scale(nl):
    """On a mesh too large for the oracle the mixed pattern still equals the FP64 GPU pattern
    (itself bit-exact against the oracle on the smaller meshes above)."""
    m = square_mesh(96, 0.1, jitter=0.2, seed=1)
    A = nl.stiffnessMatrix(m, KC, conf2d(precision="mixed"))
    B = nl.stiffnessMatrix(m, KC, conf2d())
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


@pytest.mark.parametrize("kern", ["parabola", "constant"])
def test_mixed_barycenter_2d(nl, orc, kern):
    m = square_mesh(16, 0.15, jitter=0.2, seed=4)
    k = {"function": kern, "horizon": 0.15, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf2d(method="baryCenter", precision="mixed"))
    B = orc.assemble(m, k, conf2d(method="baryCenter"))["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


def test_mixed_3d_deterministic_and_fp64_pattern(nl):
    m = cube_mesh(7, 0.1, jitter=0.1, seed=3)
    k = {"function": "constant3D", "horizon": 0.25, "outputdim": 1}
    A1 = nl.stiffnessMatrix(m, k, conf3d(precision="mixed"))
    A2 = nl.stiffnessMatrix(m, k, conf3d(precision="mixed"))
    assert same_pattern(A1, A2) and np.array_equal(A1.data, A2.data)
    B = nl.stiffnessMatrix(m, k, conf3d())
    assert same_pattern(A1, B)
    fro, mx = rel_errors(A1, B)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


@pytest.mark.parametrize("case", ["retri2d", "bary3d"])
def test_search_stamp_epochs(nl, case):
    """The pair search's 16-bit per-warp stamp epochs: later assemblies of a session reuse the
    stamps uncleared, and a warp whose epoch wraps clears its own stamps; every assembly, normal
    or replayed from the graph, gives the first one's matrix bit for bit. The epochs are moved
    once, forward (above every epoch used so far), to 16 below the wrap; the assemblies after it
    take the warps that get elements through the wrap."""
    from nlfem_gb300 import _lib
    if case == "retri2d":
        probs = [(square_mesh(40, 0.1, jitter=0.2, seed=11), KC, conf2d(precision="mixed"))]
    else:
        probs = [(cube_mesh(8, 0.1, jitter=0.1, seed=12), {"function": "constant3D", "horizon": 0.2, "outputdim": 1},
                  conf3d(precision="mixed"))]
    s = nl.Session(probs)
    try:
        assert s.lib.nlfem_session_set_search_epoch(s.h, 5) != 0   # no search has run yet
        s.assemble()
        ref = s.download(0)
        _lib.check(s.lib.nlfem_session_set_search_epoch(s.h, 0xfff0))
        for i in range(40):
            graph = i % 2 == 1
            s.assemble(graph=graph)
            A = s.download(0)
            assert same_pattern(A, ref) and np.array_equal(A.data, ref.data), (i, graph)
    finally:
        s.close()


@pytest.mark.parametrize("case", ["retri_batch", "bary3d", "fractional"])
def test_session_graph_replay_bitwise(nl, case):
    if case == "retri_batch":
        probs = [(square_mesh(20, 0.12, jitter=0.2, seed=9), {"function": "parabola", "horizon": 0.12, "outputdim": 1},
                  conf2d(precision="mixed")),
                 (square_mesh(14, 0.2, jitter=0.1, seed=2), {"function": "constant", "horizon": 0.2, "outputdim": 1},
                  conf2d(precision="mixed"))]
    elif case == "bary3d":
        probs = [(cube_mesh(5, 0.1, jitter=0.1, seed=5), {"function": "constant3D", "horizon": 0.3, "outputdim": 1},
                  conf3d(precision="mixed"))]
    else:
        probs = [(square_mesh(10, 0.2, jitter=0.1, seed=3),
                  {"function": "fractional", "horizon": 0.2, "outputdim": 1, "fractional_s": 0.4},
                  conf2d(rule="16", close="fractional", deg=3, precision="mixed"))]
    s = nl.Session(probs)
    try:
        st0 = s.assemble()
        ref = [s.download(i) for i in range(len(probs))]
        s.assemble()   # a repeated assembly builds the pattern in one pass (scratch sized by the first)
        for i, B in enumerate(ref):
            A = s.download(i)
            assert same_pattern(A, B) and np.array_equal(A.data, B.data)
        for _ in range(3):
            st = s.assemble(graph=True)
            assert st["n_pairs"] == st0["n_pairs"] and st["nnz_structural"] == st0["nnz_structural"]
            for i, B in enumerate(ref):
                A = s.download(i)
                assert same_pattern(A, B) and np.array_equal(A.data, B.data)
    finally:
        s.close()
    # a session whose first call already asks for the graph (capture right after the first run)
    s2 = nl.Session(probs)
    try:
        for _ in range(3):
            s2.assemble(graph=True)
            for i, B in enumerate(ref):
                A = s2.download(i)
                assert same_pattern(A, B) and np.array_equal(A.data, B.data)
    finally:
        s2.close()


@pytest.mark.parametrize("n,delta,kern,jit,close", [(32, 0.1, "constant", 0.0, None), (24, 0.12, "parabola", 0.2, None),
                                                    (20, 0.15, "constant", 0.2, None),
                                                    (12, 0.2, "fractional", 0.1, "fractional")])
def test_fp64_onesided_matches_oracle(nl, orc, n, delta, kern, jit, close):
    """The mixed path's algorithm in FP64 arithmetic (precision "fp64-onesided"): one-sided pass,
    closed forms, fixed-point sums with a unit of 2^-52 of the entry scale. It meets the FP64 bar
    against the oracle (1e-12), and its pattern is the reference's."""
    m = square_mesh(n, delta, jitter=jit, seed=n)
    k = {"function": kern, "horizon": delta, "outputdim": 1}
    if kern == "fractional":
        k["fractional_s"] = 0.4
        c = conf2d(rule="16", close=close, deg=3)
    else:
        c = conf2d()
    A = nl.stiffnessMatrix(m, k, dict(c, precision="fp64-onesided"))
    B = orc.assemble(m, k, c)["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < 1e-12 and mx < 1e-12, (fro, mx)
    # deterministic, like every fixed-point path
    A2 = nl.stiffnessMatrix(m, k, dict(c, precision="fp64-onesided"))
    assert np.array_equal(A.data, A2.data)


def test_fp64_onesided_refusals(nl):
    from nlfem_gb300._lib import NlfemError
    m = cube_mesh(3, 0.2)
    from nlfem_gb300 import quadrules
    P, w = quadrules.keast11()
    c = {"ansatz": "CG", "approxBalls": {"method": "baryCenter"},
         "quadrature": {"outer": {"points": P, "weights": w}, "inner": {"points": P, "weights": w}},
         "precision": "fp64-onesided"}
    with pytest.raises(NlfemError, match="2D retriangulate"):
        nl.stiffnessMatrix(m, {"function": "constant3D", "horizon": 0.2, "outputdim": 1}, c)



FIELD_CASES = {
    # constantField (model.cpp:182-191), retriangulate with caps, jittered
    "constfield": (lambda: square_mesh(12, 0.15, jitter=0.2, seed=21), {"function": "constantField", "horizon": 0.15, "outputdim": 2},
                   lambda: conf2d()),
    # the microelastic field kernel, singular: close pairs by the fractional Duffy rule
    "microfield_frac": (lambda: square_mesh(8, 0.2, jitter=0.1, seed=22),
                        {"function": "linearPrototypeMicroelasticField", "horizon": 0.2, "outputdim": 2, "fractional_s": -0.5},
                        lambda: conf2d(rule="16", close="fractional", deg=3)),
    # the same with the weakSingular close rule
    "microfield_weak": (lambda: square_mesh(8, 0.2, jitter=0.1, seed=23),
                        {"function": "linearPrototypeMicroelasticField", "horizon": 0.2, "outputdim": 2, "fractional_s": -0.5},
                        lambda: conf2d(rule="16", close="weakSingular", deg=3)),
    # 2D barycenter rule with the constant field kernel
    "constfield_bary": (lambda: square_mesh(10, 0.2, jitter=0.15, seed=24), {"function": "constantField", "horizon": 0.2, "outputdim": 2},
                        lambda: conf2d(method="baryCenter")),
    # 3D microelastic field kernel, barycenter (not singular in the reference's lookup); the inner
    # rule avoids the outer points, where the kernel is singular
    "microfield3d": (lambda: cube_mesh(3, 0.1, jitter=0.1, seed=25),
                     {"function": "linearPrototypeMicroelasticField3D", "horizon": 0.35, "outputdim": 3}, lambda: _conf3d_inner4()),
}


def _conf3d_inner4():
    pa, pb = 0.5854101966249685, 0.1381966011250105
    c = conf3d()
    c["quadrature"]["inner"] = {"points": np.array([[pb, pb, pb], [pa, pb, pb], [pb, pa, pb], [pb, pb, pa]]),
                                "weights": np.full(4, 1.0 / 24)}
    return c


@pytest.mark.parametrize("case", list(FIELD_CASES))
def test_vector_kernels_match_oracle(nl, orc, case):
    """Vector-valued kernels (outdim 2 and 3) on the GPU: the reference's general block indexing
    (integration.cpp:345-540, 910-1018, 82-288; Cassemble.cpp:721-770) in FP64 with
    deterministic fixed-point sums. Pattern bit-exact, values within 1e-12 of the oracle (which
    the reference build pins bit for bit)."""
    mk, kernel, mkconf = FIELD_CASES[case]
    m = dict(mk(), outdim=kernel["outputdim"])
    conf = mkconf()
    A = nl.stiffnessMatrix(m, kernel, conf)
    B = orc.assemble(m, kernel, conf)["A"]
    assert A.shape == B.shape == (m["vertices"].shape[0] * kernel["outputdim"],) * 2
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    A2 = nl.stiffnessMatrix(m, kernel, conf)
    assert np.array_equal(A.data, A2.data)   # deterministic


@pytest.mark.parametrize("load,outdim,dim", [("linearField", 2, 2), ("constantRightField", 2, 2), ("constantDownField", 2, 2),
                                              ("constantBothField", 2, 2), ("linearField3D", 3, 3), ("gaussian", 1, 2),
                                              ("jump", 1, 2), ("tensorsin", 1, 2)])
def test_further_forcings_match_oracle(nl, orc, load, outdim, dim):
    """The vector forcings and the scalar gaussian / jump / tensorsin (model.cpp:201-258) against
    the oracle: within 1e-13 (CUDA's exp and sin may differ from the host's in the last bit)."""
    m = square_mesh(14, 0.1, jitter=0.2, seed=26) if dim == 2 else cube_mesh(3, 0.2, jitter=0.1, seed=27)
    m = dict(m, outdim=outdim)
    conf = conf2d() if dim == 2 else conf3d()
    f = nl.loadVector(m, {"function": load}, conf)
    g = orc.assemble(m, None, conf, compute="forcing", load={"function": load})["f"]
    assert f.shape == g.shape == (m["vertices"].shape[0] * outdim,)
    np.testing.assert_allclose(f, g, rtol=1e-13, atol=1e-14 * np.abs(g).max())


def test_load_vector_domain_decomposition(nl, orc):
    """par_forcing weights each element's contribution by 1 / zeta(aT, aT) (Cassemble.cpp:901-908)."""
    m = square_mesh(12, 0.1, jitter=0.2, seed=28)
    nE = m["elements"].shape[0]
    bx = m["vertices"][m["elements"]].mean(axis=1)[:, 0]
    rows, cols = [], []
    for e in range(nE):   # two overlapping subdomains around x = 0.5
        for z, inside in enumerate((bx[e] < 0.6, bx[e] > 0.4)):
            if inside:
                rows.append(e); cols.append(z)
    Z = sp.csr_matrix((np.ones(len(rows)), (rows, cols)), shape=(nE, 2))
    m = dict(m, nZeta=2, ZetaIndicator=Z)
    f = nl.loadVector(m, {"function": "linear"}, conf2d())
    g = orc.assemble(m, None, conf2d(), compute="forcing", load={"function": "linear"})["f"]
    np.testing.assert_allclose(f, g, rtol=1e-13, atol=1e-15 * np.abs(g).max())
    f0 = nl.loadVector(dict(m, nZeta=0), {"function": "linear"}, conf2d())
    assert not np.allclose(f, f0)


def test_vector_kernel_refusals(nl):
    from nlfem_gb300._lib import NlfemError
    m = dict(square_mesh(4, 0.2), outdim=2)
    k = {"function": "constantField", "horizon": 0.2, "outputdim": 2}
    with pytest.raises(NlfemError, match="fp64 path only"):
        nl.stiffnessMatrix(m, k, conf2d(precision="mixed"))
    with pytest.raises(NlfemError, match="output components"):
        nl.stiffnessMatrix(dict(m, outdim=1), dict(k, outputdim=1), conf2d())



@pytest.mark.parametrize("n,delta,kern,jit", [(10, 0.1, "constant", 0.15), (14, 0.12, "parabola", 0.2), (9, 0.25, "constant", 0.0)])
def test_exact_ball_matches_oracle(nl, orc, n, delta, kern, jit):
    """exactBall (integration.cpp:706-907, 1300-1351, 1632-1761) on the FP64 path: the polygon
    without cap points plus up to three circular segments at their centroids. The pair search takes
    the polygon's interaction test. Within 1e-12 of the oracle (CUDA's acos / sin / pow may differ
    from the host's in the last bit)."""
    m = square_mesh(n, delta, jitter=jit, seed=n + 40)
    k = {"function": kern, "horizon": delta, "outputdim": 1}
    c = conf2d(method="exactBall")
    A = nl.stiffnessMatrix(m, k, c)
    B = orc.assemble(m, k, c)["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    pairs = orc.assemble(m, k, c, want_pairs=True)["pairs"]
    sel = pairs[np.random.Generator(np.random.PCG64(n)).choice(len(pairs), min(300, len(pairs)), replace=False)]
    g, gr = nl.pair_blocks(m, k, c, sel)
    o, orr = orc.pair_blocks(m, k, c, sel)
    np.testing.assert_array_equal(gr != 0, orr != 0)
    np.testing.assert_allclose(g, o, rtol=1e-12, atol=1e-12 * np.abs(o).max())


def test_autotune_keeps_the_matrix(nl):
    """The launch-shape autotuner (nlfem_session_autotune) times 1, 2, ... blocks per SM of the
    pair search and the persistent pass and keeps the fastest; the shapes change no bit of the
    matrix (fixed-point sums, per-element search order)."""
    m = square_mesh(48, 0.1, jitter=0.2, seed=61)
    k = {"function": "constant", "horizon": 0.1, "outputdim": 1}
    s = nl.Session([(m, k, conf2d(precision="mixed"))])
    try:
        s.assemble()
        A0 = s.download(0)
        t = s.autotune(reps=1)
        A1 = s.download(0)
        assert t["bfs"] >= 1 and len(t["bfs_ms"]) >= 1
        assert t["pass"] >= 1 and len(t["pass_ms"]) >= 1
        assert all(x > 0 for x in t["bfs_ms"] + t["pass_ms"])
        assert np.array_equal(A0.indptr, A1.indptr) and np.array_equal(A0.indices, A1.indices)
        assert np.array_equal(A0.data, A1.data)
        s.assemble(graph=True)   # a graph captured after tuning replays the tuned shapes
        s.assemble(graph=True)
        assert np.array_equal(s.download(0).data, A0.data)
    finally:
        s.close()


def test_mixed_slot_maps_window_rank_and_hash(nl, orc):
    """The one-sided pass finds matrix slots with window-rank bitmaps when the rows span narrow
    ranges of vertex numbers (a row-by-row numbering) and with per-row hash tables otherwise (here:
    a random vertex numbering). Both give the same matrix, bit for bit after renumbering, and
    both match the oracle within the mixed tolerance."""
    from nlfem_gb300 import _lib, meshes
    v, e, l = meshes.regular_square(64, 0.03, jitter=0.2, seed=21)
    m = meshes.mesh_dict(v, e, l)
    k = {"function": "constant", "horizon": 0.03, "outputdim": 1}
    c = conf2d(precision="mixed")
    A = nl.stiffnessMatrix(dict(m), k, c)
    assert _lib.stats()["slot_map"] == 1
    nV = v.shape[0]
    perm = np.random.default_rng(3).permutation(nV)   # vertex i becomes vertex perm[i]
    v2 = np.empty_like(v)
    v2[perm] = v
    m2 = meshes.mesh_dict(v2, perm[e], l)
    B = nl.stiffnessMatrix(m2, k, c)
    assert _lib.stats()["slot_map"] == 2
    Ac = A.tocoo()   # renumbered entry by entry: slots that cancelled to zero stay stored
    A2 = sp.csr_matrix((Ac.data, (perm[Ac.row], perm[Ac.col])), shape=(nV, nV))
    A2.sort_indices(); B.sort_indices()
    assert same_pattern(A2, B)
    np.testing.assert_array_equal(A2.data, B.data)
    C = orc.assemble(m, k, conf2d())["A"]
    assert same_pattern(A, C)
    fro, mx = rel_errors(A, C)
    assert fro < MIX_TOL and mx < MIX_TOL, (fro, mx)


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_far_component_capacity_retries(nl, orc, prec):
    """The search sizes its pair pool from the mesh's mean element size. A far-away extra triangle
    inflates the bounding box, so that estimate is far too small and the pool overflows: the
    search reruns with the size it counted. The pairs and the matrix are those of the oracle."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_square(32, 0.3, jitter=0.1, seed=31)
    nV = v.shape[0]
    v2 = np.vstack([v, [[50.0, 50.0], [50.01, 50.0], [50.0, 50.01]]])
    e2 = np.vstack([e, [[nV, nV + 1, nV + 2]]])
    l2 = np.concatenate([l, [1]])
    m = meshes.mesh_dict(v2, e2, l2)
    k = {"function": "constant", "horizon": 0.3, "outputdim": 1}
    A = nl.stiffnessMatrix(dict(m), k, conf2d(precision=prec))
    ref = orc.assemble(m, k, conf2d(), want_pairs=True)
    got = nl.pair_list(m, k, conf2d(precision=prec))
    rp = ref["pairs"][np.lexsort((ref["pairs"][:, 1], ref["pairs"][:, 0]))]
    np.testing.assert_array_equal(got, rp)
    assert same_pattern(A, ref["A"])
    fro, mx = rel_errors(A, ref["A"])
    tol = MIX_TOL if prec == "mixed" else FP64_TOL
    assert fro < tol and mx < tol, (fro, mx)


def test_mixed_refuses_elements_far_larger_than_the_horizon(nl, orc):
    """The margins of the mixed path's FP32 geometry hold while every element is at most 16 times
    the horizon (certified.cuh); beyond that the mixed precision is refused and FP64 runs. With a
    horizon this small, a ball around an element's own quadrature point stays inside the element,
    which the retriangulation counts as no polygon, so some elements have no pair at all."""
    from nlfem_gb300._lib import NlfemError
    m = square_mesh(8, 0.005, jitter=0.1, seed=33)
    k = {"function": "constant", "horizon": 0.005, "outputdim": 1}
    with pytest.raises(NlfemError, match="no larger than 16 times the horizon"):
        nl.stiffnessMatrix(dict(m), k, conf2d(precision="mixed"))
    A = nl.stiffnessMatrix(dict(m), k, conf2d())
    B = orc.assemble(m, k, conf2d())["A"]
    assert same_pattern(A, B)
    if B.nnz:
        fro, mx = rel_errors(A, B)
        assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)


def _split_rule(n):
    """n-point rules of the reference triangle for the FP64 pass's mask tables: the centroid, the 7- and
    16-point rules, and the 7-point rule on each of the four midpoint triangles (28 points)."""
    from nlfem_gb300 import quadrules
    if n == 1:
        return quadrules.centroid1()
    if n in (7, 16):
        return quadrules.dunavant7() if n == 7 else quadrules.dunavant16()
    P, w = quadrules.dunavant7()
    corners = [((0, 0), (.5, 0), (0, .5)), ((.5, 0), (1, 0), (.5, .5)), ((0, .5), (.5, .5), (0, 1)), ((.5, .5), (0, .5), (.5, 0))]
    pts = [np.array(a) + P[:, :1] * (np.array(b) - np.array(a)) + P[:, 1:] * (np.array(c) - np.array(a)) for a, b, c in corners]
    return np.concatenate(pts), np.tile(w / 4, 4)


@pytest.mark.parametrize("nq,kern", [(1, "constant"), (16, "constant"), (28, "constant"), (1, "parabola"), (28, "parabola"), (7, "constant")])
def test_fp64_pass_rules_numberings_and_graph(nl, orc, nq, kern):
    """The one-sided FP64 pass at outer rules of one to four mask bytes, on a graded mesh (element
    measures over two decades) with a random vertex numbering (hash slot maps), against the oracle;
    normal runs, graph replays and a batch give the same bits."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_square(14, 0.1, jitter=0.15, seed=71)
    v = np.sign(v) * np.abs(v) ** 1.7
    perm = np.random.default_rng(5).permutation(len(v))
    v2 = np.empty_like(v)
    v2[perm] = v
    m = meshes.mesh_dict(v2, perm[e], l)
    P, w = _split_rule(nq)
    c = conf2d()
    c["quadrature"] = {"outer": {"points": P, "weights": w}, "inner": {"points": P, "weights": w}}
    k = {"function": kern, "horizon": 0.11, "outputdim": 1}
    A = nl.stiffnessMatrix(dict(m), k, c)
    B = orc.assemble(m, k, c)["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    s = nl.Session([(dict(m), k, c), (square_mesh(9, 0.1, jitter=0.2, seed=72), KC, c)])
    try:
        for graph in (False, True, True):
            s.assemble(graph=graph)
            C = s.download(0)
            assert same_pattern(A, C) and np.array_equal(A.tocsr().data, C.data)
    finally:
        s.close()


def test_fp64_general_pass_still_taken(nl, orc):
    """Calls outside the one-sided FP64 pass (a sliver element, an element far above the horizon beside
    ordinary ones) take the general FP64 passes, alone and in a batch with an ordinary problem."""
    m = square_mesh(10, 0.1, jitter=0.1, seed=73)
    v = m["vertices"].copy()
    v[0] = 0.5 * (v[1] + v[11]) + 1e-13   # a corner moved onto the diagonal of its cell: slivers
    from nlfem_gb300 import meshes
    sliver = meshes.mesh_dict(v, m["elements"], m["elementLabels"])
    A = nl.stiffnessMatrix(dict(sliver), KC, conf2d())
    B = orc.assemble(sliver, KC, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    As = nl.stiffnessMatrix_batch([(dict(sliver), KC, conf2d()), (dict(m), KC, conf2d())])
    assert same_pattern(As[0], A) and abs(As[0] - A).max() == 0
    R = orc.assemble(m, KC, conf2d())["A"]
    fro, mx = rel_errors(As[1], R)
    assert same_pattern(As[1], R) and fro < FP64_TOL and mx < FP64_TOL, (fro, mx)


@pytest.mark.parametrize("dim,n,delta,nq", [(3, 3, 0.5, 11), (3, 7, 0.2, 11), (2, 13, 0.15, 1), (2, 12, 0.2, 28)])
def test_fp64_barycenter_pass(nl, orc, dim, n, delta, nq):
    """The one-sided FP64 barycenter pass (constant kernels; one to four mask bytes, a partly filled
    batch on the smallest mesh) against the oracle; graph replays give the same bits."""
    if dim == 3:
        m, c, kern = cube_mesh(n, 0.1, jitter=0.15, seed=n), conf3d(), "constant3D"
    else:
        m, c, kern = square_mesh(n, 0.1, jitter=0.15, seed=n), conf2d(method="baryCenter"), "constant"
        P, w = _split_rule(nq)
        c["quadrature"] = {"outer": {"points": P, "weights": w}, "inner": {"points": P, "weights": w}}
    k = {"function": kern, "horizon": delta, "outputdim": 1}
    A = nl.stiffnessMatrix(dict(m), k, c)
    B = orc.assemble(m, k, c)["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    s = nl.Session([(dict(m), k, c)])
    try:
        for graph in (False, True, True):
            s.assemble(graph=graph)
            C = s.download(0)
            assert same_pattern(A, C) and np.array_equal(A.tocsr().data, C.data)
    finally:
        s.close()


@pytest.mark.parametrize("scale,shift", [(1e-5, 0.0), (1e5, 5.0), (1e-11, 0.0), (1.0, 1e5)])
def test_fp64_pass_scales(nl, orc, scale, shift):
    """The FP64 path on meshes of other units and far from the origin: inside the range of the FP32
    class tests and of the Newton seeds (1e-5, 1e5), and outside of it (horizons of 1e-12, coordinates
    of 1e6 horizons), where the FP64 predicates run. The reference takes its polygon points in absolute
    coordinates, so the bar grows with the coordinates' rounding over the element size (h = 0.1)."""
    m = square_mesh(12, 0.1, jitter=0.2, seed=81)
    from nlfem_gb300 import meshes
    m = meshes.mesh_dict((m["vertices"] + shift) * scale, m["elements"], m["elementLabels"])
    k = {"function": "constant", "horizon": 0.1 * scale, "outputdim": 1}
    A = nl.stiffnessMatrix(dict(m), k, conf2d())
    B = orc.assemble(m, k, conf2d())["A"]
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    tol = FP64_TOL + 64 * 1.1e-16 * shift / 0.1
    assert fro < tol and mx < tol, (fro, mx)


def test_fp64_pass_keeps_vanishing_entries(nl, orc):
    """A sphere within rounding of a vertex: the pair's polygon is far below the elements' own rounding
    and one matrix entry is 1e-24 of the largest. The reference keeps it (only exact zeros are dropped)."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_square(26, 0.1099, jitter=0.2, seed=26)
    rng = np.random.Generator(np.random.PCG64(475299725))
    s, t = int(rng.integers(1, len(v))), int(rng.integers(1, len(e)))
    v = v + rng.uniform(-0.5, 0.5, 2)
    m = meshes.mesh_dict(np.roll(v, s, axis=0), np.roll((e + s) % len(v), t, axis=0), np.roll(l, t))
    k = {"function": "parabola", "horizon": 0.1099, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, conf2d())
    B = orc.assemble(m, k, conf2d())["A"]
    assert abs(B.tocsr().data).min() < 1e-20 * abs(B).max()   # the entry is there
    assert same_pattern(A, B)
    fro, mx = rel_errors(A, B)
    assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)


def _shell_mesh(dim, deg, seed):
    """A vertex with deg neighbours on a circle or sphere around it, and a second shell outside."""
    from scipy.spatial import Delaunay
    from nlfem_gb300 import meshes
    rng = np.random.Generator(np.random.PCG64(seed))
    d = rng.normal(size=(2 * deg, dim))
    d /= np.linalg.norm(d, axis=1)[:, None]
    r = np.where(np.arange(2 * deg) < deg, 0.5, 1.0) * rng.uniform(0.98, 1.02, 2 * deg)
    v = np.vstack([np.zeros((1, dim)), d * r[:, None]])
    e = Delaunay(v).simplices.astype(np.int64)
    vol = np.abs(np.linalg.det(v[e[:, 1:]] - v[e[:, :1]]))
    e = e[vol > 1e-6]
    return meshes.mesh_dict(v, e, np.where(np.arange(len(e)) % 7, 1, -1))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("dim,deg", [(2, 8), (2, 45), (3, 14), (3, 70)])
@pytest.mark.parametrize("delta", [0.12, 0.45, 1.1, 6.0])
def test_search_shells(nl, orc, dim, deg, delta, prec):
    """The pair search on vertices of 8 to more than 64 elements (one and several steps of a warp, with
    and without remainders), at horizons from below the elements' size (no pair near) to far above the
    mesh (every pair near): the pair set is the oracle's, exactly."""
    m = _shell_mesh(dim, deg, 7 * deg + dim)
    k = {"function": "constant" if dim == 2 else "constant3D", "horizon": delta, "outputdim": 1}
    conf = conf2d if dim == 2 else conf3d
    ref = orc.assemble(m, k, conf(), want_pairs=True)["pairs"]
    got = nl.pair_list(m, k, conf(precision=prec))
    np.testing.assert_array_equal(got, ref[np.lexsort((ref[:, 1], ref[:, 0]))])


@pytest.mark.parametrize("n,delta", [(260, 0.02), (40, 0.3)])
@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_numbering_does_not_change_the_matrix(nl, n, delta, prec):
    """Pair lists are ordered by element (near pairs apart) where an element's partners span a few thousand
    numbers, and by the walk where they span more than 131072 (n = 260 renumbered: 1.35e5 elements). Every sum
    over pairs is an integer one in the mixed path, so a renumbered mesh gives the renumbered matrix bit for
    bit; FP64 forms an element's own block in floating point (its pairs' order) and agrees to rounding."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_square(n, delta, jitter=0.2, seed=5)
    rng = np.random.Generator(np.random.PCG64(n))
    pv, pe = rng.permutation(len(v)), rng.permutation(len(e))   # new vertex i is the old pv[i]
    inv = np.argsort(pv)
    k = {"function": "constant", "horizon": delta, "outputdim": 1}
    A = nl.stiffnessMatrix(meshes.mesh_dict(v, e, l), k, conf2d(precision=prec)).tocsr()
    B = nl.stiffnessMatrix(meshes.mesh_dict(v[pv], inv[e[pe]], l[pe]), k, conf2d(precision=prec)).tocsr()
    C = B[inv][:, inv].tocsr()
    assert same_pattern(A, C)
    if prec == "mixed":
        assert np.array_equal(A.data, C.data)
    else:
        assert abs(A.data - C.data).max() < FP64_TOL * abs(A.data).max()


def _graded_mesh(n, delta, p, seed):
    """regular_square with its distances from the centre raised to the power p: elements shrink towards the centre."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_square(n, delta, jitter=0.1, seed=seed)
    d = v - 0.5
    r = np.linalg.norm(d, axis=1)
    return meshes.mesh_dict(0.5 + d * ((r / r.max()) ** (p - 1))[:, None], e, l)


@pytest.mark.parametrize("n,s,p,seed,onesided", [(16, 0.4, 4.25, 3, False), (16, 0.6, 3.75, 3, False), (10, 0.4, 5.25, 3, False),
                                                 (8, 0.5, 5.5, 5, False), (16, 0.4, 5.5, 3, False), (16, 0.4, 2.0, 3, True)])
def test_fp64_singular_sums_on_graded_meshes(nl, orc, n, s, p, seed, onesided):
    """Singular kernels have no rigorous bound for the one-sided FP64 pass's integer sums. On meshes graded
    so far that a sum of contributions, or one of them, could leave the integers' range, the call is handed
    to the general pass (slot_map 0 in the stats), in a one-shot call, in a session and in a graph session;
    moderate grading stays on the one-sided pass. All meet the FP64 bar against the oracle."""
    from nlfem_gb300 import _lib
    m = _graded_mesh(n, 0.3, p, seed)
    k = {"function": "fractional", "horizon": 0.3, "outputdim": 1, "fractional_s": s}
    c = conf2d(rule="7", close="fractional", deg=3)
    B = orc.assemble(m, k, c)["A"]

    def check(A, st):
        assert (st["slot_map"] != 0) == onesided
        assert same_pattern(A, B)
        fro, mx = rel_errors(A, B)
        assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)

    A = nl.stiffnessMatrix(dict(m), k, c)
    check(A, _lib.stats())
    for graph in (False, True):
        sess = nl.Session([(dict(m), k, c)])
        try:
            for _ in range(2):
                st = sess.assemble(graph=graph)
                check(sess.download(0), st)
        finally:
            sess.close()


def _tiny_elements_mesh():
    """Vertices moved to within 1e-7 cells of a neighbour: elements 1e-7 of the others beside them."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_square(14, 0.1, jitter=0.2, seed=91)
    for i in (52, 97, 130, 171):
        v[i] = v[i + 1] + 1e-7 / 14 * np.array([-1.0, 0.3])
    return meshes.mesh_dict(v, e, l)


@pytest.mark.parametrize("case", ["constant", "parabola", "parabola_nocaps", "constant16", "graded", "vanishing", "tiny_bary", "cube"])
def test_fp64_every_entry(nl, orc, case):
    """Every matrix entry of the one-sided FP64 passes to eight digits, not only the large ones: entries from
    slivers that a sphere cuts off are down to 1e-24 of the largest. The bound is the rounding of the
    coordinates (2^-53 of about 1.5) over the least depth of a polygon that the certified structure leaves to
    the pass's own formulas (2^-18 of the horizon, 0.1), times eight."""
    from nlfem_gb300 import meshes, _lib
    c, delta, kern = conf2d(), 0.1, "parabola"
    if case == "vanishing":   # the mesh of test_fp64_pass_keeps_vanishing_entries
        delta = 0.1099
        v, e, l = meshes.regular_square(26, delta, jitter=0.2, seed=26)
        rng = np.random.Generator(np.random.PCG64(475299725))
        s, t = int(rng.integers(1, len(v))), int(rng.integers(1, len(e)))
        v = v + rng.uniform(-0.5, 0.5, 2)
        m = meshes.mesh_dict(np.roll(v, s, axis=0), np.roll((e + s) % len(v), t, axis=0), np.roll(l, t))
    elif case == "graded":
        delta, m = 0.3, _graded_mesh(16, 0.3, 3.0, 3)
    elif case == "tiny_bary":
        delta, kern, m, c = 0.15, "constant", _tiny_elements_mesh(), conf2d(method="baryCenter")
    elif case == "cube":
        delta, kern, m, c = 0.2, "constant3D", cube_mesh(8, 0.1, jitter=0.2, seed=1), conf3d()
    else:
        m = square_mesh(32, delta, jitter=0.2, seed=1)
        if case.startswith("constant"):
            kern = "constant"
        if case == "constant16":
            c = conf2d(rule="16")
        if case == "parabola_nocaps":
            c = conf2d(caps=0)
    k = {"function": kern, "horizon": delta, "outputdim": 1}
    A = nl.stiffnessMatrix(m, k, c).tocsr()
    assert _lib.stats()["slot_map"] != 0
    B = orc.assemble(m, k, c)["A"].tocsr()
    assert same_pattern(A, B)
    off = np.abs(A.data - B.data) / np.abs(B.data)
    assert off.max() < 1e-8, (off.max(), np.abs(B.data)[off.argmax()] / np.abs(B.data).max())


@pytest.mark.parametrize("n,delta,shuffled", [(260, 0.02, True), (260, 0.02, False), (200, 0.012, False), (60, 0.1, False)])
def test_fp64_batch_keeps_the_pair_order(nl, n, delta, shuffled):
    """FP64 forms an element's own block in floating point, in the order of its pair list. That order is the
    problem's alone (element order or the walk's, at any span of the list's element numbers), so a problem behind
    another one in a batch gives the bits of its single assembly."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_square(n, delta, jitter=0.2, seed=5)
    if shuffled:
        pe = np.random.default_rng(n).permutation(len(e))
        e, l = e[pe], l[pe]
    k = {"function": "constant", "horizon": delta, "outputdim": 1}
    m, c = meshes.mesh_dict(v, e, l), conf2d()
    A = nl.stiffnessMatrix(m, k, c).tocsr()
    first = square_mesh(3, 0.1)   # 18 elements: no multiple of a bitmap word
    B = nl.stiffnessMatrix_batch([(first, KC, c), (m, k, c)])[1].tocsr()
    assert same_pattern(A, B) and np.array_equal(A.data, B.data)



@pytest.mark.parametrize("prec", ["fp64", "mixed", "fp64-onesided"])
@pytest.mark.parametrize("kern,h_over_delta", [("constant", 4), ("parabola", 6), ("constant", 6), ("constant", 10)])
def test_partners_without_pairs_of_their_own(nl, orc, kern, h_over_delta, prec):
    """With the centroid rule and elements of 4 to 14 horizons, some elements are partners (a neighbour's ball
    reaches into them) without any pair of their own, not even with themselves (their own ball lies inside
    them: no polygon). Their vertices' rows hold the blocks that their pairs add to them."""
    from nlfem_gb300 import quadrules
    m = square_mesh(14, 0.1, jitter=0.25, seed=8)
    k = {"function": kern, "horizon": 1.2 / 14 * np.sqrt(2.0) / h_over_delta, "outputdim": 1}
    P, w = quadrules.centroid1()
    c = conf2d(precision=prec)
    c["quadrature"] = {"outer": {"points": P, "weights": w}, "inner": {"points": P, "weights": w}}
    r = orc.assemble(m, k, c, want_pairs=True)
    B = r["A"]
    assert len(np.setdiff1d(r["pairs"][:, 1], r["pairs"][:, 0])) > 0
    A = nl.stiffnessMatrix(dict(m), k, c)
    assert same_pattern(A, B)
    if prec != "mixed":   # (these matrices are slivers only, where FP32 has no fixed accuracy)
        fro, mx = rel_errors(A, B)
        assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
    s = nl.Session([(dict(m), k, c)])
    try:
        for _ in range(3):
            s.assemble(graph=True)
            C = s.download(0)
            assert same_pattern(A, C) and np.array_equal(A.tocsr().data, C.data)
    finally:
        s.close()


@pytest.mark.parametrize("kern,h_over_delta,shift", [("constant", 30, 0.0), ("parabola", 52, 0.0), ("constant", 260, 0.0),
                                                     ("fractional", 52, 0.0), ("constant", 0.3, 4e4)])
def test_fp64_onesided_outside_the_certified_range(nl, orc, kern, h_over_delta, shift):
    """precision "fp64-onesided" stays one-sided for elements of 16 to 512 horizons and for meshes far from the
    origin, where its classes come from FP64 tests and every cut polygon from the exact routine."""
    from nlfem_gb300 import meshes, _lib
    n, delta = 24, 1.2 / 24 * np.sqrt(2.0) / h_over_delta
    v, e, l = meshes.regular_square(n, 0.1, jitter=0.2, seed=33)
    m = meshes.mesh_dict(v + shift, e, l)
    k = {"function": kern, "horizon": delta, "outputdim": 1}
    c = conf2d()
    if kern == "fractional":
        k["fractional_s"] = 0.4
        c = conf2d(rule="16", close="fractional", deg=3)
    A = nl.stiffnessMatrix(m, k, dict(c, precision="fp64-onesided"))
    assert _lib.stats()["slot_map"] != 0
    B = orc.assemble(m, k, c)["A"]
    assert same_pattern(A, B)
    if B.nnz:
        fro, mx = rel_errors(A, B)
        tol = FP64_TOL + 64 * 1.1e-16 * shift / 0.05   # the reference's polygon points are absolute
        assert fro < tol and mx < tol, (fro, mx)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_3d_search_elements_naming_a_vertex_twice(nl, orc, prec):
    """Collapsed tetrahedra (a vertex named twice or three times) are found once like any other element: the pair
    list and the matrix are the oracle's."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_cube(4, 0.1, jitter=0.15, seed=6)
    extra = np.array([[e[10][0], e[10][0], e[10][1], e[10][2]], [e[50][1], e[50][3], e[50][1], e[50][0]],
                      [e[90][2], e[90][2], e[90][2], e[90][3]]])
    m = meshes.mesh_dict(v, np.vstack([e, extra]), np.concatenate([l, [1, 1, 1]]))
    k = {"function": "constant3D", "horizon": 0.4, "outputdim": 1}
    ref = orc.assemble(m, k, conf3d(), want_pairs=True)
    got = nl.pair_list(m, k, conf3d(precision=prec))
    np.testing.assert_array_equal(got, ref["pairs"][np.lexsort((ref["pairs"][:, 1], ref["pairs"][:, 0]))])
    A = nl.stiffnessMatrix(m, k, conf3d(precision=prec))
    fro, mx = rel_errors(A, ref["A"])
    tol = FP64_TOL if prec == "fp64" else 1e-6
    assert fro < tol and mx < tol, (fro, mx)


@pytest.mark.parametrize("method", ["retriangulate", "baryCenter"])
@pytest.mark.parametrize("h_over_delta,onesided", [(1.0, True), (10.0, False)])
def test_fp64_outer_points_outside_the_element(nl, orc, method, h_over_delta, onesided):
    """The FP32 tests that decide fp64's search and classes hold for offsets of at most 16 horizons. An outer rule
    with points at 9 element sizes leaves that range with elements of 10 horizons: the FP64 routines take over."""
    from nlfem_gb300 import _lib, quadrules
    m = square_mesh(12, 0.1, jitter=0.2, seed=14)
    k = {"function": "constant", "horizon": 1.2 / 12 * np.sqrt(2.0) / h_over_delta, "outputdim": 1}
    c = conf2d(method=method)
    c["quadrature"]["outer"] = {"points": np.array([[6.0, -3.0], [-3.0, -2.0], [-2.0, 6.0]]), "weights": np.full(3, 1 / 6)}
    A = nl.stiffnessMatrix(m, k, c)
    assert (_lib.stats()["slot_map"] != 0) == onesided
    B = orc.assemble(m, k, c)["A"]
    assert same_pattern(A, B)
    if B.nnz:
        fro, mx = rel_errors(A, B)
        assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)


def _far_triangle(m):
    """m beside a separate triangle of 70 horizons (delta = 0.02), which no ball of m reaches."""
    from nlfem_gb300 import meshes
    v = np.vstack([m["vertices"], [[5.0, 5.0], [6.0, 5.1], [5.2, 6.0]]])
    n = len(m["vertices"])
    return meshes.mesh_dict(v, np.vstack([m["elements"], [[n, n + 1, n + 2]]]), np.append(m["elementLabels"], 1))


@pytest.mark.parametrize("case", ["sliver", "large_element", "full_search", "label_kernel"])
def test_fp64_general_pass_by_its_stats(nl, orc, case):
    """Calls outside the one-sided FP64 pass take the general one, seen in the stats (slot_map 0): alone, and together
    with an ordinary problem that takes the one-sided pass by itself."""
    from nlfem_gb300 import meshes, _lib
    m, k, c = square_mesh(10, 0.02, jitter=0.1, seed=73), {"function": "constant", "horizon": 0.02, "outputdim": 1}, conf2d()
    bad, kb, cb = m, dict(k), dict(c)
    if case == "sliver":
        v = m["vertices"].copy()
        v[0] = 0.5 * (v[1] + v[12]) + np.array([-3e-13, 3e-13])   # onto the opposite side of its triangle (0, 1, 12)
        bad = meshes.mesh_dict(v, m["elements"], m["elementLabels"])
    elif case == "large_element":
        bad = _far_triangle(m)
    elif case == "full_search":
        cb["is_fullConnectedComponentSearch"] = 1
    else:
        kb["function"] = "labeled"
        bad = labeled_mesh(10)
        kb["horizon"] = 0.1
    ref, ok = orc.assemble(bad, kb, cb)["A"], orc.assemble(m, k, c)["A"]

    def check(A, B):
        assert same_pattern(A, B)
        fro, mx = rel_errors(A, B)
        assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)

    check(nl.stiffnessMatrix(dict(m), k, c), ok)
    assert _lib.stats()["slot_map"] != 0
    check(nl.stiffnessMatrix(dict(bad), kb, cb), ref)
    assert _lib.stats()["slot_map"] == 0
    A, B = nl.stiffnessMatrix_batch([(dict(bad), kb, cb), (dict(m), k, c)])
    assert _lib.stats()["slot_map"] == 0
    check(A, ref)
    check(B, ok)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("close", ["fractional", "weakSingular"])
def test_close_pair_slots_that_hold_no_pair(nl, orc, close, prec):
    """Close-pair slots of label-0 elements, and in a batch those of a problem whose kernel has no Duffy rule,
    hold no pair and are passed over."""
    from nlfem_gb300 import meshes
    v, e, l = meshes.regular_square(15, 0.1, jitter=0.2, seed=38)
    l = np.random.default_rng(38).choice([1, 1, 1, -1, 0], size=len(e))
    m = meshes.mesh_dict(v, e, l)
    s = 0.4 if close == "fractional" else 0.3
    k = {"function": "fractional", "horizon": 0.11, "outputdim": 1, "fractional_s": s}
    c = conf2d(rule="16", close=close, deg=3, precision=prec)
    other = (square_mesh(9, 0.1, jitter=0.1, seed=2), {"function": "constant", "horizon": 0.15, "outputdim": 1},
             conf2d(rule="16", precision=prec))
    tol = FP64_TOL if prec == "fp64" else 1e-6
    A = nl.stiffnessMatrix(m, k, c)
    As = nl.stiffnessMatrix_batch([other, (m, k, c)])
    B, C = orc.assemble(m, k, c)["A"], orc.assemble(*other)["A"]
    for X, Y in ((A, B), (As[0], C), (As[1], B)):
        assert same_pattern(X, Y)
        fro, mx = rel_errors(X, Y)
        assert fro < tol and mx < tol, (fro, mx)


def test_threads_of_different_sizes(nl):
    """One-shot calls of four threads at once, of different sizes, rules, kernels and precisions (different shared-memory
    needs of the same kernels), give the bits of the same calls one after the other."""
    import threading
    calls = []
    for i, (n, rule, kern, prec) in enumerate([(4, "7", "constant", "fp64"), (30, "16", "constant", "fp64"), (12, "7", "parabola", "mixed"),
                                               (60, "7", "constant", "mixed"), (8, "16", "parabola", "fp64"), (24, "16", "parabola", "mixed"),
                                               (40, "7", "constant", "fp64"), (10, "16", "constant", "mixed")]):
        calls.append((square_mesh(n, 0.1, jitter=0.2, seed=i), {"function": kern, "horizon": 0.1, "outputdim": 1}, conf2d(rule=rule, precision=prec)))
    want = [nl.stiffnessMatrix(*c).tocsr() for c in calls]
    errors = []

    def work(t):
        try:
            for r in range(24):
                i = (5 * r + 3 * t) % len(calls)
                A = nl.stiffnessMatrix(*calls[i]).tocsr()
                if not (same_pattern(A, want[i]) and np.array_equal(A.data, want[i].data)):
                    errors.append((t, r, i))
        except Exception as ex:
            errors.append((t, repr(ex)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[:4]


@pytest.mark.parametrize("case", ["fp64", "mixed", "bary_fp64", "bary_mixed", "label_fp64", "dim3_fp64", "dim3_mixed"])
def test_pattern_of_meshes_too_large_for_bitmaps(nl, orc, case):
    """From 819,200 vertices on, a problem's vertex bitmap leaves shared memory and the rows are built from marks in
    global memory. A small mesh numbered behind unused vertices takes that path, in the passes that read pair
    arrays: its rows are those of the mesh by itself."""
    from nlfem_gb300 import meshes, _lib
    prec = case.split("_")[-1]
    k = {"function": "constant", "horizon": 0.12, "outputdim": 1}
    if case.startswith("dim3"):
        m, c, k["function"] = cube_mesh(4, 0.1, jitter=0.15, seed=3), conf3d(prec), "constant3D"
        k["horizon"] = 0.3
    else:
        m = labeled_mesh(12) if case.startswith("label") else square_mesh(13, 0.1, jitter=0.2, seed=3)
        c = conf2d(method="baryCenter" if case.startswith("bary") else "retriangulate", precision=prec)
        if case.startswith("label"):
            k["function"] = "labeled"
    pad = 820000
    v = np.vstack([np.zeros((pad, m["vertices"].shape[1])), m["vertices"]])
    v[:pad] = m["vertices"][0]
    big = meshes.mesh_dict(v, m["elements"] + pad, m["elementLabels"])
    A = nl.stiffnessMatrix(big, k, c).tocsr()
    st = _lib.stats()
    B = nl.stiffnessMatrix(dict(m), k, c).tocsr()
    assert A.indptr[pad] == 0 and st["n_pairs"] == _lib.stats()["n_pairs"]
    C = A[pad:, pad:]
    assert C.nnz == A.nnz and same_pattern(C, B)
    if prec == "mixed":
        assert abs(C - B).max() < 1e-6 * abs(B).max()
    else:
        fro, mx = rel_errors(C, orc.assemble(m, k, c)["A"])
        assert fro < FP64_TOL and mx < FP64_TOL, (fro, mx)
