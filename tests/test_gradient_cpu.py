"""The one-kernel gradient's arithmetic (gradient.cuh, compiled for the host)
against the oracle's five passes: pairing arrays, criticality and tetrahedron
codes of every cell, with ties, signed zeros, extreme values and grids down to
2 x 2 x 2.  Whole numbers: equality."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "dmtz_gb300", "csrc"))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    out = str(tmp_path_factory.mktemp("grad") / "gradient_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-o", out, os.path.join(HERE, "native", "gradient_check.cu")],
                   check=True, capture_output=True)
    return out


def cell_ids(dims):
    """Reference ids of every anchor's edges (7), triangles (12) and tetrahedra (6), -1 where absent."""
    import gen_topology as G

    W, H, D = dims
    z, y, x = (a.reshape(-1) for a in np.meshgrid(np.arange(D), np.arange(H), np.arange(W), indexing="ij"))
    c = [(W - 1) * H * D, W * (H - 1) * D, W * H * (D - 1), (W - 1) * (H - 1) * D, W * (H - 1) * (D - 1),
         (W - 1) * H * (D - 1)]
    o = np.concatenate([[0], np.cumsum(c)])
    bxy = 2 * D * (W - 1) * (H - 1)
    byz = bxy + 2 * W * (H - 1) * (D - 1)
    bxz = byz + 2 * H * (W - 1) * (D - 1)
    row, xy = (W - 1) * (H - 1), y * (W - 1) + x
    ed = [z * (W - 1) * H + xy, o[1] + z * W * (H - 1) + x * (H - 1) + y, o[2] + y * W * (D - 1) + x * (D - 1) + z,
          o[3] + z * row + xy, o[4] + x * (H - 1) * (D - 1) + y * (D - 1) + z,
          o[5] + y * (W - 1) * (D - 1) + z * (W - 1) + x, o[6] + z * row + xy]
    fa = [2 * (z * row + xy) + s for s in (0, 1)]
    fa += [bxy + 2 * (x * (H - 1) * (D - 1) + y * (D - 1) + z) + s for s in (0, 1)]
    fa += [byz + 2 * (y * (W - 1) * (D - 1) + z * (W - 1) + x) + s for s in (0, 1)]
    fa += [bxz + 6 * (z * row + xy) + s for s in range(6)]
    te = [6 * (z * row + xy) + s for s in range(6)]
    res = []
    for ids, cells in ((ed, G.EDGES), (fa, G.FACES), (te, G.TETS)):
        a = np.stack(ids, 1)
        for k, cell in enumerate(cells):
            m = [max(p[i] for p in cell) for i in range(3)]
            a[(x + m[0] >= W) | (y + m[1] >= H) | (z + m[2] >= D), k] = -1
        res.append(a)
    return res


def decode(raw, dims):
    """(PV, PE, PF, PT, crit, tcode ok) from the anchors' words, in the reference's layout."""
    import gen_topology as G

    W, H, D = dims
    V = W * H * D
    pv = raw[:V]
    eup, fup, crit, tcode = np.frombuffer(raw[V:].tobytes(), np.uint32).reshape(4, V)
    E, F, T = cell_ids(dims)
    v = np.arange(V)
    off = lambda d: d[0] + W * (d[1] + H * d[2])  # noqa: E731
    PV = np.full(V, -1)
    PE, PF, PT = (np.full(a.max() + 1, -1) for a in (E, F, T))
    for d, dv in enumerate(G.DIRS):
        lo = tuple(min(0, c) for c in dv)
        k = G.EDGE_OF[frozenset((G.sub((0, 0, 0), lo), G.sub(dv, lo)))]
        i = v[pv == d]
        PV[i] = E[i + off(lo), k]
        PE[PV[i]] = i
    for k in range(7):
        for j, (a, s, _) in enumerate(G.edge_cofaces(k)):
            i = v[((eup >> (3 * k)) & 7) == j + 1]
            assert (E[i, k] >= 0).all()
            PE[E[i, k]] = F[i + off(a), s]
            PF[F[i + off(a), s]] = E[i, k]
        assert (E[((eup >> (3 * k)) & 7) != 0, k] >= 0).all()
    for s in range(12):
        for j, (a, t, _) in enumerate(G.face_cofaces(s)):
            i = v[((fup >> (2 * s)) & 3) == j + 1]
            assert (F[i, s] >= 0).all()
            PF[F[i, s]] = T[i + off(a), t]
            PT[T[i + off(a), t]] = F[i, s]
        assert (((fup >> (2 * s)) & 3) < 3).all()
    tet = np.full(len(PT), -1)
    for t in range(6):
        code = (tcode >> (3 * t)) & 7
        assert (code[T[:, t] < 0] == 7).all()
        for j, (a, s, _) in enumerate(G.tet_faces(t)):
            i = v[code == j]
            tet[T[i, t]] = F[i + off(a), s]
    assert np.array_equal(tet, PT)
    want = (pv == 15).astype(np.uint32)
    for a, P, b in ((E, PE, 1), (F, PF, 8), (T, PT, 20)):
        for k in range(a.shape[1]):
            want |= ((a[:, k] >= 0) & (P[a[:, k]] < 0)).astype(np.uint32) << (b + k)
    assert np.array_equal(crit, want)
    return PV, PE, PF, PT


FIELDS = {
    "normal": lambda r, n: r.standard_normal(n),
    "ties": lambda r, n: r.integers(0, 3, n).astype(np.float64),
    "constant": lambda r, n: np.zeros(n),
    "zeros": lambda r, n: r.choice([0.0, -0.0, 1e-310, -1e-310], n),
    "extreme": lambda r, n: r.choice([-np.finfo(float).max, np.finfo(float).max, 0.0], n),
}


@pytest.mark.parametrize("dims", [(2, 2, 2), (2, 5, 3), (7, 2, 2), (3, 3, 3), (9, 6, 5), (33, 17, 4)])
@pytest.mark.parametrize("kind", sorted(FIELDS))
def test_stages_match_the_five_passes(exe, tmp_path, dims, kind):
    from oracle import oracle as O

    n = dims[0] * dims[1] * dims[2]
    f = FIELDS[kind](np.random.default_rng(n), n)
    src, dst = str(tmp_path / "in.bin"), str(tmp_path / "out.bin")
    with open(src, "wb") as fh:
        fh.write(np.asarray(dims, np.int32).tobytes() + f.tobytes())
    subprocess.run([exe, src, dst], check=True)
    got = decode(np.fromfile(dst, np.uint8), dims)
    for g, w, name in zip(got, O.pair(f, dims), ("PV", "PE", "PF", "PT")):
        assert np.array_equal(g, w), name
