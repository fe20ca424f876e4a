"""NumPy model of the symmetric real-basis vertex (csrc/even_impl.cuh, k_vertex_sym,
tables of csrc/even.cu, build_sym) against the complex formula.

The model keeps the kernel's storage (cyclic diagonals, entry (p, p + d) at d n + p),
its rows dealt out over lanes, the pivot column published twice over, and the sweep
with the largest remaining diagonal entry as pivot.  The bound is 1e-12 of the
largest element: 25 sweeps of rounding 1.1e-16 at condition numbers below 1e2.
"""
import numpy as np
import pytest


def sym_at(n, p, q):
    d = (q - p) % n
    return d * n + p if 2 * d < n or (2 * d == n and p < q) else (n - d) * n + q


def basis_of(No):
    pairs = [(a, b) for a in range(No) for b in range(No)]
    at = {p: i for i, p in enumerate(pairs)}
    perm = [at[(b, a)] for a, b in pairs]
    basis = [(0, l) for l in range(No * No) if perm[l] == l]
    basis += [(k, l) for k in (1, 2) for l in range(No * No) if l < perm[l]]
    return perm, basis


def transforms(No):
    """T (rows of the basis) and its inverse: A' = T A T^-1 is real."""
    perm, basis = basis_of(No)
    n = No * No
    T, Ti = np.zeros((n, n), complex), np.zeros((n, n), complex)
    for p, (k, l) in enumerate(basis):
        m = perm[l]
        if k == 0:
            T[p, l] = Ti[l, p] = 1
        else:
            f = 1 if k == 1 else 1j
            T[p, l], T[p, m] = f, f if k == 1 else -f
            Ti[l, p], Ti[m, p] = 0.5 / f, 0.5 / f if k == 1 else -0.5 / f
    assert np.allclose(T @ Ti, np.eye(n))
    h = np.array([{0: 1.0, 1: 2.0, 2: -2.0}[k] for k, _ in basis])
    return T, Ti, h


def sweep(M, rows=4):
    """-M^-1 and whether a pivot fell below an eighth of its column."""
    n = len(M)
    DG, DK = n // 2 + 1, n // 2 + 1 if n % 2 else n // 2
    G = 32 * rows // n
    assert all(0 <= r // n < G for r in range(G * n))
    a = np.array([[M[i, (i + d) % n] for d in range(DG)] for i in range(n)])
    done, bad = np.zeros(n, bool), False
    for _ in range(n):
        k = int(np.where(done, -1.0, np.abs(a[:, 0])).argmax())
        p = a[k, 0]
        col, writers = np.full(2 * n, np.nan), np.zeros(n, int)
        for i in range(n):
            dd = (k - i) % n
            if dd < DG:
                col[i] = col[i + n] = a[i, dd]
                writers[i] += 1
        for d in range(1, DK):
            j = (k + d) % n
            col[j] = col[j + n] = a[k, d]
            writers[j] += 1
        assert (writers == 1).all()  # one lane writes each entry
        new = np.empty_like(a)
        for i in range(n):
            dd, c = (k - i) % n, col[i]
            f = 1 / p if dd == 0 else -(c / p)
            bad |= bool(dd and not done[i] and abs(c) > 8 * abs(p))
            for d in range(DG):
                assert i + d < 2 * n
                new[i, d] = -f if d == dd else f * col[i + d] + (0.0 if dd == 0 else a[i, d])
        a, done[k] = new, True
    return a, bad


def chi_of(No, rng, scale):
    """A chi0(q, i nu) of an even model: symmetric, P chi P = conj chi."""
    perm, _ = basis_of(No)
    n = No * No
    x = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    x = x + x.T
    x = x + x[np.ix_(perm, perm)].conj()
    pos = rng.normal(size=(n, n))
    pos = pos @ pos.T
    pos = pos + pos[np.ix_(perm, perm)]
    return scale * (pos / np.abs(pos).max() + 0.3 * x / np.abs(x).max())


@pytest.mark.parametrize("No", [3, 4, 5])
def test_sweep_model_gives_the_vertex(No):
    rng = np.random.default_rng(No)
    n = No * No
    perm, basis = basis_of(No)
    T, Ti, h = transforms(No)
    for _ in range(3):
        s = rng.normal(size=(n, n)) * 0.02
        s = s + s.T
        S = np.eye(n) + s + s[np.ix_(perm, perm)]
        chi = chi_of(No, rng, 0.1)
        A = T @ (np.linalg.inv(S) - chi) @ Ti
        assert np.abs(A.imag).max() < 1e-13
        M = A.real * h[None, :]
        assert np.abs(M - M.T).max() < 1e-13
        W, bad = sweep(M)
        assert not bad
        half = np.array([[-W[p if sym_at(n, p, q) % n == p and (q - p) % n == sym_at(n, p, q) // n else q,
                            sym_at(n, p, q) // n] for q in range(n)] for p in range(n)])
        V = Ti @ (h[:, None] * half) @ T
        ref = S @ np.linalg.inv(np.eye(n) - chi @ S)
        assert np.abs(V - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("n", [9, 16, 25])
def test_storage_covers_every_pair_once(n):
    at = {}
    for p in range(n):
        for q in range(n):
            e = sym_at(n, p, q)
            assert 0 <= e < (n // 2 + 1) * n
            d, i = divmod(e, n)
            assert {i, (i + d) % n} == {p, q} or p == q == i and d == 0
            at.setdefault(e, set()).add(frozenset((p, q)))
    assert all(len(v) == 1 for v in at.values()) and len(at) == n * (n + 1) // 2


def test_indefinite_matrix_is_left_to_the_pivoted_kernel():
    M = np.zeros((9, 9))
    M[np.arange(9), (np.arange(9) + 1) % 9] = 1.0
    M = M + M.T + 0.01 * np.eye(9)
    assert sweep(M)[1]
