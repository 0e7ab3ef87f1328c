"""CPU check, on the oracle's operator, of the two algebraic forms that the
solver and the Gauss projection compute in (no GPU).

The operator in its spin structure: with real Wilson coefficients the 6x6 block
to the neighbour x + I follows from three colour matrices for both species,
  I = 0, 1:  quark [[m0, m2], [-+m2, m1]], antiquark [[-m1, m2], [-+m2, -m0]]
  I = 2:     quark [[m0, m2], [m1, m0]],   antiquark [[-m0, m2], [m1, -m0]]
(lower sign for I = 1; spin blocks), the backward block is -W_I(x - I)^H, the
site term 1 + i (S0 +- S1) with hermitian S0, S1 in colour alone, and A = 2 -
A^H.

The Gauss sweep in coordinates: with the adjoint matrix R of a link, T = R^T E
and E' = E + kdt (1/2 d_abc (R G)_b G'_c - G_a)."""
import numpy as np
import pytest

C = np.array([1, 1, 1, 1], dtype=complex)


def _block(oracle, n, a, links, ef, mass, dt, species, x, y):
    """The 6x6 block of A^H from site y to site x (rows and columns colour*2 + spin)."""
    V = int(np.prod(n))
    psi = np.zeros((V, 6, 6), dtype=complex)
    psi[y] = np.eye(6)
    out = oracle.cn_apply(n, a, links, ef, species * mass, C, dt, 1, psi)
    return out[x].T  # (column, row) -> row, column


def _site(n, p):
    return (p[0] % n[0]) + n[0] * ((p[1] % n[1]) + n[1] * (p[2] % n[2]))


@pytest.mark.parametrize("n,a", [((4, 3, 5), (0.05, 1.0, 1.0, 1.0)), ((3, 4, 3), (0.1, 1.0, 0.9, 1.2))])
def test_three_matrices_a_direction(oracle, n, a):
    links, ef = oracle.transverse_box(n, a, 3.0, 1.0, 0.0, 5, identity_links=False)
    mass, dt = 1.3, 1.0
    get = lambda sp, x, y: _block(oracle, n, a, links, ef, mass, dt, sp, x, y)
    spin = lambda b, r, c: b[r::2, c::2]
    # entries are sums of a few products of numbers up to one; A^H - 1 is of
    # size 0.1: rounding of 1e-16 a product
    tol = 1e-15
    p = (1, 2, 1)
    x = _site(n, p)
    for i in range(3):
        q = list(p)
        q[i] += 1
        y = _site(n, q)
        w, v = get(+1, x, y), get(-1, x, y)
        off, sgn = spin(w, 0, 1), -1 if i == 0 else 1
        if i < 2:
            m0, m1, m2 = spin(w, 0, 0), spin(w, 1, 1), off
            quark = ((m0, m2), (sgn * m2, m1))
            anti = ((-m1, m2), (sgn * m2, -m0))
        else:
            m0, m2, m1 = spin(w, 0, 0), off, spin(w, 1, 0)
            quark = ((m0, m2), (m1, m0))
            anti = ((-m0, m2), (m1, -m0))
        for r in range(2):
            for c in range(2):
                assert np.abs(spin(w, r, c) - quark[r][c]).max() < tol
                assert np.abs(spin(v, r, c) - anti[r][c]).max() < tol
        assert np.abs(m2).max() > 1e-6  # the spin-orbit term is there
        # the block back from x to y
        for sp, f in ((+1, w), (-1, v)):
            assert np.abs(get(sp, y, x) + f.conj().T).max() < tol
    s, t = get(+1, x, x) - np.eye(6), get(-1, x, x) - np.eye(6)
    for b in (s, t):
        assert max(np.abs(spin(b, 0, 1)).max(), np.abs(spin(b, 1, 0)).max()) < tol
        assert np.abs(spin(b, 0, 0) - spin(b, 1, 1)).max() < tol
    s0, s1 = (spin(s, 0, 0) + spin(t, 0, 0)) / 2j, (spin(s, 0, 0) - spin(t, 0, 0)) / 2j
    assert np.abs(s0 - s0.conj().T).max() < tol and np.abs(s1 - s1.T).max() < tol
    assert np.abs(s1.imag).max() < tol


def test_a_is_two_minus_its_adjoint(oracle):
    n, a = (3, 4, 2), (0.05, 1.0, 1.1, 1.0)
    links, ef = oracle.transverse_box(n, a, 3.0, 1.0, 0.0, 5, identity_links=False)
    rng = np.random.default_rng(1)
    V = int(np.prod(n))
    psi = rng.normal(size=(V, 6, 6)) + 1j * rng.normal(size=(V, 6, 6))
    f = [oracle.cn_apply(n, a, links, ef, 1.0, C, 1.0, h, psi) for h in (0, 1)]
    assert np.abs(f[0] + f[1] - 2 * psi).max() < 1e-14


def test_gauss_sweep_in_coordinates(oracle):
    n, a = (3, 4, 2), (0.1, 1.0, 0.9, 1.1)
    links, ef = oracle.transverse_box(n, a, 2.0, 1.0, 0.0, 9, identity_links=False)
    rng = np.random.default_rng(4)
    ef = ef + 0.02 * rng.standard_normal(ef.shape)
    want, kept = ef.copy(), links.copy()
    assert oracle.gauss_project(n, a, kept, want, tol=1e-12, max_sweeps=3) == 3

    T = np.stack([oracle.generator(k + 1) for k in range(8)])
    V = int(np.prod(n))
    u = links.reshape(V, 3, 3, 3).swapaxes(-1, -2)  # stored column by column
    R = 2 * np.einsum("aij,xkjl,blm,xkim->xkab", T, u, T, u.conj(), optimize=True).real
    d = 4 * np.einsum("aij,bjk,cki->abc", T, T, T).real
    E = ef.reshape(V, 3, 8).copy()
    idx = np.arange(V).reshape(n[2], n[1], n[0])
    up = [np.roll(idx, -1, axis=2 - k).ravel() for k in range(3)]
    dn = [np.roll(idx, 1, axis=2 - k).ravel() for k in range(3)]
    for _ in range(3):
        t = np.einsum("xkba,xkb->xka", R, E)
        G = sum((E[:, k] - t[dn[k], k]) / (a[k + 1] * a[0]) for k in range(3))
        for k in range(3):
            r = np.einsum("xab,xb->xa", R[:, k], G)
            E[:, k] += 0.01 * a[0] * (0.5 * np.einsum("abc,xb,xc->xa", d, r, G[up[k]]) - G)
    # three sweeps of numbers up to one
    assert np.abs(E - want.reshape(V, 3, 8)).max() < 3e-15
