"""Generator of the Rys quadrature tables (roots t_i^2 and weights, one to six points).

The n-point Rys quadrature integrates polynomials of degree 2n - 1 in t^2 against e^(-T t^2) on
[0, 1] (Dupuis, Rys & King, J. Chem. Phys. 65, 111 (1976)).  Per n the table holds, on intervals
of width H up to TMAX[n], a polynomial in T - (interval centre) for each root and each weight,
in monomial form (highest power last), interpolated at the Chebyshev points of the interval.
Above TMAX[n] the quadrature is the half-range Gauss-Hermite one scaled by 1/T: the integral from
1 to infinity that separates the two is below 1e-15 of every moment there.

The nodal values come from the discretised Stieltjes procedure (Gautschi, "Orthogonal
Polynomials: Computation and Approximation", sec. 2.2): the weight function on a Gauss-Legendre
grid, the recurrence coefficients by inner products, the roots by Newton's method on the
recurrence and the weights from the orthonormal polynomials, in 80-bit arithmetic.
"""
from __future__ import annotations

import os

import numpy as np

LD = np.longdouble
NMAX = 6                       # points: total angular momentum up to 10 after differentiation
H = 0.5                        # interval width
NCOEF = 12                     # polynomial coefficients per value (even: 16-byte loads)
TMAX = {1: 40.0, 2: 44.0, 3: 48.0, 4: 53.0, 5: 58.0, 6: 62.0}
PI = LD("3.14159265358979323846264338327950288")


def legendre(n, lo, hi):
    """Gauss-Legendre nodes and weights on [lo, hi] in 80-bit arithmetic."""
    x = np.polynomial.legendre.leggauss(n)[0].astype(LD)
    for _ in range(4):
        p0, p1 = np.ones_like(x), x.copy()
        for k in range(1, n):
            p0, p1 = p1, ((2 * k + 1) * x * p1 - k * p0) / (k + 1)
        d = n * (x * p1 - p0) / (x * x - 1)
        x = x - p1 / d
    w = 2 / ((1 - x * x) * d * d)
    return LD(lo) + (x + 1) * (LD(hi) - LD(lo)) / 2, w * (LD(hi) - LD(lo)) / 2


def gauss_from_measure(x, w, n):
    """n-point Gauss rules of the discrete measures (points x, weights w[..., len(x)]):
    nodes and weights, shape [..., n]."""
    pm, p = np.zeros_like(w), np.ones_like(w)
    norm_prev = None
    alpha, beta = [], []
    for k in range(n):
        norm = (w * p * p).sum(-1)
        a = (w * x * p * p).sum(-1) / norm
        b = norm if k == 0 else norm / norm_prev
        alpha.append(a)
        beta.append(b)
        pm, p = p, (x - a[..., None]) * p - (0 if k == 0 else b[..., None]) * pm
        norm_prev = norm
    J = np.zeros(w.shape[:-1] + (n, n))
    for k in range(n):
        J[..., k, k] = alpha[k]
        if k:
            J[..., k, k - 1] = J[..., k - 1, k] = np.sqrt(beta[k].astype(float))
    r = np.linalg.eigvalsh(J).astype(LD)

    def poly(z):
        q0, q1, d0, d1 = np.zeros_like(z), np.ones_like(z), np.zeros_like(z), np.zeros_like(z)
        for k in range(n):
            a, b = alpha[k][..., None], (beta[k][..., None] if k else LD(0))
            q0, q1, d0, d1 = q1, (z - a) * q1 - b * q0, d1, q1 + (z - a) * d1 - b * d0
        return q1, d1

    for _ in range(4):
        f, d = poly(r)
        r = r - f / d
    s = np.zeros_like(r)
    q0, q1 = np.zeros_like(r), np.ones_like(r) / np.sqrt(beta[0])[..., None]
    for k in range(n):
        s = s + q1 * q1
        if k + 1 < n:
            bk = np.sqrt(beta[k])[..., None] if k else LD(0)
            q0, q1 = q1, ((r - alpha[k][..., None]) * q1 - bk * q0) / np.sqrt(beta[k + 1])[..., None]
    return r, 1 / s


def rys(T, n):
    """Roots t^2 and weights of the n-point rule at the points T (80-bit)."""
    t, w = legendre(120, 0, 1)
    T = np.atleast_1d(np.asarray(T, dtype=LD))
    return gauss_from_measure(t * t, np.exp(-T[:, None] * (t * t)) * w, n)


def hermite(n):
    """Half-range Gauss-Hermite rule in x^2: squares of the nodes and weights (80-bit)."""
    t, w = legendre(400, 0, 13)
    r, q = gauss_from_measure(t * t, (np.exp(-t * t) * w)[None, :], n)
    return r[0], q[0]


def table(n):
    """Coefficients [intervals, 2n, NCOEF]: roots first, then weights."""
    m = int(round(TMAX[n] / H))
    k = np.arange(NCOEF, dtype=LD)
    z = np.cos(PI * (2 * k + 1) / (2 * NCOEF))  # Chebyshev points
    centre = (np.arange(m, dtype=LD) + LD(0.5)) * LD(H)
    r, w = rys((centre[:, None] + z * LD(H) / 2).ravel(), n)
    v = np.concatenate([r, w], 1).reshape(m, NCOEF, 2 * n)
    # Chebyshev coefficients, then monomials in z, then in T - centre
    cheb = np.cos(np.outer(k, PI * (2 * k + 1) / (2 * NCOEF))) * LD(2) / NCOEF
    cheb[0] /= 2
    mono = np.zeros((NCOEF, NCOEF), dtype=LD)
    mono[0, 0] = 1
    mono[1, 1] = 1
    for j in range(2, NCOEF):
        mono[j, 1:] = 2 * mono[j - 1, :-1]
        mono[j] -= mono[j - 2]
    c = np.einsum("jk,mkv->mvj", cheb, v)
    c = np.einsum("mvj,jp->mvp", c, mono)
    return c / (LD(H) / 2) ** k


def emit(outdir):
    """rys_layout.cuh (sizes, offsets, Hermite constants) and rys_table.cu (the coefficients)."""
    off, rows = {}, []
    pos = 0
    for n in range(1, NMAX + 1):
        c = table(n).astype(np.float64)
        off[n] = pos
        pos += c.size
        rows.append(c.ravel())
    flat = np.concatenate(rows)
    herm = [hermite(n) for n in range(1, NMAX + 1)]
    pad = lambda a: list(a.astype(np.float64)) + [0.0] * (NMAX - len(a))  # noqa: E731
    lay = ["// GENERATED by gen_rys.py -- do not edit.", "#pragma once",
           f"constexpr int kRysMaxRoots = {NMAX};",
           f"constexpr int kRysCoef = {NCOEF};", f"constexpr double kRysInvH = {1.0 / H!r};",
           f"constexpr double kRysH = {H!r};",
           "__host__ __device__ constexpr int rys_offset(int n) {", "  return " +
           " : ".join(f"n == {n} ? {off[n]}" for n in range(1, NMAX)) + f" : {off[NMAX]};", "}",
           "__host__ __device__ constexpr double rys_tmax(int n) {", "  return " +
           " : ".join(f"n == {n} ? {TMAX[n]!r}" for n in range(1, NMAX)) + f" : {TMAX[NMAX]!r};", "}",
           "// half-range Gauss-Hermite: squared nodes, then weights",
           f"static __constant__ double c_rys_herm[{NMAX}][2][{NMAX}] = {{"]
    for r, w in herm:
        lay.append("  {{" + ", ".join(map(repr, map(float, pad(r)))) + "}, {" +
                   ", ".join(map(repr, map(float, pad(w)))) + "}},")
    lay += ["};", ""]
    src = ["// GENERATED by gen_rys.py -- do not edit.", "#include <cuda_runtime.h>",
           f"__device__ __align__(16) double hfgpu_rys_table_data[{len(flat)}] = {{"]
    src += ["  " + ", ".join(repr(float(x)) for x in flat[i:i + 8]) + "," for i in range(0, len(flat), 8)]
    src += ["};", "// device address of the table on the current device (nullptr on failure)",
            "const double* hfgpu_rys_table() {", "  void* p = nullptr;",
            "  if (cudaGetSymbolAddress(&p, hfgpu_rys_table_data) != cudaSuccess) return nullptr;",
            "  return static_cast<const double*>(p);", "}", ""]
    for name, text in (("rys_layout.cuh", lay), ("rys_table.cu", src)):
        path, text = os.path.join(outdir, name), "\n".join(text)
        if not (os.path.exists(path) and open(path).read() == text):
            with open(path, "w") as f:
                f.write(text)
