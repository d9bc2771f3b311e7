// Stable Neo-Hookean energy of one tet in F = dx/dX (column-major):
//   Psi = mu/2 (|F|^2 - 3) - mu (J - 1) + lambda/2 (J - 1)^2,  J = det F,
//   dPsi/dF = mu F + s g,  d2Psi/dF2 = mu I + lambda g g^T + s d2J,
// with g = dJ/dF and s = lambda (J - 1) - mu, and the projection of the
// Hessian to positive semidefinite in closed form.
//
// With F = U diag(sg) V^T (U, V rotations, sg_2 signed), the Hessian acts on
// A = U^T dF V blockwise (Smith, de Goes, Kim 2018, "Stable Neo-Hookean Flesh
// Simulation", section 4): each pair (A_ab, A_ba), k the third index, has the
// eigenvalues mu - s sg_k (symmetric) and mu + s sg_k (antisymmetric), and the
// diagonal of A sees the 3x3 matrix mu I + lambda gs gs^T + s [off-diagonal
// sg_k]. Clamping those six values and the 3x3 matrix's eigenvalues at zero is
// the projection. The parts are:
//   m[a][c]: the diagonal's 3x3 matrix, clamped;
//   p[k], q[k]: half the sum and half the difference of the pair's clamped
//   values: A_ab is weighted by p_k, its partner A_ba by q_k.
#pragma once

namespace b2s
{
namespace snh
{
struct Projected
{
    double u[3][3], v[3][3];  // columns of U, V: u[i] is column i
    double m[3][3], p[3], q[3];
};

__device__ inline double dot3(const double* a, const double* b) { return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]; }
__device__ inline void cross3(const double* a, const double* b, double* c)
{
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

// one rotation of the columns P, Q of a and v that makes a_P and a_Q
// orthogonal; false when they already are (to rounding). A pair that is not
// finite counts as orthogonal.
template <int P, int Q>
__device__ inline bool rotate_columns(double a[3][3], double v[3][3])
{
    const double al = dot3(a[P], a[P]), be = dot3(a[Q], a[Q]), ga = dot3(a[P], a[Q]);
    if(!(ga * ga > 1e-31 * (al * be)))
        return false;
    // t = sign(z) / (|z| + sqrt(z^2 + 1)) of z = d / g without forming z
    const double d = be - al, g = 2.0 * ga;
    const double t = (d >= 0.0 ? g : -g) / (fabs(d) + sqrt(d * d + g * g));
    const double c = rsqrt(t * t + 1.0), s = c * t;
    for(int r = 0; r < 3; ++r)
    {
        const double ap = a[P][r], aq = a[Q][r], vp = v[P][r], vq = v[Q][r];
        a[P][r] = c * ap - s * aq;
        a[Q][r] = s * ap + c * aq;
        v[P][r] = c * vp - s * vq;
        v[Q][r] = s * vp + c * vq;
    }
    return true;
}

// a unit vector orthogonal to the unit vector u
__device__ inline void any_orthogonal(const double* u, double* w)
{
    const double x = fabs(u[0]), y = fabs(u[1]), z = fabs(u[2]);
    const double e[3] = {x <= y && x <= z ? 1.0 : 0.0, !(x <= y && x <= z) && y <= z ? 1.0 : 0.0,
                         !(x <= y && x <= z) && !(y <= z) ? 1.0 : 0.0};
    cross3(u, e, w);
    const double n = rsqrt(dot3(w, w));
    for(int r = 0; r < 3; ++r)
        w[r] *= n;
}

// F = U diag(sg) V^T by one-sided Jacobi: the columns of F V made orthogonal
// (V a product of rotations), sg_2 the smallest in magnitude and signed so
// that U is a rotation too
__device__ inline void rotation_svd(const double F[9], double u[3][3], double v[3][3], double sg[3])
{
    double a[3][3];
    for(int i = 0; i < 3; ++i)
        for(int r = 0; r < 3; ++r)
        {
            a[i][r] = F[3 * i + r];
            v[i][r] = i == r ? 1.0 : 0.0;
        }
    for(int sweep = 0; sweep < 12; ++sweep)
    {
        bool any = rotate_columns<0, 1>(a, v);
        any |= rotate_columns<0, 2>(a, v);
        any |= rotate_columns<1, 2>(a, v);
        if(!any)
            break;
    }
    // the shortest column last (a cyclic shift keeps det V = 1)
    double       n0 = dot3(a[0], a[0]), n1 = dot3(a[1], a[1]);
    const double n2 = dot3(a[2], a[2]);
    const bool   s0 = n0 <= n1 && n0 < n2;         // shift left: (1, 2, 0)
    const bool   s1 = !s0 && n1 < n0 && n1 < n2;  // shift right: (2, 0, 1)
    for(int r = 0; r < 3; ++r)
    {
        const double x0 = a[0][r], x1 = a[1][r], x2 = a[2][r], y0 = v[0][r], y1 = v[1][r], y2 = v[2][r];
        a[0][r] = s0 ? x1 : (s1 ? x2 : x0);
        a[1][r] = s0 ? x2 : (s1 ? x0 : x1);
        a[2][r] = s0 ? x0 : (s1 ? x1 : x2);
        v[0][r] = s0 ? y1 : (s1 ? y2 : y0);
        v[1][r] = s0 ? y2 : (s1 ? y0 : y1);
        v[2][r] = s0 ? y0 : (s1 ? y1 : y2);
    }
    const double t0 = n0, t1 = n1;
    n0 = s0 ? t1 : (s1 ? n2 : t0);
    n1 = s0 ? n2 : (s1 ? t0 : t1);
    if(n0 > 0.0)
    {
        const double i0 = rsqrt(n0);
        for(int r = 0; r < 3; ++r)
            u[0][r] = a[0][r] * i0;
    }
    else if(n1 > 0.0)
    {
        const double i1 = rsqrt(n1);
        double       w[3];
        for(int r = 0; r < 3; ++r)
            w[r] = a[1][r] * i1;
        any_orthogonal(w, u[0]);
    }
    else
        u[0][0] = 1.0, u[0][1] = 0.0, u[0][2] = 0.0;
    const double d  = dot3(a[1], u[0]);
    double       w1[3] = {a[1][0] - d * u[0][0], a[1][1] - d * u[0][1], a[1][2] - d * u[0][2]};
    const double nw = dot3(w1, w1);
    if(nw > 1e-30 * n0 && nw > 0.0)
    {
        const double iw = rsqrt(nw);
        for(int r = 0; r < 3; ++r)
            u[1][r] = w1[r] * iw;
    }
    else  // rank one: any direction across u_0
        any_orthogonal(u[0], u[1]);
    cross3(u[0], u[1], u[2]);
    for(int i = 0; i < 3; ++i)
        sg[i] = dot3(a[i], u[i]);
}

// m = Q max(w, 0) Q^T of a symmetric 3x3 matrix; returned as it is when it is
// safely positive definite (leading minors well above rounding)
__device__ inline void clamp3(double m[3][3])
{
    const double d2 = m[0][0] * m[1][1] - m[0][1] * m[0][1];
    const double d3 = m[2][2] * d2 - m[0][2] * (m[0][2] * m[1][1] - m[0][1] * m[1][2])
                      + m[1][2] * (m[0][2] * m[0][1] - m[0][0] * m[1][2]);
    const double a0 = m[0][0], a1 = m[1][1], a2 = m[2][2];
    if(a0 > 0.0 && a1 > 0.0 && a2 > 0.0 && d2 > 1e-8 * a0 * a1 && d3 > 1e-8 * a0 * a1 * a2)
        return;
    double v[3][3] = {{1.0, 0.0, 0.0}, {0.0, 1.0, 0.0}, {0.0, 0.0, 1.0}};  // v[i]: eigenvector i
    for(int sweep = 0; sweep < 20; ++sweep)
    {
        const double off = m[0][1] * m[0][1] + m[0][2] * m[0][2] + m[1][2] * m[1][2];
        const double dia = m[0][0] * m[0][0] + m[1][1] * m[1][1] + m[2][2] * m[2][2];
        if(!(off > 1e-32 * (dia + 1e-300)))
            break;
#pragma unroll
        for(int k = 0; k < 3; ++k)
        {
            const int    p = k == 2 ? 1 : 0, q = k == 0 ? 1 : 2;
            const double apq = m[p][q];
            if(fabs(apq) < 1e-300)
                continue;
            const double z = (m[q][q] - m[p][p]) / (2.0 * apq);
            const double t = (z >= 0.0 ? 1.0 : -1.0) / (fabs(z) + sqrt(z * z + 1.0));
            const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
            const int    o = 3 - p - q;
            m[p][p] -= t * apq;
            m[q][q] += t * apq;
            m[p][q] = m[q][p] = 0.0;
            const double mop = m[o][p], moq = m[o][q];
            m[o][p] = m[p][o] = c * mop - s * moq;
            m[o][q] = m[q][o] = s * mop + c * moq;
            for(int r = 0; r < 3; ++r)
            {
                const double vp = v[p][r], vq = v[q][r];
                v[p][r] = c * vp - s * vq;
                v[q][r] = s * vp + c * vq;
            }
        }
    }
    const double w[3] = {m[0][0] < 0.0 ? 0.0 : m[0][0], m[1][1] < 0.0 ? 0.0 : m[1][1], m[2][2] < 0.0 ? 0.0 : m[2][2]};
    for(int a = 0; a < 3; ++a)
        for(int c = a; c < 3; ++c)
            m[a][c] = m[c][a] = v[0][a] * w[0] * v[0][c] + v[1][a] * w[1] * v[1][c] + v[2][a] * w[2] * v[2][c];
}

// P = dPsi/dF and the projected Hessian's parts, all times `scale`
__device__ inline void derivatives(const double F[9], double mu, double lambda, double scale, double P[9],
                                            Projected& h)
{
    double g[9];
    cross3(F + 3, F + 6, g);
    cross3(F + 6, F, g + 3);
    cross3(F, F + 3, g + 6);
    const double J = dot3(F, g);
    const double s = lambda * (J - 1.0) - mu;
    for(int i = 0; i < 9; ++i)
        P[i] = scale * (mu * F[i] + s * g[i]);
    double sg[3];
    rotation_svd(F, h.u, h.v, sg);
    const double gs[3] = {sg[1] * sg[2], sg[2] * sg[0], sg[0] * sg[1]};
    for(int a = 0; a < 3; ++a)
    {
        const double sy = mu - s * sg[a], an = mu + s * sg[a];
        const double cs = sy < 0.0 ? 0.0 : sy, ca = an < 0.0 ? 0.0 : an;
        h.p[a] = 0.5 * scale * (cs + ca);
        h.q[a] = 0.5 * scale * (cs - ca);
        for(int c = 0; c < 3; ++c)
            h.m[a][c] = lambda * gs[a] * gs[c] + (a == c ? mu : s * sg[3 - a - c]);
    }
    clamp3(h.m);
    for(int a = 0; a < 3; ++a)
        for(int c = 0; c < 3; ++c)
            h.m[a][c] *= scale;
}

// the 3x3 Hessian block (row-major) of two vertices whose shape gradients are
// gq and gr in the V frame (V^T g): B[a][c] = sum gq_b gr_d H[(a,b),(c,d)] in
// the U frame, rotated back
__device__ inline void block(const Projected& h, const double gq[3], const double gr[3], double out[9])
{
    double B[3][3];
    for(int a = 0; a < 3; ++a)
        for(int c = 0; c < 3; ++c)
        {
            if(a == c)
            {
                const int b = (a + 1) % 3, d = (a + 2) % 3;
                B[a][a] = gq[a] * gr[a] * h.m[a][a] + gq[b] * gr[b] * h.p[d] + gq[d] * gr[d] * h.p[b];
            }
            else
                B[a][c] = gq[a] * gr[c] * h.m[a][c] + gq[c] * gr[a] * h.q[3 - a - c];
        }
    for(int i = 0; i < 3; ++i)
    {
        double w[3];
        for(int c = 0; c < 3; ++c)
            w[c] = h.u[0][i] * B[0][c] + h.u[1][i] * B[1][c] + h.u[2][i] * B[2][c];
        for(int k = 0; k < 3; ++k)
            out[3 * i + k] = w[0] * h.u[0][k] + w[1] * h.u[1][k] + w[2] * h.u[2][k];
    }
}
}  // namespace snh
}  // namespace b2s
