// Elastic and Drucker-Prager updates without an SVD, for moderate strains.
//
// The fixed-corotated stress 2 mu (F - R) F^T + lambda (J - 1) J I
// (shaders/slosh/models/linear_elasticity.slang:69-82) and the return mapping
// (shaders/slosh/models/drucker_prager.slang:144-200) are isotropic functions
// of the left stretch b = F F^T: with F = U S V^T, (F - R) F^T = b - sqrt(b),
// the principal log strains are those of log(b) / 2, and the projected F is
// U S' S^-1 U^T F.  So neither U nor V is needed, only b - sqrt(b), log(b)
// and exponentials of its deviator:
//
//   E = b - I = H + H^T + H H^T,  H = F - I      (no cancellation near F = I)
//   b = (1 + m) (I + X),  m = tr(E) / 3,  X traceless
//
// and a function f(X) = X P(X) of a traceless 3 x 3 matrix is
// c0 I + c1 X + c2 X^2 because X^3 = p X + q I (p = tr(X^2) / 2, q = det X,
// Cayley-Hamilton): Horner's rule on the coefficients is two FMAs a term.
// The polynomials were fitted here (Chebyshev interpolation) to sqrt(1 + x),
// log(1 + x) and exp(x) over the range below, to 2e-8 relative.
//
// Range: |X|_F <= 1/2 (principal stretches within a factor of about 1.5),
// det F > 0.  Everything else -- larger strains, inverted or non-finite F,
// and nearly isotropic stretch away from a rotation, where Drucker-Prager's
// exact zero-deviator test is discontinuous -- takes the SVD (models.cuh),
// whose FP64 fallback decides those cases.
//
// Why: the Jacobi SVD is a serial chain whose length depends on the strain
// (one to four sweeps, lanes of a warp waiting for the longest) and keeps F,
// V and F V alive at once; this form has no loop and fewer live values.
// Measured: G2P of the 4.74 M-particle sand column once it moves 308 -> 251
// us (its registers 128 -> 117, no more CTAs an SM: builds at 10 and 12 CTAs
// of 64 spill and take 281 and 352 us, 7 the same time, 6 277), of the
// elastic drop 49 -> 38 us.  Its error at small strain is that of E, not that
// of singular values near 1: after 100 substeps of 68,921 sand particles F is
// 3.5e-8 from 64-bit arithmetic (8.1e-7 with the SVD) and C 2.9e-6 (4.7e-5).
#pragma once

#include "common.cuh"

namespace slosh {

template <int N> struct Poly {
    float c[N];
};
// (sqrt(1 + x) - 1) / x and log(1 + x) / x on |x| <= 0.41, (exp(x) - 1) / x
// on |x| <= 0.29
__device__ __forceinline__ constexpr Poly<10> poly_sqrt() {
    return {{5.000000031e-01f, -1.250000154e-01f, 6.249909891e-02f, -3.906070261e-02f, 2.738568367e-02f,
             -2.056624449e-02f, 1.544016435e-02f, -1.232893841e-02f, 1.516100955e-02f, -1.346192366e-02f}};
}
__device__ __forceinline__ constexpr Poly<11> poly_log() {
    return {{9.999999986e-01f, -5.000001894e-01f, 3.333339273e-01f, -2.499778581e-01f, 1.999595576e-01f,
             -1.673850267e-01f, 1.438548302e-01f, -1.156496618e-01f, 1.001902513e-01f, -1.509783273e-01f,
             1.434815208e-01f}};
}
__device__ __forceinline__ constexpr Poly<6> poly_exp() {
    return {{1.000000004e+00f, 5.000000016e-01f, 1.666658759e-01f, 4.166651293e-02f, 8.358397232e-03f,
             1.392543452e-03f}};
}
// atanh(r) / r, sinh(r) / r and (cosh(r) - 1) / r^2 in r^2 (2D: X^2 = r^2 I)
__device__ __forceinline__ constexpr Poly<5> poly_atanh() {
    return {{1.000000007e+00f, 3.333304269e-01f, 2.001826975e-01f, 1.388846817e-01f, 1.453361987e-01f}};
}
__device__ __forceinline__ constexpr Poly<3> poly_sinh() {
    return {{1.000000005e+00f, 1.666657609e-01f, 8.360158145e-03f}};
}
__device__ __forceinline__ constexpr Poly<3> poly_cosh() {
    return {{5.000000006e-01f, 4.166655362e-02f, 1.392239799e-03f}};
}
template <int N> __device__ __forceinline__ float horner(const Poly<N> &P, float x) {
    float r = P.c[N - 1];
#pragma unroll
    for (int k = N - 2; k >= 0; --k) r = fmaf(r, x, P.c[k]);
    return r;
}

// A traceless symmetric matrix X with its square and invariants.
template <int D> struct Traceless;
template <> struct Traceless<3> {
    float x00, x11, x22, x01, x02, x12;
    float s00, s11, s22, s01, s02, s12;  // X^2
    float p, q;
    __device__ __forceinline__ void square() {
        const float a = x01 * x01, b = x02 * x02, c = x12 * x12;
        s00 = fmaf(x00, x00, a + b);
        s11 = fmaf(x11, x11, a + c);
        s22 = fmaf(x22, x22, b + c);
        s01 = fmaf(x02, x12, -(x22 * x01));
        s02 = fmaf(x01, x12, -(x11 * x02));
        s12 = fmaf(x01, x02, -(x00 * x12));
        p = 0.5f * (s00 + s11 + s22);
        q = fmaf(x00, fmaf(x11, x22, -c), fmaf(x01, s01, x02 * s02));
    }
    __device__ __forceinline__ bool zero() const {
        return x00 == 0.f && x11 == 0.f && x22 == 0.f && x01 == 0.f && x02 == 0.f && x12 == 0.f;
    }
    // k0 I + k1 X + k2 X^2
    __device__ __forceinline__ void combine(float k0, float k1, float k2, float (&M)[3][3]) const {
        M[0][0] = fmaf(k2, s00, fmaf(k1, x00, k0));
        M[1][1] = fmaf(k2, s11, fmaf(k1, x11, k0));
        M[2][2] = fmaf(k2, s22, fmaf(k1, x22, k0));
        M[0][1] = M[1][0] = fmaf(k2, s01, k1 * x01);
        M[0][2] = M[2][0] = fmaf(k2, s02, k1 * x02);
        M[1][2] = M[2][1] = fmaf(k2, s12, k1 * x12);
    }
};
template <> struct Traceless<2> {
    float x00, x01;
    float p;
    __device__ __forceinline__ void square() { p = fmaf(x00, x00, x01 * x01); }
    __device__ __forceinline__ bool zero() const { return x00 == 0.f && x01 == 0.f; }
    __device__ __forceinline__ void combine(float k0, float k1, float, float (&M)[2][2]) const {
        M[0][0] = fmaf(k1, x00, k0);
        M[1][1] = fmaf(-k1, x00, k0);
        M[0][1] = M[1][0] = k1 * x01;
    }
};

// Coefficients of X P(X) in (I, X, X^2), X^3 = p X + q I.
template <int N>
__device__ __forceinline__ void matrix_horner(const Poly<N> &P, float p, float q, float &c0, float &c1, float &c2) {
    float u0 = P.c[N - 1], u1 = 0.f, u2 = 0.f;
#pragma unroll
    for (int k = N - 2; k >= 0; --k) {
        const float v0 = fmaf(u2, q, P.c[k]), v1 = fmaf(u2, p, u0);
        u2 = u1;
        u0 = v0;
        u1 = v1;
    }
    c0 = u2 * q;
    c1 = fmaf(u2, p, u0);
    c2 = u1;
}

// exp(a X) - I = c0 I + c1 X + c2 X^2 for |a| <= 1.
template <int D>
__device__ __forceinline__ void exp_minus_one(const Traceless<D> &X, float a, float &c0, float &c1, float &c2) {
    const float a2 = a * a;
    if constexpr (D == 3) {
        matrix_horner(poly_exp(), a2 * X.p, (a2 * a) * X.q, c0, c1, c2);
        c1 *= a;
        c2 *= a2;
    } else {
        const float y = a2 * X.p;
        c0 = y * horner(poly_cosh(), y);
        c1 = a * horner(poly_sinh(), y);
        c2 = 0.f;
    }
}

// b = F F^T as (1 + m) (I + X), and det b - 1; false outside the range
// described above.
template <int D> struct Stretch {
    float m, detm1;
    Traceless<D> X;
    __device__ __forceinline__ bool of(const float (&F)[D][D]) {
        float H[D][D];
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int k = 0; k < D; ++k) H[i][k] = F[i][k] - (i == k ? 1.f : 0.f);
        auto e = [&](int i, int j) {
            float acc = H[i][j] + H[j][i];
#pragma unroll
            for (int k = 0; k < D; ++k) acc = fmaf(H[i][k], H[j][k], acc);
            return acc;
        };
        const float e00 = e(0, 0), e11 = e(1, 1), e01 = e(0, 1);
        float limit, dp;
        if constexpr (D == 3) {
            const float e22 = e(2, 2), e02 = e(0, 2), e12 = e(1, 2);
            m = (e00 + e11 + e22) * (1.f / 3.f);
            const float r = __fdividef(1.f, 1.f + m), r3 = r * (1.f / 3.f);
            // differences, so that an isotropic E gives X = 0 exactly
            X.x00 = ((e00 - e11) + (e00 - e22)) * r3;
            X.x11 = ((e11 - e00) + (e11 - e22)) * r3;
            X.x22 = -(X.x00 + X.x11);
            X.x01 = e01 * r;
            X.x02 = e02 * r;
            X.x12 = e12 * r;
            X.square();
            dp = X.q - X.p;  // det(I + X) - 1
            detm1 = m * fmaf(m, m + 3.f, 3.f);
            limit = 0.125f;
        } else {
            m = 0.5f * (e00 + e11);
            const float r = __fdividef(1.f, 1.f + m);
            X.x00 = 0.5f * (e00 - e11) * r;
            X.x01 = e01 * r;
            X.square();
            dp = -X.p;
            detm1 = m * (m + 2.f);
            limit = 0.125f;
        }
        detm1 = fmaf(detm1, dp, detm1 + dp);
        const bool isotropic = X.p <= 1.5e-10f && fabsf(m) > 2e-5f;
        return X.p <= limit && m > -0.6f && m < 4.f && !isotropic;
    }
};

// tau = 2 mu (b - sqrt(b)) + lambda (J - 1) J I.
template <int D>
__device__ __forceinline__ void stretch_corotated(const Stretch<D> &b, float lambda, float mu, float (&tau)[D][D]) {
    const float J = sqrtf(1.f + b.detm1), jm1 = __fdividef(b.detm1, 1.f + J);
    const float iso = lambda * jm1 * J, mu2 = 2.f * mu;
    if constexpr (D == 3) {
        const float sg = sqrtf(1.f + b.m);  // sqrt(b) = sg sqrt(I + X)
        float c0, c1, c2;
        matrix_horner(poly_sqrt(), b.X.p, b.X.q, c0, c1, c2);
        const float k0 = fmaf(b.m, __fdividef(sg, 1.f + sg), -(sg * c0));
        const float k1 = fmaf(-sg, c1, 1.f + b.m), k2 = -sg * c2;
        b.X.combine(fmaf(mu2, k0, iso), mu2 * k1, mu2 * k2, tau);
    } else {
        // closed form: sqrt(b) = (b + J I) / t, t^2 = tr b + 2 J
        const float t2 = fmaf(2.f, b.m, 2.f + 2.f * J), t = sqrtf(t2), it = __fdividef(1.f, t);
        const float det_e = fmaf(b.m, b.m, -((1.f + b.m) * (1.f + b.m) * b.X.p));  // det(b - I)
        const float ke = 1.f - it, k0 = -det_e * __fdividef(it, t + 1.f + J);
        // E = m I + (1 + m) X
        b.X.combine(fmaf(mu2, fmaf(ke, b.m, k0), iso), mu2 * (ke * (1.f + b.m)), 0.f, tau);
    }
}

// Drucker-Prager projection (as drucker_prager in models.cuh, on log b / 2)
// and the stress of the projected F: fixed-corotated (NH = false, lambda and
// mu of the elastic model) or Neo-Hookean.  False (nothing written) when the
// projection leaves the exponentials' range.
template <int D, bool NH>
__device__ __forceinline__ bool stretch_sand(const Stretch<D> &b, const float *plastic, float lambda, float mu,
                                             float *st, float (&F)[D][D], float (&tau)[D][D]) {
    constexpr float d = (float)D, inv_d = 1.f / (float)D;
    // log sqrt(b) = tr_l / d I + L, L traceless
    const float tr_l = 0.5f * log1pf(b.detm1);
    Traceless<D> L;
    if constexpr (D == 3) {
        float c0, c1, c2;
        matrix_horner(poly_log(), b.X.p, b.X.q, c0, c1, c2);
        c1 *= 0.5f;
        c2 *= 0.5f;
        const float t = -(2.f / 3.f) * b.X.p;  // minus tr(X^2) / 3
        L.x00 = fmaf(c2, b.X.s00 + t, c1 * b.X.x00);
        L.x11 = fmaf(c2, b.X.s11 + t, c1 * b.X.x11);
        L.x22 = -(L.x00 + L.x11);
        L.x01 = fmaf(c2, b.X.s01, c1 * b.X.x01);
        L.x02 = fmaf(c2, b.X.s02, c1 * b.X.x02);
        L.x12 = fmaf(c2, b.X.s12, c1 * b.X.x12);
    } else {
        const float c1 = 0.5f * horner(poly_atanh(), b.X.p);
        L.x00 = c1 * b.X.x00;
        L.x01 = c1 * b.X.x01;
    }
    L.square();
    const float h0 = plastic[0], h1 = plastic[1], h2 = plastic[2], h3 = plastic[3], lam_p = plastic[4], mu_p = plastic[5];
    const float q = st[1], vol = st[2], tr = tr_l + vol;
    // The friction angle and the cone slope only place the yield surface:
    // hardware approximations (a few ulp) are used for them.
    const float angle = h0 + (h1 * q - h3) * __expf(-h2 * q);
    const float s_angle = __sinf(angle);
    const float alpha = __fdividef(sqrtf(2.0f / 3.0f) * (2.0f * s_angle), 3.0f - s_angle);
    const bool tip = tr > 0.f || L.zero();
    const float devn = sqrtf(2.f * L.p);
    const float gamma = devn + __fdividef(d * lam_p + 2.0f * mu_p, 2.0f * mu_p) * tr * alpha;
    const bool shear = !tip && gamma > 0.f;
    // projected log strain: a L + t I; F' = exp(r) exp(-g L) F
    const float g = tip ? 1.f : (shear ? __fdividef(gamma, devn) : 0.f);
    if (!(g >= 0.f && g <= 1.001f)) return false;  // gamma <= |dev|, up to the rounding of the quotient
    const float a = 1.f - g;
    const float t = tip ? 0.f : (shear ? tr : tr_l) * inv_d;
    if (tip || shear) {
        const float r = tip ? -tr_l * inv_d : vol * inv_d;
        const float em1 = expm1f(r), er = 1.f + em1;
        float c0, c1, c2, W[D][D];
        exp_minus_one<D>(L, -g, c0, c1, c2);
        L.combine(fmaf(er, c0, em1), er * c1, er * c2, W);
        float Fn[D][D];
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int j = 0; j < D; ++j) {
                float acc = F[i][j];
#pragma unroll
                for (int k = 0; k < D; ++k) acc = fmaf(W[i][k], F[k][j], acc);
                Fn[i][j] = acc;
            }
#pragma unroll
        for (int i = 0; i < D; ++i)
#pragma unroll
            for (int j = 0; j < D; ++j) F[i][j] = Fn[i][j];
        // plastic determinant, hardening and the log volume gain: the
        // projection keeps tr (shear) or drops it (tip)
        const float dl = tip ? tr_l : -vol;
        st[0] = st[0] * (1.f + (tip ? expm1f(dl) : __fdividef(-em1 * (d == 3.f ? fmaf(em1, em1 + 3.f, 3.f) : em1 + 2.f),
                                                              d == 3.f ? er * er * er : er * er)));
        st[1] = q + (tip ? sqrtf(fmaf(tr * tr, inv_d, 2.f * L.p)) : gamma);
        st[2] = tip ? vol + tr_l : 0.f;
    }
    const float em1 = expm1f(t), et = 1.f + em1;  // exp(t) of the isotropic part
    float a0, a1, a2;
    exp_minus_one<D>(L, a, a0, a1, a2);  // exp(a L) - I
    // exp(2 a L) - I = (exp(a L) - I)^2 + 2 (exp(a L) - I)
    float b0, b1, b2;
    if constexpr (D == 3) {
        const float x2 = a2 * a2, x12 = 2.f * a1 * a2;
        b0 = fmaf(a0, a0 + 2.f, x12 * L.q);
        b1 = fmaf(2.f * a1, a0 + 1.f, fmaf(x12, L.p, x2 * L.q));
        b2 = fmaf(a1, a1, fmaf(2.f * a2, a0 + 1.f, x2 * L.p));
    } else {
        b0 = fmaf(a0, a0 + 2.f, a1 * a1 * L.p);
        b1 = 2.f * a1 * (a0 + 1.f);
        b2 = 0.f;
    }
    const float e2 = et * et;
    if constexpr (NH) {
        // mu (b' - I) + lambda ln J' I,  b' = exp(2 t) exp(2 a L)
        const float k0 = fmaf(e2, b0, em1 * (2.f + em1));
        L.combine(fmaf(mu, k0, lambda * t * d), mu * e2 * b1, mu * e2 * b2, tau);
    } else {
        // 2 mu (b' - sqrt(b')) + lambda (J' - 1) J' I
        const float jm1 = D == 3 ? em1 * fmaf(em1, em1 + 3.f, 3.f) : em1 * (em1 + 2.f);
        const float iso = lambda * jm1 * (1.f + jm1), mu2 = 2.f * mu;
        L.combine(fmaf(mu2, fmaf(e2, b0, et * (em1 - a0)), iso), mu2 * fmaf(e2, b1, -et * a1),
                  mu2 * fmaf(e2, b2, -et * a2), tau);
    }
    return true;
}

}  // namespace slosh
