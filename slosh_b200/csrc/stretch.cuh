// Fixed-corotated stress without an SVD, for moderate strains.
//
// The stress 2 mu (F - R) F^T + lambda (J - 1) J I
// (shaders/slosh/models/linear_elasticity.slang:69-82) is an isotropic
// function of the left stretch b = F F^T: with F = U S V^T, (F - R) F^T =
// b - sqrt(b).  So neither U nor V is needed, only the square root:
//
//   E = b - I = H + H^T + H H^T,  H = F - I      (no cancellation near F = I)
//   b = (1 + m) (I + X),  m = tr(E) / 3,  X traceless
//
// and a function f(X) = X P(X) of a traceless 3 x 3 matrix is
// c0 I + c1 X + c2 X^2 because X^3 = p X + q I (p = tr(X^2) / 2, q = det X,
// Cayley-Hamilton): Horner's rule on the coefficients is two FMAs a term.
// The polynomial was fitted here (Chebyshev interpolation) to sqrt(1 + x)
// over the range below, to 2e-8 relative.  In 2D the root is closed form.
//
// Range: |X|_F <= 1/2 (principal stretches within a factor of about 1.5),
// det F > 0.  Everything else -- larger strains, inverted or non-finite F,
// and nearly isotropic stretch away from a rotation, where the SVD counts and
// takes its FP64 fallback -- takes the SVD (models.cuh).
//
// Why: the Jacobi SVD is a serial chain whose length depends on the strain
// (one to four sweeps, lanes of a warp waiting for the longest) and keeps F,
// V and F V alive at once; this form has no loop and fewer live values.
// Measured: G2P of the 524,288-particle elastic drop 49 -> 38 us, its error
// against 64-bit arithmetic that of E, not that of singular values near 1.
// Sand keeps the SVD (models.cuh says why).
#pragma once

#include "common.cuh"

namespace slosh {

template <int N> struct Poly {
    float c[N];
};
// (sqrt(1 + x) - 1) / x on |x| <= 0.41
__device__ __forceinline__ constexpr Poly<10> poly_sqrt() {
    return {{5.000000031e-01f, -1.250000154e-01f, 6.249909891e-02f, -3.906070261e-02f, 2.738568367e-02f,
             -2.056624449e-02f, 1.544016435e-02f, -1.232893841e-02f, 1.516100955e-02f, -1.346192366e-02f}};
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
        float dp;
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
        } else {
            m = 0.5f * (e00 + e11);
            const float r = __fdividef(1.f, 1.f + m);
            X.x00 = 0.5f * (e00 - e11) * r;
            X.x01 = e01 * r;
            X.square();
            dp = -X.p;
            detm1 = m * (m + 2.f);
        }
        detm1 = fmaf(detm1, dp, detm1 + dp);
        const bool isotropic = X.p <= 1.5e-10f && fabsf(m) > 2e-5f;
        return X.p <= 0.125f && m > -0.6f && m < 4.f && !isotropic;
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

}  // namespace slosh
