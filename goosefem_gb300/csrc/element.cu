// Element quadrature kernels: Quadrature set-up (shape functions, compute_dN) and the
// element-by-element operators of GooseFEM's QuadratureBaseCartesian, for Quad4 (nne=4, ndim=2)
// and Hex8 (nne=8, ndim=3). One thread per (element, integration point) for point-wise
// operators, one thread per element for the integrals that sum over the integration points, so
// every output entry is summed in the reference's order.
#include "common.cuh"
#include "fixdot.cuh"

#include <climits>

namespace gfgpu {

// ---------------------------------------------------------------- loads

template <int N>
__device__ __forceinline__ void load(const double* __restrict__ p, double (&o)[N])
{
    if constexpr (N % 2 == 0) {
        const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
        for (int k = 0; k < N / 2; ++k) {
            double2 v = __ldg(q + k);
            o[2 * k] = v.x;
            o[2 * k + 1] = v.y;
        }
    }
    else {
#pragma unroll
        for (int k = 0; k < N; ++k) o[k] = __ldg(p + k);
    }
}

template <int N>
__device__ __forceinline__ void store(double* __restrict__ p, const double (&o)[N])
{
#pragma unroll
    for (int k = 0; k < N; ++k) p[k] = o[k];
}

// ---------------------------------------------------------------- shape functions

// ElementQuad4.h:277-300 (N and dN/dxi), evaluated with the reference's operation order.
__device__ __forceinline__ void quad4_shape(double x0, double x1, double* N, double* dn)
{
    double a0 = __dsub_rn(1.0, x0), b0 = __dadd_rn(1.0, x0);
    double a1 = __dsub_rn(1.0, x1), b1 = __dadd_rn(1.0, x1);
    if (N) {
        N[0] = __dmul_rn(__dmul_rn(0.25, a0), a1);
        N[1] = __dmul_rn(__dmul_rn(0.25, b0), a1);
        N[2] = __dmul_rn(__dmul_rn(0.25, b0), b1);
        N[3] = __dmul_rn(__dmul_rn(0.25, a0), b1);
    }
    dn[0 * 2 + 0] = __dmul_rn(-0.25, a1);
    dn[1 * 2 + 0] = __dmul_rn(+0.25, a1);
    dn[2 * 2 + 0] = __dmul_rn(+0.25, b1);
    dn[3 * 2 + 0] = __dmul_rn(-0.25, b1);
    dn[0 * 2 + 1] = __dmul_rn(-0.25, a0);
    dn[1 * 2 + 1] = __dmul_rn(-0.25, b0);
    dn[2 * 2 + 1] = __dmul_rn(+0.25, b0);
    dn[3 * 2 + 1] = __dmul_rn(+0.25, a0);
}

// ElementHex8.h:255-295.
__device__ __forceinline__ void hex8_shape(double x0, double x1, double x2, double* N, double* dn)
{
    const int sx[8] = {-1, +1, +1, -1, -1, +1, +1, -1};
    const int sy[8] = {-1, -1, +1, +1, -1, -1, +1, +1};
    const int sz[8] = {-1, -1, -1, -1, +1, +1, +1, +1};
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        double fa = sx[m] < 0 ? __dsub_rn(1.0, x0) : __dadd_rn(1.0, x0);
        double fb = sy[m] < 0 ? __dsub_rn(1.0, x1) : __dadd_rn(1.0, x1);
        double fc = sz[m] < 0 ? __dsub_rn(1.0, x2) : __dadd_rn(1.0, x2);
        if (N) N[m] = __dmul_rn(__dmul_rn(__dmul_rn(0.125, fa), fb), fc);
        dn[m * 3 + 0] = __dmul_rn(__dmul_rn(sx[m] < 0 ? -0.125 : 0.125, fb), fc);
        dn[m * 3 + 1] = __dmul_rn(__dmul_rn(sy[m] < 0 ? -0.125 : 0.125, fa), fc);
        dn[m * 3 + 2] = __dmul_rn(__dmul_rn(sz[m] < 0 ? -0.125 : 0.125, fa), fb);
    }
}

__global__ void k_shape(const double* xi, int nip, int nd, double* N, double* dNxi)
{
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= nip) return;
    if (nd == 2) {
        double n[4], d[8];
        quad4_shape(xi[q * 2], xi[q * 2 + 1], n, d);
        if (N)
            for (int k = 0; k < 4; ++k) N[q * 4 + k] = n[k];
        if (dNxi)
            for (int k = 0; k < 8; ++k) dNxi[q * 8 + k] = d[k];
    }
    else {
        double n[8], d[24];
        hex8_shape(xi[q * 3], xi[q * 3 + 1], xi[q * 3 + 2], n, d);
        if (N)
            for (int k = 0; k < 8; ++k) N[q * 8 + k] = n[k];
        if (dNxi)
            for (int k = 0; k < 24; ++k) dNxi[q * 24 + k] = d[k];
    }
}

// ElementQuad4.h:493-532 + detail.h:26-36. Strict arithmetic: dNx and vol are bit-exact.
// QuadraturePlanar (ElementQuad4Planar.h:280-318) is the same with vol = w * det(J) * thick; for
// plain Quad4 thick = 1 (an exact product, so the bits are unchanged).
__global__ void k_quad4_compute_dN(const double* __restrict__ x, int64_t nelem,
                                   const double* __restrict__ xi, const double* __restrict__ w,
                                   int nip, double thick, double* __restrict__ dNx,
                                   double* __restrict__ vol)
{
    GF_FOR(t, nelem * nip)
    {
        int64_t e = t / nip;
        int q = static_cast<int>(t - e * nip);
        double dn[8];
        quad4_shape(xi[q * 2], xi[q * 2 + 1], nullptr, dn);
        double xe[8];
        load<8>(x + e * 8, xe);
        double J[2][2];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                J[i][j] = __dadd_rn(
                    __dadd_rn(__dadd_rn(__dmul_rn(dn[0 + i], xe[0 + j]), __dmul_rn(dn[2 + i], xe[2 + j])),
                              __dmul_rn(dn[4 + i], xe[4 + j])),
                    __dmul_rn(dn[6 + i], xe[6 + j]));
        double det = __dsub_rn(__dmul_rn(J[0][0], J[1][1]), __dmul_rn(J[0][1], J[1][0]));
        double i00 = __ddiv_rn(J[1][1], det);
        double i01 = __ddiv_rn(__dmul_rn(-1.0, J[0][1]), det);
        double i10 = __ddiv_rn(__dmul_rn(-1.0, J[1][0]), det);
        double i11 = __ddiv_rn(J[0][0], det);
        double o[8];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            o[m * 2 + 0] = __dadd_rn(__dmul_rn(i00, dn[m * 2 + 0]), __dmul_rn(i01, dn[m * 2 + 1]));
            o[m * 2 + 1] = __dadd_rn(__dmul_rn(i10, dn[m * 2 + 0]), __dmul_rn(i11, dn[m * 2 + 1]));
        }
        store<8>(dNx + t * 8, o);
        vol[t] = __dmul_rn(__dmul_rn(w[q], det), thick);
    }
}

// Element.h:1178-1229 (generic, used by Hex8) + detail.h:49-69, restated as written
// (including dNx(m,i) += Jinv(i,j) * dNxi(m,i), Element.h:1220). Strict arithmetic.
__global__ void k_hex8_compute_dN(const double* __restrict__ x, int64_t nelem,
                                  const double* __restrict__ xi, const double* __restrict__ w,
                                  int nip, double* __restrict__ dNx, double* __restrict__ vol)
{
    GF_FOR(t, nelem * nip)
    {
        int64_t e = t / nip;
        int q = static_cast<int>(t - e * nip);
        double dn[24];
        hex8_shape(xi[q * 3], xi[q * 3 + 1], xi[q * 3 + 2], nullptr, dn);
        double xe[24];
        load<24>(x + e * 24, xe);
        double A[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
        for (int m = 0; m < 8; ++m)
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    A[i][j] = __dadd_rn(A[i][j], __dmul_rn(dn[m * 3 + i], xe[m * 3 + j]));
        auto M3 = [](double a, double b, double c) { return __dmul_rn(__dmul_rn(a, b), c); };
        double det = __dsub_rn(
            __dadd_rn(__dadd_rn(M3(A[0][0], A[1][1], A[2][2]), M3(A[0][1], A[1][2], A[2][0])),
                      M3(A[0][2], A[1][0], A[2][1])),
            __dadd_rn(__dadd_rn(M3(A[0][2], A[1][1], A[2][0]), M3(A[0][1], A[1][0], A[2][2])),
                      M3(A[0][0], A[1][2], A[2][1])));
        auto D = [](double a, double b, double c, double d) {
            return __dsub_rn(__dmul_rn(a, b), __dmul_rn(c, d));
        };
        double B[3][3];
        B[0][0] = __ddiv_rn(D(A[1][1], A[2][2], A[1][2], A[2][1]), det);
        B[0][1] = __ddiv_rn(D(A[0][2], A[2][1], A[0][1], A[2][2]), det);
        B[0][2] = __ddiv_rn(D(A[0][1], A[1][2], A[0][2], A[1][1]), det);
        B[1][0] = __ddiv_rn(D(A[1][2], A[2][0], A[1][0], A[2][2]), det);
        B[1][1] = __ddiv_rn(D(A[0][0], A[2][2], A[0][2], A[2][0]), det);
        B[1][2] = __ddiv_rn(D(A[0][2], A[1][0], A[0][0], A[1][2]), det);
        B[2][0] = __ddiv_rn(D(A[1][0], A[2][1], A[1][1], A[2][0]), det);
        B[2][1] = __ddiv_rn(D(A[0][1], A[2][0], A[0][0], A[2][1]), det);
        B[2][2] = __ddiv_rn(D(A[0][0], A[1][1], A[0][1], A[1][0]), det);
        double* o = dNx + t * 24;
#pragma unroll
        for (int m = 0; m < 8; ++m)
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                double acc = 0.0;
#pragma unroll
                for (int j = 0; j < 3; ++j) acc = __dadd_rn(acc, __dmul_rn(B[i][j], dn[m * 3 + i]));
                o[m * 3 + i] = acc;
            }
        vol[t] = __dmul_rn(w[q], det);
    }
}

// ---------------------------------------------------------------- point-wise operators

template <bool S>
__device__ __forceinline__ double dot4(const double* a, int sa, const double* b, int sb)
{
    // ((a0 b0 + a1 b1) + a2 b2) + a3 b3, the reference's left-to-right sum
    double r = mul<S>(a[0], b[0]);
    r = madd<S>(a[sa], b[sb], r);
    r = madd<S>(a[2 * sa], b[2 * sb], r);
    r = madd<S>(a[3 * sa], b[3 * sb], r);
    return r;
}

// mode 0: GradN_vector, 1: GradN_vector_T, 2: SymGradN_vector. TD: tensor dimension of the
// output (TD = 3 with ND = 2: QuadraturePlanar, ElementQuad4Planar.h:130-221, the in-plane block
// of a zero-filled 3x3 tensor).
template <bool S, int NNE, int ND, int MODE, int TD = ND>
__global__ void k_grad(const double* __restrict__ dNx, const double* __restrict__ elemvec,
                       int64_t nelem, int nip, double* __restrict__ qtensor)
{
    GF_FOR(t, nelem * nip)
    {
        int64_t e = t / nip;
        double g[NNE * ND], u[NNE * ND];
        load<NNE * ND>(dNx + t * NNE * ND, g);
        load<NNE * ND>(elemvec + e * NNE * ND, u);
        double o[ND * ND];
        if constexpr (NNE == 4 && ND == 2) {
            // ElementQuad4.h:349-434 (hand-unrolled overrides)
            double g00 = dot4<S>(g + 0, 2, u + 0, 2);
            double g01 = dot4<S>(g + 0, 2, u + 1, 2);
            double g10 = dot4<S>(g + 1, 2, u + 0, 2);
            double g11 = dot4<S>(g + 1, 2, u + 1, 2);
            if constexpr (MODE == 0) {
                o[0] = g00; o[1] = g01; o[2] = g10; o[3] = g11;
            }
            else if constexpr (MODE == 1) {
                o[0] = g00; o[2] = g01; o[1] = g10; o[3] = g11;
            }
            else {
                // 0.5 * (8-term left-to-right sum)
                double s = g01;
                s = madd<S>(g[1], u[0], s);
                s = madd<S>(g[3], u[2], s);
                s = madd<S>(g[5], u[4], s);
                s = madd<S>(g[7], u[6], s);
                s = mul<S>(0.5, s);
                o[0] = g00; o[3] = g11; o[1] = s; o[2] = s;
            }
        }
        else if constexpr (!S) {
            // the gradient once, then its transpose or symmetric part: 72 (78) FP64 instructions,
            // which bound the kernel, where the loops below take 144 products for the latter (1.2 M
            // points: 167 us against 265 us)
            double h[ND * ND];
#pragma unroll
            for (int i = 0; i < ND; ++i)
#pragma unroll
                for (int j = 0; j < ND; ++j) {
                    h[i * ND + j] = g[i] * u[j];
#pragma unroll
                    for (int m = 1; m < NNE; ++m) h[i * ND + j] = fma(g[m * ND + i], u[m * ND + j], h[i * ND + j]);
                }
#pragma unroll
            for (int i = 0; i < ND; ++i)
#pragma unroll
                for (int j = 0; j < ND; ++j) {
                    if constexpr (MODE == 0) o[i * ND + j] = h[i * ND + j];
                    else if constexpr (MODE == 1) o[j * ND + i] = h[i * ND + j];
                    else if (i <= j) o[i * ND + j] = o[j * ND + i] = i == j ? h[i * ND + i] : 0.5 * (h[i * ND + j] + h[j * ND + i]);
                }
        }
        else {
            // Element.h:925-1022 (generic loops from a zero-filled output)
#pragma unroll
            for (int k = 0; k < ND * ND; ++k) o[k] = 0.0;
#pragma unroll
            for (int m = 0; m < NNE; ++m)
#pragma unroll
                for (int i = 0; i < ND; ++i)
#pragma unroll
                    for (int j = 0; j < ND; ++j) {
                        if constexpr (MODE == 0) {
                            o[i * ND + j] = madd<S>(g[m * ND + i], u[m * ND + j], o[i * ND + j]);
                        }
                        else if constexpr (MODE == 1) {
                            o[j * ND + i] = madd<S>(g[m * ND + i], u[m * ND + j], o[j * ND + i]);
                        }
                        else {
                            double h = mul<S>(0.5, g[m * ND + i]);
                            o[i * ND + j] = madd<S>(h, u[m * ND + j], o[i * ND + j]);
                            o[j * ND + i] = madd<S>(h, u[m * ND + j], o[j * ND + i]);
                        }
                    }
        }
        if constexpr (TD == ND) {
            store<ND * ND>(qtensor + t * ND * ND, o);
        }
        else {
            double* out = qtensor + t * TD * TD;
#pragma unroll
            for (int i = 0; i < TD; ++i)
#pragma unroll
                for (int j = 0; j < TD; ++j) out[i * TD + j] = (i < ND && j < ND) ? o[i * ND + j] : 0.0;
        }
    }
}

// InterpQuad_vector: ElementQuad4.h:325-346 (n = 2, unrolled) / Element.h:893-922.
template <bool S>
__global__ void k_interp(const double* __restrict__ N, const double* __restrict__ elemvec,
                         int64_t nelem, int nne, int nip, int n, double* __restrict__ qvector)
{
    GF_FOR(t, nelem * nip)
    {
        int64_t e = t / nip;
        int q = static_cast<int>(t - e * nip);
        const double* Nq = N + q * nne;
        const double* u = elemvec + e * nne * n;
        double* o = qvector + t * n;
        for (int i = 0; i < n; ++i) {
            double acc;
            if (nne == 4 && n == 2) {
                acc = mul<S>(Nq[0], u[i]);
                for (int m = 1; m < 4; ++m) acc = madd<S>(Nq[m], u[m * n + i], acc);
            }
            else {
                acc = 0.0;
                for (int m = 0; m < nne; ++m) acc = madd<S>(Nq[m], u[m * n + i], acc);
            }
            o[i] = acc;
        }
    }
}

// ---------------------------------------------------------------- integrals (thread per element)

// Int_gradN_dot_tensor2_dV: ElementQuad4.h:467-491 / ElementHex8.h:355-383.
// TD = 3 with ND = 2: QuadraturePlanar (ElementQuad4Planar.h:254-277), the in-plane block of
// each 3x3 tensor.
template <bool S, int NNE, int ND, int TD = ND>
__global__ void k_int_grad_tensor2(const double* __restrict__ dNx, const double* __restrict__ vol,
                                   const double* __restrict__ qtensor, int64_t nelem, int nip,
                                   double* __restrict__ elemvec)
{
    GF_FOR(e, nelem)
    {
        double f[NNE * ND];
#pragma unroll
        for (int k = 0; k < NNE * ND; ++k) f[k] = 0.0;
        for (int q = 0; q < nip; ++q) {
            int64_t t = e * nip + q;
            double g[NNE * ND], s[ND * ND];
            load<NNE * ND>(dNx + t * NNE * ND, g);
            if constexpr (ND == 2 && TD == 2) load<4>(qtensor + t * 4, s);
            else if constexpr (ND == 2) {
                s[0] = __ldg(qtensor + t * 9 + 0);
                s[1] = __ldg(qtensor + t * 9 + 1);
                s[2] = __ldg(qtensor + t * 9 + 3);
                s[3] = __ldg(qtensor + t * 9 + 4);
            }
            else {
#pragma unroll
                for (int k = 0; k < 9; ++k) s[k] = __ldg(qtensor + t * 9 + k);
            }
            double v = __ldg(vol + t);
#pragma unroll
            for (int m = 0; m < NNE; ++m)
#pragma unroll
                for (int j = 0; j < ND; ++j) {
                    double acc = mul<S>(g[m * ND + 0], s[0 * ND + j]);
#pragma unroll
                    for (int i = 1; i < ND; ++i) acc = madd<S>(g[m * ND + i], s[i * ND + j], acc);
                    f[m * ND + j] = madd<S>(acc, v, f[m * ND + j]);
                }
        }
        store<NNE * ND>(elemvec + e * NNE * ND, f);
    }
}

// Int_N_vector_dV: Element.h:1025-1056.
template <bool S>
__global__ void k_int_n_vector(const double* __restrict__ N, const double* __restrict__ vol,
                               const double* __restrict__ qvector, int64_t nelem, int nne, int nip,
                               int n, double* __restrict__ elemvec)
{
    GF_FOR(t, nelem * nne * n)
    {
        int64_t e = t / (nne * n);
        int r = static_cast<int>(t - e * nne * n);
        int m = r / n, i = r - m * n;
        double acc = 0.0;
        for (int q = 0; q < nip; ++q)
            acc = madd<S>(mul<S>(N[q * nne + m], qvector[(e * nip + q) * n + i]), vol[e * nip + q],
                          acc);
        elemvec[t] = acc;
    }
}

// Int_N_scalar_NT_dV: ElementQuad4.h:437-464 / ElementHex8.h:324-352. Thread per elemmat entry.
template <bool S>
__global__ void k_int_n_scalar(const double* __restrict__ N, const double* __restrict__ vol,
                               const double* __restrict__ qscalar, int64_t nelem, int nne,
                               int nip, int nd, double* __restrict__ elemmat)
{
    int K = nne * nd;
    GF_FOR(t, nelem * K * K)
    {
        int64_t e = t / (K * K);
        int rc = static_cast<int>(t - e * K * K);
        int r = rc / K, c = rc - r * K;
        double acc = 0.0;
        if (r % nd == c % nd) {
            int m = r / nd, n = c / nd;
            for (int q = 0; q < nip; ++q)
                acc = madd<S>(mul<S>(mul<S>(N[q * nne + m], qscalar[e * nip + q]), N[q * nne + n]),
                              vol[e * nip + q], acc);
        }
        elemmat[t] = acc;
    }
}

// Diagonal of Int_N_scalar_NT_dV only (the lumped mass of MatrixDiagonal::assemble,
// MatrixDiagonal.h:151-167): thread per (e, m), out elemvec (e, m, i) = elemmat(e, m*nd+i, m*nd+i)
// with k_int_n_scalar's operations for that entry (same bits). With offdiag != null the row's
// off-diagonal entries (m, n != m) are summed too and *offdiag is cleared if one exceeds
// DBL_EPSILON in magnitude (Element::isDiagonal, Element.h:122-145); nothing of the full
// [nelem, nne*nd, nne*nd] matrix is stored.
template <bool S>
__global__ void k_int_n_scalar_diag(const double* __restrict__ N, const double* __restrict__ vol,
                                    const double* __restrict__ qscalar, int64_t nelem, int nne,
                                    int nip, int nd, double* __restrict__ out, int* __restrict__ offdiag)
{
    const double eps = 2.220446049250313080847e-16; // DBL_EPSILON
    GF_FOR(t, nelem * nne)
    {
        const int64_t e = t / nne;
        const int m = static_cast<int>(t - e * nne);
        double acc = 0.0;
        for (int q = 0; q < nip; ++q)
            acc = madd<S>(mul<S>(mul<S>(N[q * nne + m], qscalar[e * nip + q]), N[q * nne + m]),
                          vol[e * nip + q], acc);
        for (int i = 0; i < nd; ++i) out[t * nd + i] = acc;
        if (offdiag) {
            for (int n = 0; n < nne; ++n) {
                if (n == m) continue;
                double o = 0.0;
                for (int q = 0; q < nip; ++q)
                    o = madd<S>(mul<S>(mul<S>(N[q * nne + m], qscalar[e * nip + q]), N[q * nne + n]),
                                vol[e * nip + q], o);
                if (fabs(o) > eps) *offdiag = 0;
            }
        }
    }
}

// Int_gradN_dot_tensor4_dot_gradNT_dV: Element.h:1132-1176, strict arithmetic. Thread per elemmat
// entry; the entry (m*nd+j, n*nd+k) accumulates over q, then i, then l as in the reference loop
// nest. td: tensor dimension of C (td = 3 with nd = 2: QuadraturePlanar, the in-plane indices of a
// [3,3,3,3] tensor).
__global__ void k_int_tensor4_strict(const double* __restrict__ dNx, const double* __restrict__ vol,
                                     const double* __restrict__ C, int64_t nelem, int nne, int nip,
                                     int nd, int td, double* __restrict__ elemmat)
{
    int K = nne * nd;
    GF_FOR(t, nelem * K * K)
    {
        int64_t e = t / (K * K);
        int rc = static_cast<int>(t - e * K * K);
        int r = rc / K, c = rc - r * K;
        int m = r / nd, j = r - m * nd, n = c / nd, k = c - n * nd;
        double acc = 0.0;
        for (int q = 0; q < nip; ++q) {
            const double* g = dNx + (e * nip + q) * nne * nd;
            const double* Cq = C + (e * nip + q) * td * td * td * td;
            double v = vol[e * nip + q];
            for (int i = 0; i < nd; ++i)
                for (int l = 0; l < nd; ++l)
                    acc = madd<true>(mul<true>(mul<true>(g[m * nd + i], Cq[((i * td + j) * td + k) * td + l]),
                                               g[n * nd + l]),
                                     v, acc);
        }
        elemmat[t] = acc;
    }
}

// The same, fast arithmetic, in two steps: T[m,j,k,l] = sum_i (v g[m,i]) C[i,j,k,l], then
// K[(m,j),(n,k)] += sum_l T[m,j,k,l] g[n,l]. FP64 instructions bound it (FP64 issues 2 per SM and
// clock): 200 (nd = 2) and 2400 (nd = 3) per integration point against 768 and 15552 of the form
// above, whose three factors are multiplied anew for every (i, l) of every entry. A thread owns the
// row (m, j) and the columns (n, k) of one k, so that its T never leaves registers; the NNE * ND^2
// threads of an element read its tensors, gradients and v * gradients from shared memory, filled
// (and the matrices written back) in address order. EPB elements per block make whole warps
// (16 x 16 and 72 x 4 threads). For rules other than the Gauss ones (k_int_tensor4_fix).
template <int NNE, int ND>
struct Tensor4Block {
    static constexpr int K = NNE * ND, C4 = ND * ND * ND * ND, G = NNE * ND;
    static constexpr int TPE = NNE * ND * ND;        // threads per element
    static constexpr int EPB = ND == 2 ? 16 : 4;     // elements per block
    static constexpr int THREADS = TPE * EPB;
    static constexpr int QC = NNE;                   // integration points staged at a time
    static constexpr int SZ = QC * (C4 + 2 * G) + 2; // per element, + 2: elements on other banks
    static_assert(SZ >= K * K && THREADS % 32 == 0, "shared layout");
};

template <int NNE, int ND, int TD>
__global__ void __launch_bounds__(Tensor4Block<NNE, ND>::THREADS)
k_int_tensor4(const double* __restrict__ dNx, const double* __restrict__ vol,
              const double* __restrict__ C, int64_t nelem, int nip, double* __restrict__ elemmat)
{
    using B = Tensor4Block<NNE, ND>;
    constexpr int K = B::K, C4 = B::C4, G = B::G, QC = B::QC, SZ = B::SZ, T4 = TD * TD * TD * TD;
    __shared__ double sm[B::EPB * SZ];
    const int tid = threadIdx.x;
    const int el = tid / B::TPE, r = tid - el * B::TPE;
    const int m = r / (ND * ND), j = (r / ND) % ND, k = r % ND;
    const int64_t e0 = static_cast<int64_t>(blockIdx.x) * B::EPB;
    const int ne = static_cast<int>(nelem - e0 < B::EPB ? nelem - e0 : B::EPB);
    double* se = sm + el * SZ;
    double acc[NNE];
#pragma unroll
    for (int n = 0; n < NNE; ++n) acc[n] = 0.0;
    for (int q0 = 0; q0 < nip; q0 += QC) {
        const int nq = nip - q0 < QC ? nip - q0 : QC;
        // per element: [QC][C4] tensors, [QC][G] gradients, [QC][G] v * gradients
        for (int i = tid; i < ne * nq * C4; i += B::THREADS) {
            const int x = i / (nq * C4), y = i - x * nq * C4;
            if constexpr (TD == ND) {
                sm[x * SZ + y] = __ldg(C + ((e0 + x) * nip + q0) * T4 + y);
            }
            else {
                // the in-plane entries of [TD]^4 (ND = 2)
                const int q = y / C4, c = y - q * C4;
                const int at = (((c >> 3) * TD + ((c >> 2) & 1)) * TD + ((c >> 1) & 1)) * TD + (c & 1);
                sm[x * SZ + y] = __ldg(C + ((e0 + x) * nip + q0 + q) * T4 + at);
            }
        }
        for (int i = tid; i < ne * nq * G; i += B::THREADS) {
            const int x = i / (nq * G), y = i - x * nq * G, q = y / G;
            const double g = __ldg(dNx + ((e0 + x) * nip + q0) * G + y);
            sm[x * SZ + QC * C4 + y] = g;
            sm[x * SZ + QC * (C4 + G) + y] = __ldg(vol + (e0 + x) * nip + q0 + q) * g;
        }
        __syncthreads();
        if (el < ne) {
            for (int q = 0; q < nq; ++q) {
                const double* c = se + q * C4 + (j * ND + k) * ND;
                const double* g = se + QC * C4 + q * G;
                const double* gv = se + QC * (C4 + G) + q * G + m * ND;
                double t[ND];
#pragma unroll
                for (int l = 0; l < ND; ++l) t[l] = gv[0] * c[l];
#pragma unroll
                for (int i = 1; i < ND; ++i)
#pragma unroll
                    for (int l = 0; l < ND; ++l) t[l] = fma(gv[i], c[i * ND * ND * ND + l], t[l]);
#pragma unroll
                for (int n = 0; n < NNE; ++n)
#pragma unroll
                    for (int l = 0; l < ND; ++l) acc[n] = fma(t[l], g[n * ND + l], acc[n]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int n = 0; n < NNE; ++n) se[(m * ND + j) * K + n * ND + k] = acc[n];
    __syncthreads();
    for (int i = tid; i < ne * K * K; i += B::THREADS) {
        const int x = i / (K * K);
        elemmat[e0 * K * K + i] = sm[x * SZ + i - x * K * K];
    }
}

// The same two contractions on the integer pipes (fixdot.cuh) for rules of NNE points (the Gauss and the
// nodal rule, or any other): FP64 issue bounds the kernel above at 200 and 2400 instructions per
// integration point. The tensors, the gradients and the volume * gradients of an element are brought to
// one exponent each over all its points, so that the entries of its matrix are integer sums until the
// end. A thread (m, j, k) loads the (j, k) block of the tensor of point m and a few gradients, the largest
// exponents meet in shared memory, and the threads leave the limbs of what they loaded there for all,
// with the exponents. What the limbs cut off is judged entry by entry: after the products a thread takes
// the largest exponent of any term v g[m,i] C[i,j,k,l] g[n,l] of each of its entries, and if one lies more
// than kSpread below that of the largest values (points of very different scale, a weak tensor block), or
// a value leaves the range, the thread takes the FP64 form on operands in global memory.
// 9177 Hex8 elements 326 -> 200 us against the FP64 form, 49k Quad4 80 -> 62 us, with a third of its
// error; the integer multiply-add pipe is 59 % busy (half of it the multiply-adds, the rest the
// conversions), 2 blocks per SM (registers; Quad4 3). Looking at point m first saves forming the exponents
// of all terms beside the products (a call on the Hex8 mesh 208 us, 237 with them). The nodal rule, whose
// gradients hold zeros, looks at all points: 225 us.
template <int NNE, int ND>
struct Tensor4Fix {
    static constexpr int K = NNE * ND, C4 = ND * ND * ND * ND, G = NNE * ND, JK = ND * ND;
    static constexpr int TPE = NNE * ND * ND;
    static constexpr int EPB = ND == 2 ? 16 : 4;
    static constexpr int THREADS = TPE * EPB;
    static constexpr int NE = 3;           // exponents per element: tensors, gradients, v * gradients
    // An entry's error is at most NNE * ND * (ND + 4) * 2^-82 (2^-74.6 for Hex8) of the product of the three
    // scales, its largest term at least 2^-(kSpread + 3): an error below 2^-53 of that term.
    static constexpr int kSpread = 18;
    static constexpr int NG = NNE * G;     // gradients per element
    static constexpr int SL = NNE * (C4 + 2 * G) + 1; // limbs per element (+ 1: elements on other banks)
    // the limbs, or the matrices that take their place, then the exponents
    static constexpr size_t BODY = sizeof(int4) * EPB * SL > sizeof(double) * EPB * K * K ? sizeof(int4) * EPB * SL
                                                                                         : sizeof(double) * EPB * K * K;
    static constexpr size_t SMEM = BODY + sizeof(int) * EPB * NE;
};

// top[n] = max(top[n], exponents of the terms of entry (m, j), (n, k) at point q)
template <int NNE, int ND>
__device__ __forceinline__ void tensor4_top(const int4* lim, int m, int j, int k, int q, int (&top)[NNE])
{
    using B = Tensor4Fix<NNE, ND>;
    const int4* lc = lim + q * B::C4 + (j * ND + k) * ND;
    const int4* lg = lim + NNE * B::C4 + q * B::G;
    const int4* lv = lg + B::NG + m * ND;
#pragma unroll
    for (int l = 0; l < ND; ++l) {
        int w = kFxNone;
#pragma unroll
        for (int i = 0; i < ND; ++i) w = max(w, lv[i].w + lc[i * ND * ND * ND + l].w);
#pragma unroll
        for (int n = 0; n < NNE; ++n) top[n] = max(top[n], w + lg[n * ND + l].w);
    }
}

template <int NNE, int ND, int TD>
__global__ void __launch_bounds__(Tensor4Fix<NNE, ND>::THREADS, ND == 2 ? 3 : 2)
k_int_tensor4_fix(const double* __restrict__ dNx, const double* __restrict__ vol, const double* __restrict__ C,
                  int64_t nelem, double* __restrict__ elemmat)
{
    using B = Tensor4Fix<NNE, ND>;
    constexpr int K = B::K, C4 = B::C4, G = B::G, JK = B::JK, T4 = TD * TD * TD * TD, NE = B::NE, SL = B::SL;
    constexpr int TPE = B::TPE, NG = B::NG, GT = (NG + TPE - 1) / TPE; // gradients per thread
    static_assert(3 * ND * NNE < 128, "ND * NNE products of limbs fit a 64-bit sum");
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x;
    const int el = tid / TPE, r = tid - el * TPE;
    const int m = r / (ND * ND), j = (r / ND) % ND, k = r % ND;
    const int64_t e0 = static_cast<int64_t>(blockIdx.x) * B::EPB;
    const int ne = static_cast<int>(nelem - e0 < B::EPB ? nelem - e0 : B::EPB);
    const bool on = el < ne;
    int4* lim = reinterpret_cast<int4*>(smem) + el * SL;
    double* out = reinterpret_cast<double*>(smem);
    int* ex = reinterpret_cast<int*>(smem + B::BODY) + el * NE;
    if (r < NE) ex[r] = 0;
    // this thread's values: point m's C[i, j, k, l], and gradients r, r + TPE, ... of the element
    const double* Ce = C + (e0 + el) * NNE * T4;
    const double* ge = dNx + (e0 + el) * NG;
    double c[JK], g[GT], gv[GT];
    int xc = 0, xg = 0, xv = 0;
    if (on) {
#pragma unroll
        for (int t = 0; t < JK; ++t) {
            c[t] = __ldg(Ce + m * T4 + (((t / ND) * TD + j) * TD + k) * TD + t % ND);
            xc = max(xc, fx_exponent(c[t]));
        }
#pragma unroll
        for (int t = 0; t < GT; ++t) {
            const int y = r + t * TPE;
            g[t] = gv[t] = 0.0;
            if (y < NG) {
                g[t] = __ldg(ge + y);
                gv[t] = __ldg(vol + (e0 + el) * NNE + y / G) * g[t];
            }
            xg = max(xg, fx_exponent(g[t]));
            xv = max(xv, fx_exponent(gv[t]));
        }
    }
    __syncthreads();
    if (on) {
        atomicMax(ex, xc);
        atomicMax(ex + 1, xg);
        atomicMax(ex + 2, xv);
    }
    __syncthreads();
    int ec = 0, eg = 0, ev = 0;
    bool fix = false;
    if (on) {
        ec = ex[0];
        eg = ex[1];
        ev = ex[2];
        const int sum = ec + eg + ev - 3 * 1022;
        fix = ec > 100 && eg > 100 && ev > 100 && ec < 0x7ff && eg < 0x7ff && ev < 0x7ff && sum > -800 && sum < 900;
        if (fix) {
#pragma unroll
            for (int t = 0; t < JK; ++t) lim[m * C4 + ((t / ND * ND + j) * ND + k) * ND + t % ND] = fx_from_double(c[t], ec);
#pragma unroll
            for (int t = 0; t < GT; ++t) {
                const int y = r + t * TPE;
                if (y < NG) {
                    lim[NNE * C4 + y] = fx_from_double(g[t], eg);
                    lim[NNE * C4 + NG + y] = fx_from_double(gv[t], ev);
                }
            }
        }
    }
    __syncthreads();
    double res[NNE];
    if (fix) {
        FxSum acc[NNE];
#pragma unroll
        for (int n = 0; n < NNE; ++n) fx_zero(acc[n]);
        const int4* lc = lim + (j * ND + k) * ND;
        const int4* lg = lim + NNE * C4;
        const int4* lv = lg + NG + m * ND;
#pragma unroll 1
        for (int q = 0; q < NNE; ++q, lc += C4, lg += G, lv += G) {
            int4 t[ND];
#pragma unroll
            for (int l = 0; l < ND; ++l) {
                FxSum s;
                fx_zero(s);
#pragma unroll
                for (int i = 0; i < ND; ++i) fx_mad(s, lv[i], lc[i * ND * ND * ND + l]);
                t[l] = fx_limbs(s);
            }
#pragma unroll
            for (int n = 0; n < NNE; ++n)
#pragma unroll
                for (int l = 0; l < ND; ++l) fx_mad(acc[n], t[l], lg[n * ND + l]);
        }
        const int scale = ec + ev + eg - 3 * 1022 + 2;
#pragma unroll
        for (int n = 0; n < NNE; ++n) res[n] = fx_to_double(acc[n], scale);
        // the largest exponents of the entries' terms at point m, where they are nearly always enough, else
        // at all points; an entry of zeros alone (below 0) is exact
        int top[NNE], low = INT_MAX;
#pragma unroll
        for (int n = 0; n < NNE; ++n) top[n] = kFxNone;
        tensor4_top<NNE, ND>(lim, m, j, k, m, top);
#pragma unroll
        for (int n = 0; n < NNE; ++n) low = min(low, top[n]);
        const int need = ec + ev + eg - B::kSpread;
        if (low < need) {
#pragma unroll 1
            for (int q = 0; q < NNE; ++q) tensor4_top<NNE, ND>(lim, m, j, k, q, top);
#pragma unroll
            for (int n = 0; n < NNE; ++n) fix = fix && (top[n] < 0 || top[n] >= need);
        }
    }
    if (on && !fix) {
#pragma unroll
        for (int n = 0; n < NNE; ++n) res[n] = 0.0;
#pragma unroll 1
        for (int q = 0; q < NNE; ++q) {
            const double* cq = Ce + q * T4;
            const double* gq = ge + q * G;
            const double v = __ldg(vol + (e0 + el) * NNE + q);
            double t[ND];
#pragma unroll
            for (int l = 0; l < ND; ++l) {
                t[l] = 0.0;
#pragma unroll
                for (int i = 0; i < ND; ++i)
                    t[l] = fma(v * __ldg(gq + m * ND + i), __ldg(cq + ((i * TD + j) * TD + k) * TD + l), t[l]);
            }
#pragma unroll
            for (int n = 0; n < NNE; ++n)
#pragma unroll
                for (int l = 0; l < ND; ++l) res[n] = fma(t[l], __ldg(gq + n * ND + l), res[n]);
        }
    }
    __syncthreads(); // the limbs are read: the matrices take their place
    if (on)
#pragma unroll
        for (int n = 0; n < NNE; ++n) out[el * K * K + (m * ND + j) * K + n * ND + k] = res[n];
    __syncthreads();
    for (int i = tid; i < ne * K * K; i += B::THREADS) elemmat[e0 * K * K + i] = out[i];
}

template <int NNE, int ND, int TD = ND>
static int launch_int_tensor4(const double* dNx, const double* vol, const double* C, int64_t nelem, int nip,
                              double* elemmat, cudaStream_t s)
{
    using B = Tensor4Block<NNE, ND>;
    using X = Tensor4Fix<NNE, ND>;
    if (strict_mode()) {
        k_int_tensor4_strict<<<grid_for(nelem * B::K * B::K), kBlock, 0, s>>>(dNx, vol, C, nelem, NNE, nip, ND, TD,
                                                                             elemmat);
    }
    else if (nip == NNE) {
        // 66 KB of limbs for 4 Hex8 elements
        auto kernel = k_int_tensor4_fix<NNE, ND, TD>;
        GF_TRY(check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(X::SMEM)),
                          "cudaFuncSetAttribute"));
        kernel<<<grid_for(nelem, X::EPB), X::THREADS, X::SMEM, s>>>(dNx, vol, C, nelem, elemmat);
    }
    else {
        k_int_tensor4<NNE, ND, TD><<<grid_for(nelem, B::EPB), B::THREADS, 0, s>>>(dNx, vol, C, nelem, nip, elemmat);
    }
    return GFGPU_OK;
}

// Linear elastic stress (plane strain for nd = 2), strict arithmetic: the oracle's operation order.
__global__ void k_stress_strict(const double* __restrict__ eps, const double* __restrict__ K,
                                const double* __restrict__ G, int64_t nelem, int nip, int nd,
                                double* __restrict__ sig)
{
    GF_FOR(t, nelem * nip)
    {
        int64_t e = t / nip;
        const double* s = eps + t * nd * nd;
        double* o = sig + t * nd * nd;
        double g2 = mul<true>(2.0, G[e]);
        double tr = 0.0;
        for (int i = 0; i < nd; ++i) tr = add<true>(tr, s[i * nd + i]);
        double Kt = mul<true>(K[e], tr);
        double m = __ddiv_rn(tr, 3.0);
        for (int i = 0; i < nd; ++i)
            for (int j = 0; j < nd; ++j)
                o[i * nd + j] = (i == j) ? madd<true>(g2, sub<true>(s[i * nd + j], m), Kt)
                                         : mul<true>(g2, s[i * nd + j]);
    }
}

// The same, fast arithmetic: sigma = lam tr I + 2 G eps with lam = K - 2 G / 3, which needs no
// division (an FP64 division is a dozen instructions at 2 per SM and clock): 57 us for 4.1 M 2-d
// points (4.6 TB/s) against 192 us in the form above; 40 against 96 us for 1.2 M 3-d points. For a
// symmetric strain, as SymGradN gives it, the products below the diagonal are copies of those above;
// the others are formed when a lane of the warp needs one.
template <int ND>
__device__ __forceinline__ void stress_point(double (&s)[ND * ND], double lam, double g2, bool all)
{
    double tr = s[0];
#pragma unroll
    for (int i = 1; i < ND; ++i) tr += s[i * ND + i];
    const double lt = trace_stress(lam, tr);
#pragma unroll
    for (int i = 0; i < ND; ++i) {
        s[i * ND + i] = fma(g2, s[i * ND + i], lt);
#pragma unroll
        for (int j = 0; j < i; ++j) {
            s[j * ND + i] *= g2;
            if (all) s[i * ND + j] = s[j * ND + i];
            else s[i * ND + j] *= g2;
        }
    }
}

template <int ND>
__device__ __forceinline__ bool stress_symmetric(const double (&s)[ND * ND])
{
    bool sym = true;
#pragma unroll
    for (int i = 0; i < ND; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j)
            sym = sym && __double_as_longlong(s[i * ND + j]) == __double_as_longlong(s[j * ND + i]);
    return sym;
}

// A thread per point; its ND^2 values go through shared memory, so that global memory is read and
// written in address order.
template <int ND>
__global__ void __launch_bounds__(kBlock)
k_stress(const double* __restrict__ eps, const double* __restrict__ K, const double* __restrict__ G,
         int64_t npoint, uint32_t nip, double* __restrict__ sig)
{
    constexpr int T = ND * ND;
    __shared__ double sm[kBlock * T];
    const int64_t t0 = static_cast<int64_t>(blockIdx.x) * kBlock, t = t0 + threadIdx.x;
    const int n = static_cast<int>(npoint - t0 < kBlock ? npoint - t0 : kBlock);
    const bool on = static_cast<int>(threadIdx.x) < n;
    double s[T];
    for (int i = threadIdx.x; i < n * T; i += kBlock) sm[i] = __ldg(eps + t0 * T + i);
    __syncthreads();
    if (on) {
#pragma unroll
        for (int k = 0; k < T; ++k) s[k] = sm[threadIdx.x * T + k];
        const uint32_t e = static_cast<uint32_t>(t) / nip;
        const double Ge = __ldg(G + e), lam = fma(-2.0 / 3.0, Ge, __ldg(K + e));
        const bool all = __all_sync(__activemask(), stress_symmetric<ND>(s));
        stress_point<ND>(s, lam, Ge + Ge, all);
#pragma unroll
        for (int k = 0; k < T; ++k) sm[threadIdx.x * T + k] = s[k];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * T; i += kBlock) sig[t0 * T + i] = sm[i];
}

// 2-d tensors as two aligned double2 a point, P points of one element per thread (`groups` of them per
// element): the element's moduli once, and P times the loads in flight. 4.1 M points: one 64 us, two
// 57 us, four 66 us (a quarter of each 128-byte line per load).
template <int P>
__global__ void __launch_bounds__(kBlock)
k_stress_2d(const double2* __restrict__ eps, const double* __restrict__ K, const double* __restrict__ G,
            int64_t n, uint32_t groups, double2* __restrict__ sig)
{
    GF_FOR(t, n)
    {
        double s[P][4];
        bool sym = true;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const double2 x = __ldg(eps + 2 * (P * t + p)), y = __ldg(eps + 2 * (P * t + p) + 1);
            s[p][0] = x.x;
            s[p][1] = x.y;
            s[p][2] = y.x;
            s[p][3] = y.y;
        }
        const uint32_t e = static_cast<uint32_t>(t) / groups;
        const double Ge = __ldg(G + e), lam = fma(-2.0 / 3.0, Ge, __ldg(K + e));
#pragma unroll
        for (int p = 0; p < P; ++p) sym = sym && stress_symmetric<2>(s[p]);
        const bool all = __all_sync(__activemask(), sym);
#pragma unroll
        for (int p = 0; p < P; ++p) {
            stress_point<2>(s[p], lam, Ge + Ge, all);
            sig[2 * (P * t + p)] = make_double2(s[p][0], s[p][1]);
            sig[2 * (P * t + p) + 1] = make_double2(s[p][2], s[p][3]);
        }
    }
}

static bool aligned16(const void* p)
{
    return (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
}

static int check_elem(int nne, int nd)
{
    if ((nne == 4 && nd == 2) || (nne == 8 && nd == 3)) return GFGPU_OK;
    return fail(GFGPU_ERR_UNSUPPORTED, "only Quad4 (nne=4, ndim=2) and Hex8 (nne=8, ndim=3)");
}

} // namespace gfgpu

using namespace gfgpu;

#define DISPATCH_S(...)                                                                         \
    do {                                                                                        \
        if (strict_mode()) {                                                                    \
            constexpr bool kS = true;                                                           \
            __VA_ARGS__;                                                                        \
        }                                                                                       \
        else {                                                                                  \
            constexpr bool kS = false;                                                          \
            __VA_ARGS__;                                                                        \
        }                                                                                       \
    } while (0)

template <int MODE>
static int grad(const double* dNx, const double* elemvec, int64_t nelem, int32_t nne, int32_t nip,
                int32_t nd, double* qtensor, gfgpu_stream_t stream, bool planar = false)
{
    GF_REQUIRE(dNx && elemvec && qtensor && nip > 0, "bad argument");
    GF_TRY(check_elem(nne, nd));
    GF_REQUIRE(!too_big(nelem * nip * 24), "too many elements");
    GF_REQUIRE(aligned16(dNx) && aligned16(elemvec), "dNx and elemvec must be 16-byte aligned");
    if (nelem == 0) return GFGPU_OK;
    const Shape l = spread(nelem * nip);
    if (planar)
        DISPATCH_S(k_grad<kS, 4, 2, MODE, 3><<<l.grid, l.block, 0, S(stream)>>>(dNx, elemvec, nelem, nip, qtensor));
    else if (nd == 2)
        DISPATCH_S(k_grad<kS, 4, 2, MODE><<<l.grid, l.block, 0, S(stream)>>>(dNx, elemvec, nelem, nip, qtensor));
    else
        DISPATCH_S(k_grad<kS, 8, 3, MODE><<<l.grid, l.block, 0, S(stream)>>>(dNx, elemvec, nelem, nip, qtensor));
    return check_launch("grad_n_vector");
}

extern "C" {

static int compute_dN(int nd, const double* x, int64_t nelem, const double* xi, const double* w,
                      int32_t nip, double* N, double* dNxi, double* dNx, double* vol,
                      gfgpu_stream_t stream, double thick = 1.0)
{
    GF_REQUIRE(x && xi && w && dNx && vol && nip > 0 && nelem >= 0, "bad argument");
    GF_REQUIRE(!too_big(nelem * nip * 24), "too many elements");
    GF_REQUIRE(aligned16(x) && aligned16(dNx), "x and dNx must be 16-byte aligned");
    if (N || dNxi) k_shape<<<1, 64, 0, S(stream)>>>(xi, nip, nd, N, dNxi);
    if (nelem > 0) {
        if (nd == 2)
            k_quad4_compute_dN<<<grid_for(nelem * nip), kBlock, 0, S(stream)>>>(x, nelem, xi, w, nip,
                                                                              thick, dNx, vol);
        else
            k_hex8_compute_dN<<<grid_for(nelem * nip), kBlock, 0, S(stream)>>>(x, nelem, xi, w, nip,
                                                                             dNx, vol);
    }
    return check_launch("compute_dN");
}

int gfgpu_quad4_compute_dN(const double* x, int64_t nelem, const double* xi, const double* w,
                           int32_t nip, double* N, double* dNxi, double* dNx, double* vol,
                           gfgpu_stream_t stream)
{
    return compute_dN(2, x, nelem, xi, w, nip, N, dNxi, dNx, vol, stream);
}

int gfgpu_hex8_compute_dN(const double* x, int64_t nelem, const double* xi, const double* w,
                          int32_t nip, double* N, double* dNxi, double* dNx, double* vol,
                          gfgpu_stream_t stream)
{
    return compute_dN(3, x, nelem, xi, w, nip, N, dNxi, dNx, vol, stream);
}

int gfgpu_interp_quad_vector(const double* N, const double* elemvec, int64_t nelem, int32_t nne,
                             int32_t nip, int32_t n, double* qvector, gfgpu_stream_t stream)
{
    GF_REQUIRE(N && elemvec && qvector && nne > 0 && nip > 0 && n > 0, "bad argument");
    GF_REQUIRE(!too_big(nelem * nip * n), "too many elements");
    if (nelem == 0) return GFGPU_OK;
    DISPATCH_S(k_interp<kS><<<grid_for(nelem * nip), kBlock, 0, S(stream)>>>(N, elemvec, nelem, nne,
                                                                             nip, n, qvector));
    return check_launch("interp_quad_vector");
}

int gfgpu_grad_n_vector(const double* dNx, const double* elemvec, int64_t nelem, int32_t nne,
                        int32_t nip, int32_t ndim, double* qtensor, gfgpu_stream_t stream)
{
    return grad<0>(dNx, elemvec, nelem, nne, nip, ndim, qtensor, stream);
}

int gfgpu_grad_n_vector_T(const double* dNx, const double* elemvec, int64_t nelem, int32_t nne,
                          int32_t nip, int32_t ndim, double* qtensor, gfgpu_stream_t stream)
{
    return grad<1>(dNx, elemvec, nelem, nne, nip, ndim, qtensor, stream);
}

int gfgpu_sym_grad_n_vector(const double* dNx, const double* elemvec, int64_t nelem, int32_t nne,
                            int32_t nip, int32_t ndim, double* qtensor, gfgpu_stream_t stream)
{
    return grad<2>(dNx, elemvec, nelem, nne, nip, ndim, qtensor, stream);
}

int gfgpu_int_n_vector_dv(const double* N, const double* vol, const double* qvector,
                          int64_t nelem, int32_t nne, int32_t nip, int32_t n, double* elemvec,
                          gfgpu_stream_t stream)
{
    GF_REQUIRE(N && vol && qvector && elemvec && nne > 0 && nip > 0 && n > 0, "bad argument");
    GF_REQUIRE(!too_big(nelem * nne * n), "too many elements");
    if (nelem == 0) return GFGPU_OK;
    DISPATCH_S(k_int_n_vector<kS><<<grid_for(nelem * nne * n), kBlock, 0, S(stream)>>>(
        N, vol, qvector, nelem, nne, nip, n, elemvec));
    return check_launch("int_n_vector_dv");
}

int gfgpu_int_n_scalar_nt_dv(const double* N, const double* vol, const double* qscalar,
                             int64_t nelem, int32_t nne, int32_t nip, int32_t ndim,
                             double* elemmat, gfgpu_stream_t stream)
{
    GF_REQUIRE(N && vol && qscalar && elemmat && nip > 0, "bad argument");
    GF_TRY(check_elem(nne, ndim));
    int64_t K = nne * ndim;
    GF_REQUIRE(!too_big(nelem * K * K), "too many elements");
    if (nelem == 0) return GFGPU_OK;
    DISPATCH_S(k_int_n_scalar<kS><<<grid_for(nelem * K * K), kBlock, 0, S(stream)>>>(
        N, vol, qscalar, nelem, nne, nip, ndim, elemmat));
    return check_launch("int_n_scalar_nt_dv");
}

int gfgpu_int_n_scalar_nt_dv_diag(const double* N, const double* vol, const double* qscalar,
                                  int64_t nelem, int32_t nne, int32_t nip, int32_t ndim,
                                  double* elemvec, int* is_diag, gfgpu_stream_t stream)
{
    GF_REQUIRE(N && vol && qscalar && elemvec && nip > 0, "bad argument");
    GF_TRY(check_elem(nne, ndim));
    GF_REQUIRE(!too_big(nelem * nne * ndim), "too many elements");
    cudaStream_t s = S(stream);
    int* flag = nullptr;
    if (is_diag) {
        GF_TRY(check_cuda(cudaMallocAsync(reinterpret_cast<void**>(&flag), sizeof(int), s), "cudaMallocAsync"));
        const int one = 1;
        int rc = check_cuda(cudaMemcpyAsync(flag, &one, sizeof(int), cudaMemcpyHostToDevice, s), "cudaMemcpyAsync");
        if (rc != GFGPU_OK) {
            cudaFreeAsync(flag, s);
            return rc;
        }
    }
    int rc = GFGPU_OK;
    if (nelem > 0) {
        DISPATCH_S(k_int_n_scalar_diag<kS><<<grid_for(nelem * nne), kBlock, 0, s>>>(
            N, vol, qscalar, nelem, nne, nip, ndim, elemvec, flag));
        rc = check_launch("int_n_scalar_nt_dv_diag");
    }
    if (!is_diag) return rc;
    *is_diag = 0;
    if (rc == GFGPU_OK) rc = check_cuda(cudaMemcpyAsync(is_diag, flag, sizeof(int), cudaMemcpyDeviceToHost, s), "cudaMemcpyAsync");
    const int rc_free = check_cuda(cudaFreeAsync(flag, s), "cudaFreeAsync");
    if (rc == GFGPU_OK) rc = rc_free;
    if (rc == GFGPU_OK) rc = check_cuda(cudaStreamSynchronize(s), "cudaStreamSynchronize");
    return rc;
}

int gfgpu_int_grad_n_dot_tensor2_dv(const double* dNx, const double* vol, const double* qtensor,
                                    int64_t nelem, int32_t nne, int32_t nip, int32_t ndim,
                                    double* elemvec, gfgpu_stream_t stream)
{
    GF_REQUIRE(dNx && vol && qtensor && elemvec && nip > 0, "bad argument");
    GF_TRY(check_elem(nne, ndim));
    GF_REQUIRE(!too_big(nelem * nip * 24), "too many elements");
    GF_REQUIRE(aligned16(dNx) && aligned16(qtensor), "dNx and qtensor must be 16-byte aligned");
    if (nelem == 0) return GFGPU_OK;
    const Shape l = spread(nelem, 128);
    if (ndim == 2)
        DISPATCH_S(k_int_grad_tensor2<kS, 4, 2><<<l.grid, l.block, 0, S(stream)>>>(dNx, vol, qtensor, nelem,
                                                                                   nip, elemvec));
    else
        DISPATCH_S(k_int_grad_tensor2<kS, 8, 3><<<l.grid, l.block, 0, S(stream)>>>(dNx, vol, qtensor, nelem,
                                                                                   nip, elemvec));
    return check_launch("int_grad_n_dot_tensor2_dv");
}

int gfgpu_int_grad_n_dot_tensor4_dot_grad_nt_dv(const double* dNx, const double* vol,
                                                const double* qtensor4, int64_t nelem,
                                                int32_t nne, int32_t nip, int32_t ndim,
                                                double* elemmat, gfgpu_stream_t stream)
{
    GF_REQUIRE(dNx && vol && qtensor4 && elemmat && nip > 0, "bad argument");
    GF_TRY(check_elem(nne, ndim));
    int64_t K = nne * ndim;
    GF_REQUIRE(!too_big(nelem * K * K), "too many elements");
    if (nelem == 0) return GFGPU_OK;
    if (ndim == 2)
        GF_TRY((launch_int_tensor4<4, 2>(dNx, vol, qtensor4, nelem, nip, elemmat, S(stream))));
    else
        GF_TRY((launch_int_tensor4<8, 3>(dNx, vol, qtensor4, nelem, nip, elemmat, S(stream))));
    return check_launch("int_grad_n_dot_tensor4_dot_grad_nt_dv");
}

// ---------------------------------------------------------------- QuadraturePlanar

int gfgpu_quad4_planar_compute_dN(const double* x, int64_t nelem, const double* xi,
                                  const double* w, int32_t nip, double thick, double* N,
                                  double* dNxi, double* dNx, double* vol, gfgpu_stream_t stream)
{
    return compute_dN(2, x, nelem, xi, w, nip, N, dNxi, dNx, vol, stream, thick);
}

int gfgpu_grad_n_vector_planar(const double* dNx, const double* elemvec, int64_t nelem,
                               int32_t nip, double* qtensor, gfgpu_stream_t stream)
{
    return grad<0>(dNx, elemvec, nelem, 4, nip, 2, qtensor, stream, true);
}

int gfgpu_grad_n_vector_T_planar(const double* dNx, const double* elemvec, int64_t nelem,
                                 int32_t nip, double* qtensor, gfgpu_stream_t stream)
{
    return grad<1>(dNx, elemvec, nelem, 4, nip, 2, qtensor, stream, true);
}

int gfgpu_sym_grad_n_vector_planar(const double* dNx, const double* elemvec, int64_t nelem,
                                   int32_t nip, double* qtensor, gfgpu_stream_t stream)
{
    return grad<2>(dNx, elemvec, nelem, 4, nip, 2, qtensor, stream, true);
}

int gfgpu_int_grad_n_dot_tensor2_dv_planar(const double* dNx, const double* vol,
                                           const double* qtensor, int64_t nelem, int32_t nip,
                                           double* elemvec, gfgpu_stream_t stream)
{
    GF_REQUIRE(dNx && vol && qtensor && elemvec && nip > 0, "bad argument");
    GF_REQUIRE(!too_big(nelem * nip * 9), "too many elements");
    GF_REQUIRE(aligned16(dNx), "dNx must be 16-byte aligned");
    if (nelem == 0) return GFGPU_OK;
    unsigned g = grid_for(nelem, 128);
    DISPATCH_S(k_int_grad_tensor2<kS, 4, 2, 3><<<g, 128, 0, S(stream)>>>(dNx, vol, qtensor, nelem,
                                                                         nip, elemvec));
    return check_launch("int_grad_n_dot_tensor2_dv_planar");
}

int gfgpu_int_grad_n_dot_tensor4_dot_grad_nt_dv_planar(const double* dNx, const double* vol,
                                                       const double* qtensor4, int64_t nelem,
                                                       int32_t nip, double* elemmat,
                                                       gfgpu_stream_t stream)
{
    GF_REQUIRE(dNx && vol && qtensor4 && elemmat && nip > 0, "bad argument");
    GF_REQUIRE(!too_big(nelem * 64) && !too_big(nelem * nip * 81), "too many elements");
    if (nelem == 0) return GFGPU_OK;
    GF_TRY((launch_int_tensor4<4, 2, 3>(dNx, vol, qtensor4, nelem, nip, elemmat, S(stream))));
    return check_launch("int_grad_n_dot_tensor4_dot_grad_nt_dv_planar");
}

int gfgpu_elastic_stress(const double* eps, const double* K, const double* G, int64_t nelem,
                         int32_t nip, int32_t ndim, double* sig, gfgpu_stream_t stream)
{
    GF_REQUIRE(eps && K && G && sig && nip > 0 && (ndim == 2 || ndim == 3), "bad argument");
    GF_REQUIRE(!too_big(nelem * nip * 9), "too many elements");
    if (nelem == 0) return GFGPU_OK;
    const unsigned g = grid_for(nelem * nip);
    cudaStream_t s = S(stream);
    if (strict_mode())
        k_stress_strict<<<g, kBlock, 0, s>>>(eps, K, G, nelem, nip, ndim, sig);
    else if (ndim == 3)
        k_stress<3><<<g, kBlock, 0, s>>>(eps, K, G, nelem * nip, nip, sig);
    else if (aligned16(eps) && aligned16(sig)) {
        auto run = [&](auto kernel, int p) {
            kernel<<<grid_for(nelem * nip / p), kBlock, 0, s>>>(reinterpret_cast<const double2*>(eps), K, G,
                                                                nelem * nip / p, static_cast<uint32_t>(nip / p),
                                                                reinterpret_cast<double2*>(sig));
        };
        if (nip % 2 == 0) run(k_stress_2d<2>, 2);
        else run(k_stress_2d<1>, 1);
    }
    else
        k_stress<2><<<g, kBlock, 0, s>>>(eps, K, G, nelem * nip, nip, sig);
    return check_launch("elastic_stress");
}

} // extern "C"
