// Projection of element Hessians to positive definite by a group of lanes per matrix:
// k_project_pd_warp (18 x 18 and 24 x 24 in float and double, 30 x 30 in double, one warp per matrix)
// and k_project_pd_tile12 (12 x 12 in double, three matrices per warp); and row-major 12 x 12 in
// float by a thread per matrix (k_project_pd_rows12).
//
// Reference: project_to_PD_inplace (symx/src/solver/second_order/project_to_PD.cpp:12-81), applied
// per element by ElementHessians.cpp:48-67.
//
// Steps per matrix H (N x N, NB = N / 3 nodes):
//   1. When H annihilates the rigid translations (every elastic energy's does, up to rounding), it
//      is deflated: B = Q^T H Q, Q the Helmert basis of the node space orthogonal to (1, ..., 1)
//      (x) I3, M = N - 3.  Otherwise B = H, M = N.
//   2. A Cholesky factorization of B - eps I in float (B deflated).  With pivots above 16 M u of B's
//      largest diagonal entry (float), or when it stands a further shift by a bound of all rounding
//      errors (double: no eigenvalue of B is below eps then), H stays as it is (the projection would
//      only lift the translations' eigenvalues from 0 to eps).
//   3. Cyclic Jacobi of B in float (jacobi_sweeps).
//   4. double: the float eigenvectors X precondition the double decomposition.  X is
//      orthonormalized in double, X <- X (I - E / 2 + 3/8 E^2) with E = X^T X - I (the series of
//      (I + E)^-1/2, error E^3 ~ 1e-18), and Jacobi runs on S = X^T B X, whose off-diagonal part
//      is already ~1e-7 of it: one sweep and a first-order correction find the invariant subspace of
//      the clamped eigenvalues to rounding (OpenSubspace), where a start from B takes seven
//      sweeps.  On GB300 an FP64 instruction holds a quarter SM's FP64 pipe for 64 clocks per
//      warp, so their number is the time.
//   5. The eigenvalues below eps enter as a correction, H + Q (sum over them of (lam' - lam) v v^T)
//      Q^T, plus the lifted translations: eigenpairs that stay do not touch H.
#include <algorithm>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>

#include "kernels.cuh"
#include "project_pd.cuh"

namespace symxg {

namespace {

template <typename T>
struct Vec2;
template <>
struct Vec2<float> {
    using type = float2;
};
template <>
struct Vec2<double> {
    using type = double2;
};

// Lanes of a warp that share one matrix: L lanes (gl: lane within the group; member: false for
// the lanes past the last group).  Every reduction and barrier below is the whole warp's; groups
// without work follow along on their own shared memory.
template <int L>
__device__ __forceinline__ float group_max(float v, float* red, int gl, bool member)
{
    if constexpr (L == 32) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
        return v;
    } else {
        if (member) red[gl] = v;
        __syncwarp();
        float m = v;
        if (member) {
#pragma unroll
            for (int k = 0; k < L; ++k) m = fmaxf(m, red[k]);
        }
        __syncwarp();
        return m;
    }
}

// Jacobi rotation of the 2 x 2 block (app, apq; apq, aqq): (c, s), and the block after it.
__device__ __forceinline__ void rotate_pair(float& app, float& apq, float& aqq, float& c, float& s)
{
    const float t = symxg_dev::jacobi_t(app, aqq, apq);
    c = symxg_dev::inv_hypot1(t);
    s = t * c;
    app = app - t * apq;
    aqq = aqq + t * apq;
    apq = 0.f;
}
// In double the tangent is taken in float (values scaled into float's range): the rotation then
// leaves 1e-7 of a_pq, which is kept.  The cosine is the
// float rsqrt with two Newton steps, so (c, s) is a rotation to double's rounding; FP64 square
// roots and divisions would cost as much as the rest of the round.
__device__ __forceinline__ void rotate_pair(double& app, double& apq, double& aqq, double& c, double& s)
{
    const double t = (double)symxg_dev::jacobi_t(0.f, (float)(aqq - app), (float)apq);
    const double u = fma(t, t, 1.0);
    c = (double)rsqrtf((float)u);
    c = fma(0.5 * c, fma(-u * c, c, 1.0), c);
    c = fma(0.5 * c, fma(-u * c, c, 1.0), c);
    s = t * c;
    const double p1 = c * app - s * apq, p2 = c * apq - s * aqq, q1 = s * app + c * apq, q2 = s * apq + c * aqq;
    app = c * p1 - s * p2;
    apq = s * p1 + c * p2;
    aqq = s * q1 + c * q2;
}

// Parallel cyclic Jacobi on the symmetric M x M matrix A (shared memory, row stride LD, upper
// triangle), M even, in the odd-even order (R. P. Brent, F. T. Luk, "The solution of singular-value and
// symmetric eigenvalue problems on multiprocessor arrays", SIAM J. Sci. Stat. Comput. 6 (1985)): round 2 r rotates the neighbouring positions (0, 1),
// (2, 3), ..., round 2 r + 1 the positions (1, 2), (3, 4), ..., and every rotation also swaps its
// two positions, so after M rounds (a sweep) every pair of indices has met while the positions,
// hence all addresses and registers, are the same two patterns throughout (the round-robin
// order needs an offset table and moves every eigenvector register in each round).  In odd rounds
// positions M - 1 and 0 form a pair that only turns by 90 degrees: with the swap, both stay (one
// changes sign).  Written per 2 x 2 block of pairs (k, l): B_kl <- R_k^T B_kl R_l, swapped.
//   * lane k < M / 2 forms pair k's rotation from its diagonal block and publishes (c, s);
//   * the blocks above the diagonal are spread over the group's lanes;
//   * lane i < M holds row i of the eigenvectors, column j at position j.
// Stops when the largest off-diagonal entry is at most tol in every group whose `work` is set.
//
// Shared-memory banks: the four entries of a block have the same parity of columns in every lane, so
// odd lanes take their column pair in the other order (a rotation of (q, p) is the rotation of (p, q)
// with -s), and LD is chosen per N so that the rows of blocks continue each other's banks (wavefronts
// of a round's reads at 30 x 30: 34 at LD = 31 without the exchange, 25 at LD = 38).
template <typename T, int M, int L, int LD>
struct Jacobi {
    static constexpr int NP = M / 2, NOFF = NP * (NP - 1) / 2, SLOTS = (NOFF + L - 1) / L;
    using T2 = typename Vec2<T>::type;
    struct Slot {
        int k, l;          // the block's pairs
        int even0, even1;  // offsets of its first row's entries in even rounds, the second row's + LD
        int odd0, odd1;    // ... in odd rounds; the second row's of odd1 + odd_step
        int odd_step;
    };
    Slot slot[SLOTS];
    T flip;    // -1 in lanes that take the columns of a block in the other order
    int diag;  // offset of the lane's pair (first position of the even round)

    __device__ __forceinline__ explicit Jacobi(int gl)
    {
        const bool other = (gl & 1) != 0;
        flip = other ? T(-1) : T(1);
        diag = 2 * gl * (LD + 1);
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            int b = gl + L * j, k = 0;
            if (b >= NOFF) b = 0;
            while (b >= NP - 1 - k) {
                b -= NP - 1 - k;
                ++k;
            }
            const int l = k + 1 + b;
            Slot& s = slot[j];
            s.k = k;
            s.l = l;
            const int e = 2 * k * LD + 2 * l, o = (2 * k + 1) * LD + 2 * l + 1;
            // columns 2 l, 2 l + 1; in odd rounds 2 l + 1, 2 l + 2, and for the last pair M - 1 and 0
            // (column 0's entries lie transposed in row 0)
            const bool wrap = l == NP - 1;
            const int o_second = wrap ? 2 * k + 1 : o + 1;
            s.even0 = other ? e + 1 : e;
            s.even1 = other ? e : e + 1;
            s.odd0 = other ? o_second : o;
            s.odd1 = other ? o : o_second;
            s.odd_step = wrap ? 1 : LD;
        }
    }
    // B_kl <- R_k^T B_kl R_l with both pairs swapped; b00, b01 (row p of pair k), b10, b11 (row q)
    static __device__ __forceinline__ void rotate_block(T& b00, T& b01, T& b10, T& b11, const T2& rk, T cl, T sl)
    {
        const T r00 = rk.x * b00 - rk.y * b10, r01 = rk.x * b01 - rk.y * b11;
        const T r10 = rk.y * b00 + rk.x * b10, r11 = rk.y * b01 + rk.x * b11;
        b11 = cl * r00 - sl * r01;
        b10 = sl * r00 + cl * r01;
        b01 = cl * r10 - sl * r11;
        b00 = sl * r10 + cl * r11;
    }
    template <int PARITY>
    __device__ __forceinline__ void round(T* A, T2* CS, T (&v)[M], int gl, bool member, float negligible)
    {
        if (member && gl < NP) {
            T2 cs;
            if (PARITY == 1 && gl == NP - 1) {  // the pair (M - 1, 0)
                A[M - 1] = -A[M - 1];
                cs.x = T(0);
                cs.y = T(1);
            } else {
                T* d = A + diag + PARITY * (LD + 1);
                T app = d[0], apq = d[1], aqq = d[LD + 1];
                cs.x = T(1);
                cs.y = T(0);
                if (fabsf((float)apq) > negligible) rotate_pair(app, apq, aqq, cs.x, cs.y);
                else apq = T(0);
                d[0] = aqq;
                d[1] = apq;
                d[LD + 1] = app;
            }
            CS[gl] = cs;
        }
        __syncwarp();
        if (member) {
#pragma unroll
            for (int j = 0; j < SLOTS; ++j) {
                if ((j + 1) * L <= NOFF || gl + L * j < NOFF) {
                    const Slot& sl = slot[j];
                    const T2 rk = CS[sl.k], rl = CS[sl.l];
                    T* x = A + (PARITY == 0 ? sl.even0 : sl.odd0);
                    T* y = A + (PARITY == 0 ? sl.even1 : sl.odd1);
                    T *x2 = x + LD, *y2 = y + LD;
                    if (PARITY == 1) {  // the column that wraps keeps its rows next to each other
                        const bool other = flip < T(0);
                        if (other) x2 = x + sl.odd_step;
                        else y2 = y + sl.odd_step;
                    }
                    T b00 = *x, b01 = *y, b10 = *x2, b11 = *y2;
                    rotate_block(b00, b01, b10, b11, rk, rl.x, rl.y * flip);
                    *x = b00;
                    *y = b01;
                    *x2 = b10;
                    *y2 = b11;
                }
            }
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const int p = 2 * k + PARITY, q = p + 1 < M ? p + 1 : 0;
                const T2 cs = CS[k];
                const T vp = v[p], vq = v[q];
                v[q] = cs.x * vp - cs.y * vq;
                v[p] = cs.y * vp + cs.x * vq;
            }
        }
        __syncwarp();
    }
    // Whether the entry a of A at (r, c) keeps the iteration going.
    struct LargeEntries {  // any above tol
        float tol;
        __device__ __forceinline__ bool operator()(const T*, int, int, T a) const { return fabsf((float)a) > tol; }
    };
    // Sweeps until no entry above the diagonal is `open` in a group whose `work` is set; false in a
    // group that reached the cap.  A group without open entries sits the others' sweeps out: its result
    // does not depend on the matrices that share its warp.  Entries below negligible (under the rounding of max |H|) are dropped
    // instead of rotated: between equal eigenvalues such an entry would turn its pair by 45 degrees in
    // every sweep and mix what the other rotations have separated.
    template <typename Open>
    __device__ __forceinline__ bool sweeps(T* A, T2* CS, float* red, T (&v)[M], int gl, bool member, bool work,
                                           float negligible, int max_sweeps, Open is_open)
    {
        for (int sweep = 0;; ++sweep) {
            float m = 0.f;
            if (member)
                for (int i = gl; i < M * M; i += L) {
                    const int r = i / M, c = i % M;
                    if (r < c && is_open(A, r, c, A[r * LD + c])) m = 1.f;
                }
            const bool open = group_max<L>(m, red, gl, member) > 0.f && work;
            if (!__any_sync(0xffffffffu, open)) return true;
            if (sweep == max_sweeps) return !open;
#pragma unroll 1
            for (int r = 0; r < M / 2; ++r) {
                round<0>(A, CS, v, gl, member && open, negligible);
                round<1>(A, CS, v, gl, member && open, negligible);
            }
        }
    }
};

// Row stride of the matrices in shared memory.
template <int N>
constexpr int kStride = N == 12 ? 13 : N == 18 ? 22 : N == 24 ? 25 : 38;

// What ends the double Jacobi: only the invariant subspace of the clamped eigenvalues (below eps) has
// to be found, not the single eigenvectors.  An entry between a clamped and a kept position may stay
// up to 2^-27 of their distance: the first-order correction that follows leaves its square.  Entries
// between two positions of the same kind may stay while they are small against the distances to
// eps (the sign of lam - eps then holds for the whole subspace).
template <int M, int LD>
struct OpenSubspace {
    double eps;
    float tol;
    __device__ __forceinline__ bool operator()(const double* A, int r, int c, double a) const
    {
        const float x = fabsf((float)a);
        if (!(x > tol)) return false;
        const double dr = A[r * LD + r] - eps, dc = A[c * LD + c] - eps;
        if ((dr < 0.0) != (dc < 0.0)) return x > 7.4505806e-09f * fabsf((float)(dr - dc));
        return x * (float)M > fminf(fabsf((float)dr), fabsf((float)dc));
    }
};

// Helmert column m of the translations' complement: 1 / sqrt(m (m + 1)) for the nodes before m,
// -m times that for node m.
template <typename T, int NB>
struct Helmert {
    T c[NB];
    __device__ __forceinline__ Helmert()
    {
        c[0] = T(0);
#pragma unroll
        for (int m = 1; m < NB; ++m) c[m] = T(1) / sqrt(T(m * (m + 1)));  // constants, folded at compile time
    }
};

// Shared memory of one group: two matrices (three in double) of N x N, row stride kStride, the (c, s)
// of a round, and the reductions' scratch.
template <typename T, int N>
struct GroupMem {
    static constexpr int LD = kStride<N>, mat = N * LD;
    static constexpr size_t bytes =
        ((sizeof(T) == 8 ? 3 : 2) * (size_t)mat * sizeof(T) + (size_t)N * sizeof(T) + 32 * sizeof(float) + 15) / 16 * 16;
    T *a, *b, *s;
    typename Vec2<T>::type* cs;
    float* red;
    __device__ __forceinline__ explicit GroupMem(unsigned char* p)
    {
        a = reinterpret_cast<T*>(p);
        b = a + mat;
        s = sizeof(T) == 8 ? b + mat : b;
        cs = reinterpret_cast<typename Vec2<T>::type*>(s + mat);
        red = reinterpret_cast<float*>(reinterpret_cast<T*>(cs) + N);
    }
};

// The matrix h times `scale` into g.a (row-major), amax = max |entry| of it, and g.b = Q^T (scale h) Q
// (M x M).  Returns whether it is translation-invariant: max |H t| <= tol max |H|.  In double, scale
// is the power of two that brings amax into [1, 2), so the float stages cannot overflow, or a smaller
// one when eps times it could leave double's range (a matrix that is zero beside eps).
template <typename T, int N, int L, bool Rows>
__device__ __forceinline__ bool load_and_deflate(const T* __restrict__ h, const GroupMem<T, N>& g, int gl, bool member,
                                                 bool work, T eps, float& amax, T& scale)
{
    constexpr int LD = kStride<N>, NB = N / 3, M = N - 3;
    const Helmert<T, NB> hm;
    T hmax = T(0);
    if (work)
        for (int idx = gl; idx < N * N; idx += L) {  // read in storage order
            const int blk = idx / 9, r = idx % 9;
            const T v = h[idx];
            g.a[Rows ? (idx / N) * LD + idx % N : ((blk / NB) * 3 + r / 3) * LD + (blk % NB) * 3 + r % 3] = v;
            hmax = fmax(hmax, fabs(v));
        }
    scale = T(1);
    if constexpr (sizeof(T) == 8) {
        int ex = -1000;
        if (eps > 0.0 && eps < (double)INFINITY) ex = max(ex, ilogb(eps) - 1000);
        if (hmax > 0.0 && hmax < (double)INFINITY) ex = max(ex, ilogb(hmax));
        ex = (int)group_max<L>((float)(ex + 2000), g.red, gl, member) - 2000;
        scale = scalbn(1.0, -ex);
        __syncwarp();  // the loop below reads what other lanes stored (group_max<32> orders no memory)
        if (work && scale != 1.0)
            for (int idx = gl; idx < N * N; idx += L) g.a[(idx / N) * LD + idx % N] *= scale;
    }
    amax = group_max<L>((float)(hmax * scale), g.red, gl, member);
    __syncwarp();
    // rows of H Q by prefix sums over the node blocks; the full sums are the translation residual
    float outside = 0.f;
    if (member)
        for (int i = gl; i < N; i += L) {
            T acc[3] = {T(0), T(0), T(0)};
#pragma unroll
            for (int m = 0; m < NB; ++m)
#pragma unroll
                for (int e = 0; e < 3; ++e) {
                    const T a = g.a[i * LD + 3 * m + e];
                    if (m >= 1) g.b[i * LD + 3 * (m - 1) + e] = (acc[e] - T(m) * a) * hm.c[m];
                    acc[e] += a;
                }
#pragma unroll
            for (int e = 0; e < 3; ++e)
                if (!(fabs(acc[e]) <= symxg_dev::DeflationTol<T>::value() * (T)amax)) outside = 1.f;
        }
    const bool invariant = group_max<L>(outside, g.red, gl, member) == 0.f;
    __syncwarp();
    if (member)  // columns of Q^T (H Q), written over rows 0 .. M - 1 of the same column
        for (int c = gl; c < M; c += L) {
            T acc[3] = {T(0), T(0), T(0)};
#pragma unroll
            for (int m = 0; m < NB; ++m)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const T t = g.b[(3 * m + d) * LD + c];
                    if (m >= 1) g.b[(3 * (m - 1) + d) * LD + c] = (acc[d] - T(m) * t) * hm.c[m];
                    acc[d] += t;
                }
        }
    __syncwarp();
    return invariant;
}

// Float: true when B - eps I (M x M, row stride LD) has a Cholesky factorization with every pivot
// above 16 M u of B's largest diagonal entry.  Double: true when a float one proves that every
// eigenvalue of B is at least eps (DefiniteShift).  f: M x M floats, stride LD.  One warp.
template <typename T, int M, int LD>
__device__ __forceinline__ bool eigenvalues_above(const T* B, float* f, float eps, int lane)
{
    for (int idx = lane; idx < M * M; idx += 32) {
        const int i = idx / M, j = idx % M;
        if (i >= j) f[i * LD + j] = (float)B[i * LD + j];
    }
    __syncwarp();
    const float u = symxg_dev::UnitRoundoff<float>::value();
    const float d0 = lane < M ? f[lane * LD + lane] : 0.f;
    float shift = fmaxf(eps, 0.f), tau = 0.f;
    if constexpr (sizeof(T) == 4) {
        float dmax = d0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dmax = fmaxf(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
        tau = 16.f * M * u * dmax;
    } else {
        float trace = d0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) trace += __shfl_xor_sync(0xffffffffu, trace, o);
        shift += symxg_dev::DefiniteShift<M>::converted * u * trace;
    }
// (not unrolled as a whole: 8,000 positive definite 24 x 24 matrices in float 55.1 us, so 53.9)
#pragma unroll 3
    for (int j = 0; j < M; ++j) {
        const float d = f[j * LD + j] - shift;  // the same value in every lane
        if (!(d > tau)) return false;
        const float r = 1.f / sqrtf(d);
        const bool mine = lane > j && lane < M;
        const float lij = mine ? f[lane * LD + j] * r : 0.f;
        __syncwarp();
        if (mine) f[lane * LD + j] = lij;
        __syncwarp();
        if (mine)
            for (int k = j + 1; k <= lane; ++k) f[lane * LD + k] -= lij * f[k * LD + j];
        __syncwarp();
    }
    return true;
}

// Off-diagonal entries relative to max |H|: 2^-19 ends the float Jacobi, 2^-20 the one that
// preconditions; at 2^-48 an entry of the double one counts as zero (rounding leaves about a tenth of
// each).
constexpr float kOffFloat = 1.9073486e-06f, kOffPrecondition = 9.5367432e-07f, kOffDouble = 3.5527137e-15f;
constexpr int kMaxSweepsFloat = 16, kMaxSweepsDouble = 20;

// Steps 3 to 5 for a loaded matrix: B = g.b when deflated, else g.a.  Returns false in a group that
// reached a sweep cap.
template <typename T, int N, int L, bool Deflate, bool Rows>
__device__ __forceinline__ bool decompose_and_correct(T* __restrict__ h, const GroupMem<T, N>& g, int gl, bool member,
                                                      bool work, float amax, T scale, T eps, bool mirroring)
{
    constexpr int NB = N / 3, M = Deflate ? N - 3 : N, M2 = (M + 1) & ~1, LD = kStride<N>;
    static_assert(M2 <= L, "a lane per row");
    const bool mine = member && gl < M2;
    eps *= scale;
    // an index M of its own when M is odd, with an eigenvalue that is never clamped
    const T pad = fmax((T)amax, eps);
    T* const B = Deflate ? g.b : g.a;
    T* const other = Deflate ? g.a : g.b;
    T *A, *V, *W;  // the diagonalized matrix, the eigenvectors (row i: components i), the correction
    bool ok;
    T v[M2];
    if constexpr (sizeof(T) == 4) {
        A = W = B;
        V = other;
        if (mine && M2 > M) A[gl * LD + M] = gl == M ? pad : 0.f;
#pragma unroll
        for (int k = 0; k < M2; ++k) v[k] = gl == k ? 1.f : 0.f;
        __syncwarp();
        using Jac = Jacobi<float, M2, L, LD>;
        ok = Jac(gl).sweeps(A, g.cs, g.red, v, gl, member, work, kOffFloat / 64.f * amax, kMaxSweepsFloat,
                            typename Jac::LargeEntries{kOffFloat * amax});
    } else {
        A = other;
        V = g.s;
        W = B;
        {
            float* F = reinterpret_cast<float*>(g.s);
            const float fpad = fmaxf(2.f, (float)pad);
            if (member)
                for (int idx = gl; idx < M2 * M2; idx += L) {
                    const int i = idx / M2, j = idx % M2;
                    F[i * LD + j] = i < M && j < M ? (float)B[i * LD + j] : i == j ? fpad : 0.f;
                }
            float x[M2];
#pragma unroll
            for (int k = 0; k < M2; ++k) x[k] = gl == k ? 1.f : 0.f;
            __syncwarp();
            using Jac = Jacobi<float, M2, L, LD>;
            ok = Jac(gl).sweeps(F, reinterpret_cast<float2*>(g.cs), g.red, x, gl, member, work,
                                kOffPrecondition / 64.f * amax, kMaxSweepsFloat,
                                typename Jac::LargeEntries{kOffPrecondition * amax});
            if (mine)
#pragma unroll
                for (int k = 0; k < M2; ++k) other[gl * LD + k] = (double)x[k];
        }
        __syncwarp();
        // lane j: column j of E = X^T X - I, of P = -E / 2 + 3/8 E^2 (E^2 ~ 1e-12: in float) and of
        // X + X P
        double y[M2];
        if (mine) {
#pragma unroll
            for (int k = 0; k < M2; ++k) y[k] = other[k * LD + gl];
#pragma unroll 1
            for (int i = 0; i < M2; ++i) {
                double t = i == gl ? -1.0 : 0.0;
#pragma unroll
                for (int k = 0; k < M2; ++k) t = fma(other[k * LD + i], y[k], t);
                g.s[i * LD + gl] = t;
            }
        }
        __syncwarp();
        if (mine) {
            float e[M2];
#pragma unroll
            for (int k = 0; k < M2; ++k) e[k] = (float)g.s[k * LD + gl];
#pragma unroll
            for (int i = 0; i < M2; ++i) {
                float t = 0.f;
#pragma unroll
                for (int k = 0; k < M2; ++k) t = fmaf((float)g.s[i * LD + k], e[k], t);
                y[i] = fma(-0.5, g.s[i * LD + gl], 0.375 * (double)t);
            }
        }
        __syncwarp();
        if (mine)
#pragma unroll 1
            for (int i = 0; i < M2; ++i) {
                double t = other[i * LD + gl];
#pragma unroll
                for (int k = 0; k < M2; ++k) t = fma(other[i * LD + k], y[k], t);
                g.s[i * LD + gl] = t;
            }
        __syncwarp();
        // lane j: B x_j, then column j of S = X^T B X
        if (mine) {
#pragma unroll
            for (int k = 0; k < M2; ++k) y[k] = g.s[k * LD + gl];
#pragma unroll 1
            for (int i = 0; i < M; ++i) {
                double t = 0.0;
#pragma unroll
                for (int k = 0; k < M; ++k) t = fma(B[i * LD + k], y[k], t);
                other[i * LD + gl] = t;
            }
            if (M2 > M) other[M * LD + gl] = pad * y[M2 - 1];
#pragma unroll
            for (int k = 0; k < M2; ++k) y[k] = other[k * LD + gl];
#pragma unroll 1
            for (int i = 0; i < M2; ++i) {
                double t = 0.0;
#pragma unroll
                for (int k = 0; k < M2; ++k) t = fma(g.s[k * LD + i], y[k], t);
                other[i * LD + gl] = t;
            }
#pragma unroll
            for (int k = 0; k < M2; ++k) v[k] = g.s[gl * LD + k];
        }
        __syncwarp();
        ok = Jacobi<double, M2, L, LD>(gl).sweeps(A, g.cs, g.red, v, gl, member, work, kOffDouble / 64.f * amax,
                                                  kMaxSweepsDouble, OpenSubspace<M2, LD>{eps, kOffDouble * amax}) && ok;
    }
    if (mine)
#pragma unroll
        for (int k = 0; k < M2; ++k) V[gl * LD + k] = v[k];
    __syncwarp();
    bool changed = false;
    if constexpr (sizeof(T) == 8) {
        // clamped vectors: v_k + sum over the kept u of v_u S_uk / (S_kk - S_uu), the quotients (below
        // 2^-27) in float
        if (mine)
            for (int k = 0; k < M2; ++k) {
                const T lam = A[k * LD + k];
                if (!(lam < eps)) continue;
                T t = V[gl * LD + k];
#pragma unroll 4
                for (int u = 0; u < M2; ++u) {
                    const T lu = A[u * LD + u];
                    if (lu < eps) continue;
                    const float q = (float)(u < k ? A[u * LD + k] : A[k * LD + u]) / (float)(lam - lu);
                    t = fma(V[gl * LD + u], (T)q, t);
                }
                V[gl * LD + k] = t;  // row gl is this lane's, and kept columns are not written
            }
        __syncwarp();
    }
    // row gl of the correction sum v_k (f(S_cc) - S_cc)_kl v_l^T over the clamped positions, f(lam) = eps
    // or -lam; S_cc is diagonal to rounding in float
    T w[M];
#pragma unroll
    for (int j = 0; j < M; ++j) w[j] = T(0);
    if (mine)
        for (int k = 0; k < M2; ++k) {
            const T lam = A[k * LD + k];
            if (!(lam < eps)) continue;
            changed = true;
            T t = ((mirroring ? -lam : eps) - lam) * V[gl * LD + k];
            if constexpr (sizeof(T) == 8) {
                for (int l = 0; l < M2; ++l) {
                    if (l == k || !(A[l * LD + l] < eps)) continue;
                    t = fma((mirroring ? T(-2) : T(-1)) * (l < k ? A[l * LD + k] : A[k * LD + l]), V[gl * LD + l], t);
                }
            }
#pragma unroll
            for (int j = 0; j < M; ++j) w[j] = fma(t, V[j * LD + k], w[j]);
        }
    const T unscale = T(1) / scale;  // a power of two
    // 12 x 12: both triangles from one value, as in the forms with a thread per matrix
    constexpr bool both = N == 12;
    auto add_both = [&](int i, int j, T correction) {
        T* const p = h + symxg_dev::h_index<N, Rows>(i, j);
        const T sum = *p + correction;
        *p = sum;
        h[symxg_dev::h_index<N, Rows>(j, i)] = sum;
    };
    __syncwarp();
    if constexpr (!Deflate) {
        if (work && changed && gl < M)
#pragma unroll
            for (int j = 0; j < M; ++j) {
                if constexpr (!both) h[Rows ? gl * N + j : ((gl / 3) * NB + j / 3) * 9 + (gl % 3) * 3 + j % 3] += w[j] * unscale;
                else if (j >= gl) add_both(gl, j, w[j] * unscale);
            }
    } else {
        // Q w Q^T by suffix sums over the nodes: columns of the own row, then rows of the own columns;
        // the translations' eigenvalues 0 -> eps (0 when mirroring)
        const Helmert<T, NB> hm;
        T lam_t = T(0);
        if (T(0) < eps) {
            changed = true;
            lam_t = mirroring ? T(0) : eps;
        }
        if (member && gl < M) {
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                T tail = T(0);
#pragma unroll
                for (int m = NB - 1; m >= 1; --m) {
                    const T t = hm.c[m] * w[3 * (m - 1) + e];
                    W[gl * LD + 3 * m + e] = tail - T(m) * t;
                    tail += t;
                }
                W[gl * LD + e] = tail;
            }
        }
        changed = group_max<L>(changed ? 1.f : 0.f, g.red, gl, member) > 0.f;  // lanes past M2 write columns too
        __syncwarp();
        if (work && changed)
            for (int c = gl; c < N; c += L) {
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const T lift = c % 3 == d ? lam_t / T(NB) : T(0);
                    T tail = T(0);
                    T* const hc = h + (Rows ? d * N + c : (c / 3) * 9 + d * 3 + c % 3);
#pragma unroll
                    for (int m = NB - 1; m >= 1; --m) {
                        const T t = hm.c[m] * W[(3 * (m - 1) + d) * LD + c];
                        if constexpr (!both) hc[m * 3 * N] += (tail - T(m) * t + lift) * unscale;
                        else if (3 * m + d <= c) add_both(3 * m + d, c, (tail - T(m) * t + lift) * unscale);
                        tail += t;
                    }
                    if constexpr (!both) hc[0] += (tail + lift) * unscale;
                    else if (d <= c) add_both(d, c, (tail + lift) * unscale);
                }
            }
    }
    __syncwarp();  // the next matrix reuses the group's shared memory
    return ok;
}

// ---- one warp per matrix
// Measured against Jacobi over all N indices (round-robin order, FP64 throughout in double): 16,687
// 24 x 24 Hessians in float 891 -> 558 us (bound by issue and shared memory), 2,001 in double (70 %
// indefinite) 3.74 -> 0.97 ms (bound by the FP64 pipe: the fullest quarter SM's is busy for 81 % of the
// time, the average one's for 47 %).  30 x 30 in float stays with that form (k_project_pd_pairs, 631 us for 5,940):
// this one takes 449 us, but its other rounding moves the positions at which a Newton solve of
// quadratic tetrahedra stops in mixed precision by up to 5e-9 of them.
//
// A block tests a tile of matrices, one per warp, and its warps then share the listed ones evenly
// (with the decomposition right after the test, warps that met only positive definite matrices
// waited for those that met none).  One block of eight warps per SM in double: with two of four,
// each block's fifth matrix fell on the same quarter SM and its FP64 pipe.
constexpr int kMaxTile = 512;
template <typename T, int N>
struct WarpCfg {
    static constexpr int warps = 8;
    // float: 80 registers, at most 24 bytes of spills (four blocks per SM spill more: 600 us where three
    // take 558); double: 255
    static constexpr int min_blocks = sizeof(T) == 4 ? 3 : 1;
    static constexpr size_t smem = warps * GroupMem<T, N>::bytes;
};

template <typename T, int N, bool Rows>
__global__ void __launch_bounds__(WarpCfg<T, N>::warps * 32, WarpCfg<T, N>::min_blocks)
    k_project_pd_warp(T* __restrict__ H, int64_t count, int tile, T eps, int mirroring, int* not_converged,
                      const int64_t* __restrict__ sel)
{
    constexpr int W = WarpCfg<T, N>::warps;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ short list[kMaxTile];  // matrices of the tile to decompose; general ones as -1 - index
    __shared__ int n_list;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const GroupMem<T, N> g(smem + w * GroupMem<T, N>::bytes);
    float amax;
    T scale;
    bool ok = true;
    for (int64_t base = (int64_t)blockIdx.x * tile; base < count; base += (int64_t)gridDim.x * tile) {
        const int n = (int)(count - base < tile ? count - base : tile);
        auto at = [&](int i) { return H + (sel ? sel[base + i] : base + i) * (int64_t)(N * N); };
        if (threadIdx.x == 0) n_list = 0;
        __syncthreads();
        for (int i = w; i < n; i += W) {
            const bool invariant = load_and_deflate<T, N, 32, Rows>(at(i), g, lane, true, true, eps, amax, scale);
            bool done = false;
            if (invariant)
                done = eigenvalues_above<T, N - 3, kStride<N>>(g.b, reinterpret_cast<float*>(sizeof(T) == 8 ? g.s : g.a),
                                                               (float)(eps * scale), lane);
            if (!done && lane == 0) list[atomicAdd(&n_list, 1)] = (short)(invariant ? i : -1 - i);
            __syncwarp();
        }
        __syncthreads();
        const int pending = n_list;
        for (int k = w; k < pending; k += W) {
            const int i = list[k];
            T* h = at(i < 0 ? -1 - i : i);
            load_and_deflate<T, N, 32, Rows>(h, g, lane, true, true, eps, amax, scale);
            if (i >= 0)
                ok = decompose_and_correct<T, N, 32, true, Rows>(h, g, lane, true, true, amax, scale, eps, mirroring != 0) && ok;
            else
                ok = decompose_and_correct<T, N, 32, false, Rows>(h, g, lane, true, true, amax, scale, eps, mirroring != 0) && ok;
        }
        __syncthreads();
    }
    if (!ok) *not_converged = 1;
}

// ---- 12 x 12 in double: tiles of matrices
// A block sorts a tile of matrices, one per thread in float (positive definite ones are done; the
// translation residual is formed in double), then decomposes the others with dense warps: three
// deflated matrices per warp (10 lanes each) or two full ones (16 lanes each).  One thread per
// matrix in double (a serial chain of ~60,000 FP64 operations) took 1.2 ms for any count up to
// the 19,456 that fill the chip once.
constexpr int kTileThreads = 128;

template <bool Rows>
__global__ void __launch_bounds__(kTileThreads, 3)
    k_project_pd_tile12(double* __restrict__ H, int64_t count, int tile, double eps, int mirroring, int* not_converged,
                        const int64_t* __restrict__ sel)
{
    constexpr int N = 12, W = kTileThreads / 32;
    using Mem = GroupMem<double, N>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int64_t list[2][kTileThreads];
    __shared__ int n_list[2];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    bool ok = true;
    for (int64_t base = (int64_t)blockIdx.x * tile; base < count; base += (int64_t)gridDim.x * tile) {
        if (tid < 2) n_list[tid] = 0;
        __syncthreads();
        if (tid < tile && base + tid < count) {
            const int64_t m = sel ? sel[base + tid] : base + tid;
            const int c = symxg_dev::classify12<Rows>(H + m * (N * N), eps);
            if (c) list[c - 1][atomicAdd(&n_list[c - 1], 1)] = m;
        }
        __syncthreads();
        const int n1 = n_list[0], n2 = n_list[1];
        const int turn = (w + (int)((int64_t)blockIdx.x * W / gridDim.x)) % W;  // an SM's blocks start on different quarters
        for (int i0 = turn * 3; i0 < n1; i0 += 3 * W) {
            const int grp = lane / 10, gl = lane % 10;
            const bool member = grp < 3, work = member && i0 + grp < n1;
            const Mem g(smem + (w * 3 + (member ? grp : 2)) * Mem::bytes);
            double* h = H + (work ? list[0][i0 + grp] : 0) * (N * N);
            float amax;
            double scale;
            load_and_deflate<double, N, 10, Rows>(h, g, gl, member, work, eps, amax, scale);
            ok = decompose_and_correct<double, N, 10, true, Rows>(h, g, gl, member, work, amax, scale, eps, mirroring != 0) && ok;
        }
        for (int i0 = turn * 2; i0 < n2; i0 += 2 * W) {
            const int grp = lane / 16, gl = lane % 16;
            const bool work = i0 + grp < n2;
            const Mem g(smem + (w * 3 + grp) * Mem::bytes);
            double* h = H + (work ? list[1][i0 + grp] : 0) * (N * N);
            float amax;
            double scale;
            load_and_deflate<double, N, 16, Rows>(h, g, gl, true, work, eps, amax, scale);
            ok = decompose_and_correct<double, N, 16, false, Rows>(h, g, gl, true, work, amax, scale, eps, mirroring != 0) && ok;
        }
        __syncthreads();
    }
    if (!ok) *not_converged = 1;
}

// ---- row-major 12 x 12 in float: tiles of matrices, a thread per matrix
// A block tests a tile of matrices and lists those to decompose; its warps then share the list, so
// the decompositions (Jacobi in registers, bound by issue) run in full warps.  The blocks take the
// matrices in turn: neighbouring elements tend to be indefinite together.  200,003 Hessians of a
// deformed mesh through project_pd: 591 us with block-major copies around a kernel that tests and
// decomposes in the same thread (318 us), 314 us with this one on the rows themselves (225 us).
constexpr int kMaxTile12 = 1024;
__global__ void __launch_bounds__(kTileThreads, 3)
    k_project_pd_rows12(float* __restrict__ H, int64_t count, int tile, float eps, int mirroring, int* __restrict__ work)
{
    constexpr int N = 12, M = 9, W = kTileThreads / 32;
    __shared__ short list[kMaxTile12];
    __shared__ int n_list;
    const int tid = threadIdx.x;
    // the blocks of an SM start their lists on different quarters of it
    const int first = ((tid >> 5) + (int)((int64_t)blockIdx.x * W / gridDim.x)) % W * 32 + (tid & 31);
    int nc = 0;
    for (int64_t base = blockIdx.x; base < count; base += (int64_t)gridDim.x * tile) {
        const int64_t left = (count - base + gridDim.x - 1) / gridDim.x;
        const int n = (int)(left < tile ? left : tile);
        if (tid == 0) n_list = 0;
        __syncthreads();
        for (int i = tid; i < n; i += kTileThreads) {
            const int64_t m = base + (int64_t)i * gridDim.x;
            float b[M * (M + 1) / 2];
            if (!symxg_dev::deflate_translations<float, N / 3, true>(H + m * (N * N), b))
                work[2 + atomicAdd(work + 1, 1)] = (int)m;
            else if (!symxg_dev::eigenvalues_above_by_cholesky<float, M>(b, eps))  // those stay as they are
                list[atomicAdd(&n_list, 1)] = (short)i;
        }
        __syncthreads();
        for (int k = first; k < n_list; k += kTileThreads) {
            float* h = H + (base + (int64_t)list[k] * gridDim.x) * (N * N);
            float b[M * (M + 1) / 2];
            if (symxg_dev::deflate_translations<float, N / 3, true>(h, b))
                symxg_dev::project_deflated_finish<float, N / 3, true>(h, b, eps, mirroring != 0, &nc);
        }
        __syncthreads();
    }
    if (nc) work[0] = 1;
}

// Dynamic shared memory of `kernel` allowed once per device, and its blocks resident at once.
template <typename K>
unsigned resident_blocks(K kernel, int threads, size_t smem)
{
    static std::mutex m;
    static std::map<std::pair<const void*, int>, unsigned> cache;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(m);
    const auto key = std::make_pair((const void*)kernel, dev);
    const auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess)
        throw std::runtime_error(std::string("symx_gb300: projection shared memory: ") + cudaGetErrorString(e));
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    return cache[key] = (unsigned)std::max(1, sms * std::max(1, per_sm));
}

void check(const char* what)
{
    count_launch();
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        throw std::runtime_error(std::string("symx_gb300: launch of ") + what + " failed: " + cudaGetErrorString(e));
}

// Matrices per tile: the count shared evenly by the resident blocks in as few passes as `most` allows,
// at least `least`.
int tile_size(int64_t count, int64_t resident, int least, int most)
{
    const int64_t passes = (count + resident * most - 1) / (resident * most);
    return (int)std::max<int64_t>(least, (count + resident * passes - 1) / (resident * passes));
}

template <typename T, int N, bool Rows>
void launch_warp(T* H, int64_t count, T eps, bool mirroring, int* not_converged, const int64_t* sel, cudaStream_t s)
{
    using Cfg = WarpCfg<T, N>;
    const int64_t resident = resident_blocks(k_project_pd_warp<T, N, Rows>, Cfg::warps * 32, Cfg::smem);
    const int tile = tile_size(count, resident, Cfg::warps, kMaxTile);
    const int64_t grid = std::min<int64_t>(resident, (count + tile - 1) / tile);
    k_project_pd_warp<T, N, Rows><<<(unsigned)grid, Cfg::warps * 32, Cfg::smem, s>>>(H, count, tile, eps, mirroring, not_converged,
                                                                                    sel);
    check("project_pd_warp");
}

template <bool Rows>
void launch_tile12(double* H, int64_t count, double eps, bool mirroring, int* not_converged, const int64_t* sel, cudaStream_t s)
{
    const size_t smem = (kTileThreads / 32) * 3 * GroupMem<double, 12>::bytes;
    const int64_t resident = resident_blocks(k_project_pd_tile12<Rows>, kTileThreads, smem);
    const int tile = tile_size(count, resident, 1, kTileThreads);
    const int64_t grid = std::min<int64_t>(resident, (count + tile - 1) / tile);
    k_project_pd_tile12<Rows><<<(unsigned)grid, kTileThreads, smem, s>>>(H, count, tile, eps, mirroring, not_converged, sel);
    check("project_pd_tile12");
}

}  // namespace

void launch_project_pd_rows12(float* H, int64_t count, float eps, bool mirroring, int* work, cudaStream_t s)
{
    const int64_t resident = resident_blocks(k_project_pd_rows12, kTileThreads, 0);
    const int tile = tile_size(count, resident, 32, kMaxTile12);
    const int64_t grid = std::min<int64_t>(resident, (count + tile - 1) / tile);
    k_project_pd_rows12<<<(unsigned)grid, kTileThreads, 0, s>>>(H, count, tile, eps, mirroring, work);
    check("project_pd_rows12");
}

template <typename T, bool Rows>
bool launch_project_pd_warp(T* H, int N, int64_t count, T eps, bool mirroring, int* not_converged, const int64_t* sel,
                            cudaStream_t s)
{
    if (N == 18) launch_warp<T, 18, Rows>(H, count, eps, mirroring, not_converged, sel, s);
    else if (N == 24) launch_warp<T, 24, Rows>(H, count, eps, mirroring, not_converged, sel, s);
    else if constexpr (sizeof(T) == 8) {
        if (N == 12) launch_tile12<Rows>(H, count, eps, mirroring, not_converged, sel, s);
        else if (N == 30) launch_warp<T, 30, Rows>(H, count, eps, mirroring, not_converged, sel, s);
        else return false;
    } else
        return false;
    return true;
}
#define INSTANTIATE(T, ROWS) \
    template bool launch_project_pd_warp<T, ROWS>(T*, int, int64_t, T, bool, int*, const int64_t*, cudaStream_t);
INSTANTIATE(float, false)
INSTANTIATE(float, true)
INSTANTIATE(double, false)
INSTANTIATE(double, true)

}  // namespace symxg
