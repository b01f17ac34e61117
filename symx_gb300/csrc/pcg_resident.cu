// Block-Jacobi PCG with the matrix held in shared memory: all iterations in one cooperative
// launch of at most one block per SM (see k_pcg_resident).
//
// Reference: bsm::solve_pcg (solve_pcg.h:82-232) with the block-diagonal preconditioner of
// BlockedSparseMatrix.h:1146-1361.
#include <algorithm>
#include <map>
#include <mutex>
#include <stdexcept>
#include <string>

#include "kernels.cuh"
#include "pcg_device.cuh"

namespace symxg {

namespace {

// ---- sums: float-float for the FP32 PCG's dot products, double for FP64
__device__ __forceinline__ FF sum_add(FF a, FF b) { return ff_add(a, b); }
__device__ __forceinline__ double sum_add(double a, double b) { return a + b; }
__device__ __forceinline__ FF sum_xor(FF a, int o) { return ff_shfl_xor(a, o); }
__device__ __forceinline__ double sum_xor(double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ FF product(float x, float y) { return ff_prod(x, y); }
__device__ __forceinline__ double product(double x, double y) { return x * y; }
__device__ __forceinline__ void add_prod(FF& s, float x, float y) { s = ff_add(s, ff_prod(x, y)); }
__device__ __forceinline__ void add_prod(double& s, double x, double y) { s = fma(x, y, s); }
__device__ __forceinline__ double sum_value(FF a) { return (double)a.hi + (double)a.lo; }
__device__ __forceinline__ double sum_value(double a) { return a; }
__device__ __forceinline__ unsigned long long sum_bits(FF a)
{
    return ((unsigned long long)__float_as_uint(a.hi) << 32) | __float_as_uint(a.lo);
}
__device__ __forceinline__ unsigned long long sum_bits(double a) { return (unsigned long long)__double_as_longlong(a); }
__device__ __forceinline__ void sum_from_bits(unsigned long long b, FF& a)
{
    a = FF{__uint_as_float((unsigned)(b >> 32)), __uint_as_float((unsigned)b)};
}
__device__ __forceinline__ void sum_from_bits(unsigned long long b, double& a) { a = __longlong_as_double((long long)b); }
template <typename T>
struct SumOf;
template <>
struct SumOf<float> {
    using type = FF;
    static __device__ __forceinline__ FF zero() { return FF{0.f, 0.f}; }
};
template <>
struct SumOf<double> {
    using type = double;
    static __device__ __forceinline__ double zero() { return 0.0; }
};

// ---- words that carry their own arrival
// A 16-byte word is stored and loaded as one 128-bit access and holds a tag beside its payload:
// a reader that sees the tag of the iteration it waits for has the payload too, so handing data
// to another block is one store and one poll (about 1 us on GB300), without a fence, a counter
// and a second read.
struct Word {
    unsigned long long a, b;
};
__device__ __forceinline__ void st_word(Word* p, unsigned long long a, unsigned long long b)
{
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(a), "l"(b)
                 : "memory");
}
__device__ __forceinline__ Word ld_word(const Word* p)
{
    Word w;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(w.a), "=l"(w.b)
                 : "l"(p)
                 : "memory");
    return w;
}
__device__ __forceinline__ unsigned long long pack32(unsigned lo, unsigned hi)
{
    return ((unsigned long long)hi << 32) | lo;
}

// One block row of z as tagged words: {x, y, z, tag} in float, {x, y.lo, tag} {z, y.hi, tag} in
// double.
__device__ __forceinline__ void publish_row(Word* zt, int row, const Row4<float>& z, unsigned tag)
{
    st_word(zt + row, pack32(__float_as_uint(z.x), __float_as_uint(z.y)), pack32(__float_as_uint(z.z), tag));
}
__device__ __forceinline__ void publish_row(Word* zt, int row, const Row4<double>& z, unsigned tag)
{
    const unsigned long long y = (unsigned long long)__double_as_longlong(z.y);
    st_word(zt + 2 * (int64_t)row, (unsigned long long)__double_as_longlong(z.x), pack32((unsigned)y, tag));
    st_word(zt + 2 * (int64_t)row + 1, (unsigned long long)__double_as_longlong(z.z), pack32((unsigned)(y >> 32), tag));
}
// False when the row has not arrived yet.
__device__ __forceinline__ bool read_row(const Word* zt, int row, unsigned tag, Row4<float>& z)
{
    const Word w = ld_word(zt + row);
    z = Row4<float>{__uint_as_float((unsigned)w.a), __uint_as_float((unsigned)(w.a >> 32)), __uint_as_float((unsigned)w.b),
                    0.f};
    return (unsigned)(w.b >> 32) == tag;
}
__device__ __forceinline__ bool read_row(const Word* zt, int row, unsigned tag, Row4<double>& z)
{
    const Word v = ld_word(zt + 2 * (int64_t)row), w = ld_word(zt + 2 * (int64_t)row + 1);
    z = Row4<double>{__longlong_as_double((long long)v.a),
                     __longlong_as_double((long long)pack32((unsigned)v.b, (unsigned)w.b)),
                     __longlong_as_double((long long)w.a), 0.0};
    return (unsigned)(v.b >> 32) == tag && (unsigned)(w.b >> 32) == tag;
}

// ---- grid-wide sums
// Blocks form groups of kGroup; a block publishes its sum, adds its group's in member order,
// publishes that, and adds one copy of every group's in group order (one level when the grid is
// one group).  With every block polling every other one, the polls of 152 blocks on the same
// lines made one exchange 3.0 us; 13 x 12 blocks take two hops of 1 us.  The order is fixed, so
// every block holds the same bits.
constexpr int kSums = 5;  // r.r, r.z, z.w, z.q + p.w, p.q
constexpr int kGroup = 13, kMaxGroups = 12, kGroupStride = 16;
constexpr int kMaxGrid = kGroup * kMaxGroups;
constexpr int kLevel0Words = kMaxGroups * kGroupStride, kLevel1Words = kGroup * kGroupStride;  // per sum
// Two sets, alternating: a block reuses a word two exchanges later, when every block that reads it
// has published sums of the exchange in between, hence left the earlier one.
constexpr int kSetWords = kSums * (kLevel0Words + kLevel1Words);
constexpr size_t kSumBytes = sizeof(Word) * 2 * kSetWords;
static_assert(kSumBytes <= 2 * sizeof(double) * kResidentPartials, "the exchange words fit in the partials");

// Waits are bounded: one that runs out of polls sets *abort (in shared memory).  Waits for rows that
// begin after that give up at once, and the block leaves after the exchange of that iteration, so a block
// spends at most three times the limit.  (Looking at the flag in every poll made an iteration of 9,000
// rows 0.06 us longer; once per wait costs nothing measurable.)
template <typename S>
__device__ __forceinline__ bool poll_sums(const Word* w, bool mine, unsigned long long tag, S& v, long long max_polls,
                                          volatile int* abort)
{
    for (long long polls = 0; polls < max_polls; ++polls) {
        if (mine) {
            const Word x = ld_word(w);
            if (x.b == tag) {
                sum_from_bits(x.a, v);
                mine = false;
            }
        }
        if (!__any_sync(0xffffffffu, mine)) return true;
    }
    *abort = 1;
    return false;
}
template <typename S>
__device__ __forceinline__ S sum16(S v)  // lanes 0 .. 15, the others hold zero
{
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = sum_add(v, sum_xor(v, o));
    return v;
}

// Where a block stands in the exchange (computed once: the divisions would cost more than a hop's
// arithmetic), and per lane the member whose copy of group `lane`'s sum it reads.
struct SumPlace {
    int own0, first0, members, own1, groups;
    int copy[kGroupStride];
};
__device__ __forceinline__ void sum_place(SumPlace& s)
{
    const int G = gridDim.x, b = blockIdx.x, C = G <= kGroupStride ? G : kGroup, g = b / C, m = b % C;
    s.first0 = g * kGroupStride;
    s.own0 = s.first0 + m;
    s.members = min(C, G - g * C);
    s.own1 = m * kGroupStride + g;
    s.groups = (G + C - 1) / C;
    for (int k = 0; k < s.groups; ++k) s.copy[k] = (m % min(C, G - k * C)) * kGroupStride + k;
}

// One warp: the grid's total of this block's sum v (lane 0's), valid in lane 0 unless a wait gave up.
template <typename S>
__device__ __forceinline__ void grid_sum(const SumPlace& at, Word* level0, Word* level1, unsigned long long tag, S& v,
                                         long long max_polls, volatile int* abort)
{
    const int lane = threadIdx.x & 31;
    S t;
    sum_from_bits(0, t);
    if (lane == 0) st_word(level0 + at.own0, sum_bits(v), tag);
    if (!poll_sums(level0 + at.first0 + lane, lane < at.members, tag, t, max_polls, abort)) return;
    v = sum16(t);
    if (at.groups == 1) return;
    if (lane == 0) st_word(level1 + at.own1, sum_bits(v), tag);
    sum_from_bits(0, t);
    const bool reads = lane < at.groups;
    if (poll_sums(level1 + (reads ? at.copy[lane] : 0), reads, tag, t, max_polls, abort)) v = sum16(t);
}

// Warp sums of eight values, transposing as it goes (a lane keeps half of its values and sends
// the other half): value j's total ends in lane 4 j.  Fixed order.
template <typename S>
__device__ __forceinline__ S warp_sums8(const S (&v)[8])
{
    const int lane = threadIdx.x & 31;
    S w[4], u[2];
    const bool b2 = (lane & 16) != 0, b1 = (lane & 8) != 0, b0 = (lane & 4) != 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = sum_add(b2 ? v[i + 4] : v[i], sum_xor(b2 ? v[i] : v[i + 4], 16));
#pragma unroll
    for (int i = 0; i < 2; ++i) u[i] = sum_add(b1 ? w[i + 2] : w[i], sum_xor(b1 ? w[i] : w[i + 2], 8));
    S t = sum_add(b0 ? u[1] : u[0], sum_xor(b0 ? u[0] : u[1], 4));
    t = sum_add(t, sum_xor(t, 2));
    return sum_add(t, sum_xor(t, 1));
}

// ---- the scalar recurrence.  Float: quotients of float-float sums rounded to float without an
// FP64 instruction (a double division costs about 0.4 us here: 1/64 rate and a long chain).
__device__ __forceinline__ FF ff_scale(FF a, float s)
{
    const FF p = ff_prod(a.hi, s);
    const float lo = fmaf(a.lo, s, p.lo);
    const float h = __fadd_rn(p.hi, lo);
    return FF{h, __fsub_rn(lo, __fsub_rn(h, p.hi))};
}
__device__ __forceinline__ float quotient(FF a, FF b)
{
    const float q = __fdiv_rn(a.hi, b.hi);
    const FF t = ff_scale(b, -q);
    return __fadd_rn(q, __fdiv_rn(ff_add(a, t).hi, b.hi));
}
__device__ __forceinline__ double quotient(double a, double b) { return a / b; }
__device__ __forceinline__ FF p_dot_q(FF zw, FF zq_pw, FF pq, float beta)
{
    return ff_add(zw, ff_add(ff_scale(zq_pw, beta), ff_scale(ff_scale(pq, beta), beta)));
}
__device__ __forceinline__ double p_dot_q(double zw, double zq_pw, double pq, double beta)
{
    return fma(beta, fma(beta, pq, zq_pw), zw);
}
// 2^e, within T's normal numbers
__device__ __forceinline__ void power_of_two(int e, float& x) { x = __int_as_float((127 + e) << 23); }
__device__ __forceinline__ void power_of_two(int e, double& x) { x = __hiloint2double((1023 + e) << 20, 0); }
__device__ __forceinline__ bool positive(FF a) { return a.hi > 0.f; }
__device__ __forceinline__ bool positive(double a) { return a > 0.0; }

// Product of one block row [kb, ke) with the vector xv(col), taken by a group of LPR lanes (q:
// lane within the group, 4 or 16 lanes), U blocks of the row per lane in flight; component j of
// the product ends in lane j * LPR / 4 of the group.  Every lane of the warp must call it; rows
// without blocks pass kb == ke.  Fixed order.
template <typename T, int LPR, int U, typename I, typename XV>
__device__ __forceinline__ T group_row_product(int kb, int ke, int q, const I* cols, const T* vals, int64_t stride, XV xv)
{
    T a0 = T(0), a1 = T(0), a2 = T(0);
    for (int base = kb + q; __any_sync(0xffffffffu, base < ke); base += LPR * U) {
        Row4<T> x[U];
#pragma unroll
        for (int i = 0; i < U; ++i) x[i] = base + LPR * i < ke ? xv(cols[base + LPR * i]) : Row4<T>{};
#pragma unroll
        for (int i = 0; i < U; ++i) {
            const int k = base + LPR * i;
            if (k < ke) {
                const T* m = vals + k;
                a0 += m[0] * x[i].x + m[stride] * x[i].y + m[2 * stride] * x[i].z;
                a1 += m[3 * stride] * x[i].x + m[4 * stride] * x[i].y + m[5 * stride] * x[i].z;
                a2 += m[6 * stride] * x[i].x + m[7 * stride] * x[i].y + m[8 * stride] * x[i].z;
            }
        }
    }
    // transposing sums: a lane keeps part of its components and sends the others
    if constexpr (LPR == 16) {
        const bool b8 = (q & 8) != 0, b4 = (q & 4) != 0;
        const T u0 = (b8 ? a2 : a0) + __shfl_xor_sync(0xffffffffu, b8 ? a0 : a2, 8);
        const T u1 = (b8 ? T(0) : a1) + __shfl_xor_sync(0xffffffffu, b8 ? a1 : T(0), 8);
        T v = (b4 ? u1 : u0) + __shfl_xor_sync(0xffffffffu, b4 ? u0 : u1, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 2);
        return v + __shfl_xor_sync(0xffffffffu, v, 1);
    } else {
        const bool b2 = (q & 2) != 0, b1 = (q & 1) != 0;
        const T w0 = (b2 ? a2 : a0) + __shfl_xor_sync(0xffffffffu, b2 ? a0 : a2, 2);
        const T w1 = (b2 ? T(0) : a1) + __shfl_xor_sync(0xffffffffu, b2 ? a1 : T(0), 2);
        return (b1 ? w1 : w0) + __shfl_xor_sync(0xffffffffu, b1 ? w0 : w1, 1);
    }
}

// First row of block b of G: the rows are cut so that each block gets the same share of
// blocks(row) + (mean blocks per row), so no block has more than 2 n / G + 2 rows.  One warp,
// 32-way search over row_ptr.
__device__ __forceinline__ int block_first_row(int b, int G, int n, const int32_t* __restrict__ row_ptr)
{
    const int lane = threadIdx.x & 31;
    const long long base = row_ptr[0], nnzb = row_ptr[n] - base;
    const long long target = (long long)b * (2 * nnzb * n) / G;
    int lo = 0, hi = n;
    while (lo < hi) {
        const int step = (hi - lo + 31) / 32, pos = lo + step * lane;
        const bool reached = pos >= hi || (row_ptr[pos] - base) * (long long)n + nnzb * pos >= target;
        const unsigned m = __ballot_sync(0xffffffffu, reached);
        const int first = m ? __ffs((int)m) - 1 : 32;
        if (first == 0) {
            hi = lo;
        } else {
            hi = min(hi, lo + step * first);
            lo += step * (first - 1) + 1;
        }
    }
    return lo;
}

// Per row in shared memory: x, r, z, p, q, w (3 each) and the 6 entries of Dinv.
constexpr int kStateValues = 24;

template <typename T>
constexpr int resident_threads()
{
    return sizeof(T) == 4 ? 1024 : 512;
}
constexpr int kSumWarps = kSums + 1;  // the exchange's warps (one per sum) and the convergence test's

// Block-Jacobi PCG (the reference's iteration, solve_pcg.h:82-232) for systems whose vectors fit
// in the SMs' shared memory together, and most of the matrix with them (152 x 227 KB on GB300).
//
// At these sizes (up to ~100,000 block rows) an iteration moves a few MB and takes a microsecond
// or two of arithmetic; what two launches per iteration, or two grid barriers with fences, spend
// is latency.  Us per iteration in float, before (k_pcg_solve_staged in the solver, two launches
// stand-alone) and now: 4,913 rows 13.7 / 22.9 -> 6.0, 35,937 rows 17.0 / 28.4 -> 8.8, 117,649
// rows 25.1 / 36.9 -> 17.5; double: 2,197 rows 24.8 -> 8.5, 15,625 rows 34.1 -> 15.6 (from there
// on the FP64 pipe, 2 operations per clock and SM, bounds the product).  So:
//   * each block owns a contiguous range of rows for the whole solve and keeps their matrix blocks
//     (copied once; rows that do not fit are read from L2 in every iteration), vectors and Dinv in
//     shared memory;
//   * the only vector that crosses blocks is z, in tagged words: a block polls the rows its product
//     needs (each distinct column once, listed at the start) into shared memory;
//   * one exchange of sums per iteration, after A. T. Chronopoulos and C. W. Gear ("s-step iterative
//     methods for symmetric linear systems", J. Comput. Appl. Math. 25 (1989)).  With w = A z, the sums r.r, r.z, z.w, z.q + p.w and p.q of
//     the last p and q give beta = r.z / (r.z)_old and
//         p.Ap = z.w + beta (z.q + p.w) + beta^2 p.q     for p <- z + beta p, q = A p <- w + beta q
//     without assuming any orthogonality, so the iterates are those of the two-exchange form up
//     to rounding.  q carries the rounding of its recurrence: the residual that a solve can reach
//     is a few per cent above that of q = A p formed anew (26,970 rows of 27 blocks, float 1.81e-7 of |b|
//     and 1.75e-7, double 5.04e-16 and 4.99e-16).  r.r is that of the current iterate: the convergence test runs one product
//     late, on the iterate the two-exchange form tests.
//   * no fence: a tagged word is its own release, a block's sums are published after its product,
//     hence after its reads of z, and z is overwritten only after every block's sums arrived.
//
// LPR lanes take one block row: 4 where the block's rows fill its threads, 16 for fewer or long rows
// (a shorter chain of products per lane).  zt: 4 values per row, cleared before the launch.
template <typename T, int LPR>
__global__ void __launch_bounds__(resident_threads<T>(), 1) k_pcg_resident(PcgBuffers<T> B, Word* zt, int smem_bytes)
{
    using S = typename SumOf<T>::type;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ PcgState st0;  // as the initialisation kernel left it
    __shared__ S red[kSums][32], total[kSums];
    __shared__ int cut[2], scan[33];
    __shared__ SumPlace place;
    __shared__ int b_exponent;
    __shared__ int abort_flag;  // a wait of this block ran out of polls; set at any time
    // scalars of the iteration, thread 0's but for `converged` and `gave_up` (in shared memory: the
    // other threads hold no registers for them).  They change only between the barrier of the exchange's
    // warps and the block's next barrier, so every thread leaves the loop in the same iteration.
    __shared__ struct {
        S rz, pAp;
        double thr_abs, thr_rel;
        T alpha, beta;
        int stop;       // 1: p.Ap <= 0
        int converged;  // 1: converged, 2: out of iterations
        int gave_up;    // abort_flag, as the convergence test's thread found it after the exchange
    } ctl;
    const int tid = threadIdx.x, threads = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int G = gridDim.x, n = B.n_blocks;
    if (tid == 96) {  // a warp of its own: the first three do what follows at the same time
        st0 = *B.state;
        // The solve runs on b / 2^k, exactly, with |b| / 2^k about 2^20: the sums over all rows, in float's
        // range for float, then do not overflow for any b that its type holds, and r.r can fall by 2^-180
        // (tolerances of 1e-27) before it vanishes.
        constexpr int limit = sizeof(T) == 4 ? 126 : 1000;
        b_exponent = st0.bb > 0.0 && st0.bb < (double)INFINITY ? min(max(ilogb(st0.bb) / 2 - 20, -limit), limit) : 0;
        st0.bb = scalbn(st0.bb, -2 * b_exponent);
    }
    if (tid == 64) sum_place(place);
    if (warp < 2) {
        const int r = block_first_row(blockIdx.x + warp, G, n, B.row_ptr);
        if (lane == 0) cut[warp] = r;
    }
    __syncthreads();
    if (st0.done) return;
    const int row0 = cut[0], rows = cut[1] - cut[0], R = (rows + 3) & ~3;
    T* sx = reinterpret_cast<T*>(smem);
    T* sr = sx + 3 * R;
    T* sz = sr + 3 * R;
    T* sp = sz + 3 * R;
    T* sq = sp + 3 * R;
    T* sw = sq + 3 * R;
    T* sD = sw + 3 * R;  // 00, 01, 02, 11, 12, 22
    int* rp = reinterpret_cast<int*>(sD + 6 * R);
    int used = (int)(sizeof(T) * kStateValues * R + sizeof(int) * (rows + 1) + 15) & ~15;

    // ---- vectors of the own rows, the first z published
    for (int i = tid; i <= rows; i += threads) rp[i] = B.row_ptr[row0 + i];
    for (int j = tid; j < 3 * R; j += threads) sx[j] = sr[j] = sz[j] = sp[j] = sq[j] = sw[j] = T(0);
    __syncthreads();
    T to_unit, from_unit;
    power_of_two(-b_exponent, to_unit);
    power_of_two(b_exponent, from_unit);
    for (int i = tid; i < rows; i += threads) {
        const int64_t g = row0 + i;
        Row4<T> r = ld4(B.r + 4 * g), z = ld4(B.z + 4 * g);
        r = Row4<T>{r.x * to_unit, r.y * to_unit, r.z * to_unit, T(0)};
        z = Row4<T>{z.x * to_unit, z.y * to_unit, z.z * to_unit, T(0)};
        publish_row(zt, row0 + i, z, 1u);
        sr[i] = r.x;
        sr[R + i] = r.y;
        sr[2 * R + i] = r.z;
        sz[i] = z.x;
        sz[R + i] = z.y;
        sz[2 * R + i] = z.z;
        const Row4<T> m0 = ld4(B.Dinv + 12 * g), m1 = ld4(B.Dinv + 12 * g + 4);
        sD[i] = m0.x;
        sD[R + i] = m0.y;
        sD[2 * R + i] = m0.z;
        sD[3 * R + i] = m1.y;
        sD[4 * R + i] = m1.z;
        sD[5 * R + i] = B.Dinv[12 * g + 10];
    }
    // ---- the distinct columns of the own rows, by a bitmap over all columns (in the tail of the
    // shared memory, which the matrix values take over afterwards)
    const int words = (n + 31) / 32;
    unsigned* bits = reinterpret_cast<unsigned*>(smem + (smem_bytes & ~15)) - 2 * words;
    int* rank0 = reinterpret_cast<int*>(bits + words);  // set bits before each word
    for (int i = tid; i < words; i += threads) bits[i] = 0u;
    __syncthreads();
    const int kb0 = rp[0], nnz = rp[rows] - kb0;
    for (int i = tid; i < nnz; i += threads) {
        const int c = B.cols[kb0 + i];
        atomicOr(&bits[c >> 5], 1u << (c & 31));
    }
    __syncthreads();
    const int per = (words + threads - 1) / threads, w_begin = min(words, tid * per), w_end = min(words, w_begin + per);
    int mine = 0;
    for (int i = w_begin; i < w_end; ++i) mine += __popc(bits[i]);
    int before = mine;  // inclusive scan over the warp, then over the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += t;
    }
    if (lane == 31) scan[warp] = before;
    __syncthreads();
    if (warp == 0) {
        const int warps = threads / 32, own = lane < warps ? scan[lane] : 0;
        int t = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
        }
        scan[lane] = t - own;
        if (lane == 31) scan[32] = t;
    }
    __syncthreads();
    const int n_halo = scan[32];  // columns to gather
    // in shared memory when the list, the gathered rows, the rows' columns and the bitmap fit and an
    // index fits in 16 bits; otherwise the product polls the rows itself
    const int halo_bytes = n_halo * (int)(sizeof(int) + sizeof(Row4<T>)) + 16;
    const int bitmap_at = (smem_bytes & ~15) - 8 * words;
    const bool halo = n_halo <= 65536 && used + (int64_t)halo_bytes + 2 * (int64_t)nnz <= bitmap_at;
    Row4<T>* hz = reinterpret_cast<Row4<T>*>(smem + used);
    int* hcol = reinterpret_cast<int*>(hz + n_halo);
    if (halo) {
        int k = scan[warp] + before - mine;
        for (int i = w_begin; i < w_end; ++i) {
            rank0[i] = k;
            for (unsigned b = bits[i]; b; b &= b - 1) hcol[k++] = 32 * i + __ffs((int)b) - 1;
        }
        used = (used + halo_bytes) & ~15;
    }
    __syncthreads();
    // ---- columns of all rows as halo indices, then the values of the leading rows that fit (over
    // the bitmap, which the translation reads)
    unsigned short* scols = reinterpret_cast<unsigned short*>(smem + used);
    if (halo) {
        for (int i = tid; i < nnz; i += threads) {
            const int c = B.cols[kb0 + i];
            scols[i] = (unsigned short)(rank0[c >> 5] + __popc(bits[c >> 5] & ((1u << (c & 31)) - 1u)));
        }
        used = (used + 2 * nnz + 15) & ~15;
    }
    __syncthreads();
    const int cap = halo ? (smem_bytes - used) / (int)(9 * sizeof(T)) & ~3 : 0;
    int n_res = 0;
    for (int i = 0; i < rows; i += threads) {
        const int j = i + tid;
        n_res += __syncthreads_count(j < rows && rp[j + 1] - kb0 <= cap);
    }
    T* svals = reinterpret_cast<T*>(smem + used);
    const int nnz_res = rp[n_res] - kb0, stride = (nnz_res + 3) & ~3;
    for (int i = tid; i < nnz_res; i += threads)
#pragma unroll
        for (int m = 0; m < 9; ++m) svals[m * stride + i] = B.vals[m * B.vals_stride + kb0 + i];
    if (tid == 0) {
        sum_from_bits(0, ctl.rz);
        sum_from_bits(0, ctl.pAp);
        // sqrt(rr / bb) < abs_tol  and  sqrt(rr / bb) / error0 < rel_tol, as comparisons of rr; rr = 0
        // passes any positive tolerance, also one whose square is below double's range
        const double least = 4.9406564584124654e-324;
        ctl.thr_abs = fmax(st0.abs_tol * st0.abs_tol * st0.bb, st0.abs_tol > 0.0 ? least : 0.0);
        ctl.thr_rel = fmax(st0.rel_tol * st0.error0 * st0.rel_tol * st0.error0 * st0.bb, st0.rel_tol > 0.0 ? least : 0.0);
        ctl.alpha = ctl.beta = T(0);
        ctl.stop = ctl.converged = ctl.gave_up = abort_flag = 0;
    }
    __syncthreads();

    const int sum_warps = min((3 * R + 31) / 32, threads / 32);
    const long long max_polls = B.staged.max_polls;
    volatile int* const abort = &abort_flag;
    int it = 0;
    for (;; ++it) {
        const unsigned tag = (unsigned)it + 1u;
        // ---- z of the gathered columns
        auto wait_row = [&](int c) {
            Row4<T> z;
            const long long limit = *abort ? 0 : max_polls;
            for (long long polls = 0; !read_row(zt, c, tag, z); ++polls)
                if (polls >= limit) {
                    *abort = 1;
                    break;
                }
            return z;
        };
        if (halo) {
            for (int i = tid; i < n_halo; i += threads) hz[i] = wait_row(hcol[i]);
            __syncthreads();
        }
        // ---- w = A z
        auto from_halo = [hz](int c) { return hz[c]; };
        constexpr int U = LPR == 4 ? 4 : 1;
        for (int i0 = 0; i0 < n_res; i0 += threads / LPR) {
            const int i = i0 + tid / LPR, q = tid % LPR;
            const bool valid = i < n_res;
            const T v = group_row_product<T, LPR, U>(valid ? rp[i] - kb0 : 0, valid ? rp[i + 1] - kb0 : 0, q, scols, svals,
                                                     stride, from_halo);
            if (valid && q % (LPR / 4) == 0 && q / (LPR / 4) < 3) sw[q / (LPR / 4) * R + i] = v;
        }
        for (int i0 = n_res; i0 < rows; i0 += threads / 16) {  // rows whose values stay in global memory
            const int i = i0 + tid / 16, q = tid % 16;
            const bool valid = i < rows;
            const int kb = valid ? rp[i] - kb0 : 0, ke = valid ? rp[i + 1] - kb0 : 0;
            const T* vals = B.vals + kb0;
            const T v = halo ? group_row_product<T, 16, 1>(kb, ke, q, scols, vals, B.vals_stride, from_halo)
                             : group_row_product<T, 16, 1>(kb, ke, q, B.cols + kb0, vals, B.vals_stride, wait_row);
            if (valid && q % 4 == 0 && q < 12) sw[q / 4 * R + i] = v;
        }
        __syncthreads();
        // ---- the sums
        if (warp < sum_warps) {
            // one component per thread; more only where the block has over threads / 3 rows (the
            // entries past the last row are zeros)
            S v[8];
#pragma unroll
            for (int k = kSums; k < 8; ++k) v[k] = SumOf<T>::zero();
            for (int j = tid; j < 3 * R || j == tid; j += threads) {
                const bool in = j < 3 * R;
                const T r = in ? sr[j] : T(0), z = in ? sz[j] : T(0), w = in ? sw[j] : T(0), p = in ? sp[j] : T(0),
                        q = in ? sq[j] : T(0);
                if (j == tid) {
                    v[0] = product(r, r);
                    v[1] = product(r, z);
                    v[2] = product(z, w);
                    v[3] = product(z, q);
                    v[4] = product(p, q);
                } else {
                    add_prod(v[0], r, r);
                    add_prod(v[1], r, z);
                    add_prod(v[2], z, w);
                    add_prod(v[3], z, q);
                    add_prod(v[4], p, q);
                }
                add_prod(v[3], p, w);
            }
            const S t = warp_sums8(v);
            if ((lane & 3) == 0 && lane < 4 * kSums) red[lane >> 2][warp] = t;
        }
        __syncthreads();
        if (warp < kSumWarps) {
            if (warp < kSums) {
                S v = SumOf<T>::zero();
                if (lane < sum_warps) v = red[warp][lane];
                if (sum_warps > 16) v = sum_add(v, sum_xor(v, 16));
                if (sum_warps > 8) v = sum_add(v, sum_xor(v, 8));
                if (sum_warps > 4) v = sum_add(v, sum_xor(v, 4));
                if (sum_warps > 2) v = sum_add(v, sum_xor(v, 2));
                if (sum_warps > 1) v = sum_add(v, sum_xor(v, 1));
                Word* level0 = reinterpret_cast<Word*>(B.partials) + (it & 1) * kSetWords;
                Word* level1 = level0 + kSums * kLevel0Words;
                grid_sum(place, level0 + warp * kLevel0Words, level1 + warp * kLevel1Words, tag, v, max_polls, abort);
                if (lane == 0) total[warp] = v;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kSumWarps) : "memory");
            if (tid == 0) {
                const T beta = it > 0 ? quotient(total[1], ctl.rz) : T(0);
                const S pAp = p_dot_q(total[2], total[3], total[4], beta);
                ctl.beta = beta;
                ctl.rz = total[1];
                ctl.pAp = pAp;
                if (positive(pAp)) ctl.alpha = quotient(total[1], pAp);
                else ctl.stop = 1;  // indefinite (or NaN): stop as the reference does
            }
            if (tid == 32 * kSums) {
                ctl.gave_up = *abort;
                const double rr = sum_value(total[0]);
                if (it > 0 && (rr < ctl.thr_abs || rr < ctl.thr_rel)) ctl.converged = 1;
                else if (it > 0 && it >= st0.max_iterations) ctl.converged = 2;
            }
        }
        __syncthreads();
        if (ctl.gave_up | ctl.converged | ctl.stop) break;
        // ---- p, q, x, r, z
        const T alpha = ctl.alpha, beta = ctl.beta;
        if constexpr (sizeof(T) == 4) {  // a thread per row
            for (int i = tid; i < rows; i += threads) {
                T r[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const T p = fma(beta, sp[d * R + i], sz[d * R + i]), q = fma(beta, sq[d * R + i], sw[d * R + i]);
                    sp[d * R + i] = p;
                    sq[d * R + i] = q;
                    sx[d * R + i] = fma(alpha, p, sx[d * R + i]);
                    sr[d * R + i] = r[d] = fma(-alpha, q, sr[d * R + i]);
                }
                const T d01 = sD[R + i], d02 = sD[2 * R + i], d12 = sD[4 * R + i];
                const Row4<T> z{sD[i] * r[0] + d01 * r[1] + d02 * r[2], d01 * r[0] + sD[3 * R + i] * r[1] + d12 * r[2],
                                d02 * r[0] + d12 * r[1] + sD[5 * R + i] * r[2], T(0)};
                publish_row(zt, row0 + i, z, tag + 1u);
                sz[i] = z.x;
                sz[R + i] = z.y;
                sz[2 * R + i] = z.z;
            }
        } else {  // three times the chain of FP64 instructions on a third of the warps: spread it
            for (int i0 = 0; i0 < rows; i0 += threads / 4) {  // a quad per row, lane d: component d
                const int i = i0 + tid / 4, d = tid & 3, j = d * R + i, quad = lane & ~3;
                const bool own = i < rows && d < 3;
                T r = T(0);
                if (own) {
                    const T p = fma(beta, sp[j], sz[j]), q = fma(beta, sq[j], sw[j]);
                    sp[j] = p;
                    sq[j] = q;
                    sx[j] = fma(alpha, p, sx[j]);
                    sr[j] = r = fma(-alpha, q, sr[j]);
                }
                const T r0 = __shfl_sync(0xffffffffu, r, quad), r1 = __shfl_sync(0xffffffffu, r, quad + 1),
                        r2 = __shfl_sync(0xffffffffu, r, quad + 2);
                T z = T(0);
                if (own)  // row d of Dinv from its upper triangle
                    sz[j] = z = sD[d * R + i] * r0 + sD[(d == 0 ? 1 : d + 2) * R + i] * r1 +
                                sD[(d == 0 ? 2 : d + 3) * R + i] * r2;
                const T z0 = __shfl_sync(0xffffffffu, z, quad), z1 = __shfl_sync(0xffffffffu, z, quad + 1),
                        z2 = __shfl_sync(0xffffffffu, z, quad + 2);
                if (own && d == 0) publish_row(zt, row0 + i, Row4<T>{z0, z1, z2, T(0)}, tag + 1u);
            }
        }
        if (!halo) __syncthreads();  // the next product writes w
    }
    for (int i = tid; i < rows; i += threads)
        st4(B.x + 4 * (int64_t)(row0 + i), Row4<T>{sx[i] * from_unit, sx[R + i] * from_unit, sx[2 * R + i] * from_unit, T(0)});
    if (ctl.gave_up) {
        if (tid == 0) atomicExch(&B.state->wait_failed, 1);
        return;
    }
    if (blockIdx.x == 0 && tid == 0) {
        PcgState* st = B.state;
        const bool indefinite = !ctl.converged && ctl.stop;
        st->iteration = indefinite ? it + 1 : it;
        st->converged = ctl.converged == 1;
        st->indefinite = indefinite;
        st->done = 1;
        st->pAp = scalbn(sum_value(ctl.pAp), 2 * b_exponent);
        st->alpha = ctl.alpha;
        st->beta = ctl.beta;
        st->rz = scalbn(sum_value(ctl.rz), 2 * b_exponent);
        st->rr = scalbn(sum_value(total[0]), 2 * b_exponent);
        st->error = it > 0 ? sqrt(sum_value(total[0]) / st0.bb) : st0.error;
    }
}

// SM count, shared memory per block and L2 of the current device (looked up once per device).
struct DeviceLimits {
    int sms = 0, smem = 0, l2 = 0;
};
template <typename K>
void allow_smem(K kernel, int bytes)
{
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess)
        throw std::runtime_error(std::string("symx_gb300: resident PCG shared memory: ") + cudaGetErrorString(e));
}
DeviceLimits device_limits()
{
    static std::mutex m;
    static std::map<int, DeviceLimits> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(m);
    auto it = cache.find(dev);
    if (it != cache.end()) return it->second;
    DeviceLimits d;
    int coop = 0, optin = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (coop) {
        cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        cudaDeviceGetAttribute(&d.l2, cudaDevAttrL2CacheSize, dev);
        d.smem = (optin - 4096) & ~15;  // less the kernel's static shared memory
        allow_smem(k_pcg_resident<float, 4>, d.smem);
        allow_smem(k_pcg_resident<float, 16>, d.smem);
        allow_smem(k_pcg_resident<double, 4>, d.smem);
        allow_smem(k_pcg_resident<double, 16>, d.smem);
    }
    cache[dev] = d;
    return d;
}

}  // namespace

// Every system whose state and bitmap fit is taken (on GB300 up to about 145,200 rows in float and 80,100
// in double) while its values, as far as shared memory does not hold them, come from L2 or from HBM
// faster here than in the kernels that stream them with more loads in flight.  Where that ends, by
// bytes of all values:
//   * float solver (staged kernel; two launches for Tet10, whose rows are too long for its ring), 13/16 of
//     L2 (110 of 135.5 MB).  Us per iteration, those -> this: Tet4 76 MB 28.4 -> 19.4, Tet10 103 MB
//     62.1 -> 54.0, 108 MB 62.1 -> 60.2, 112.5 MB 64.0 -> 67.1, 127 MB 73 -> 78; Hex8 105 MB
//     34.4 -> 29.1, 110 MB 34.9 -> 33.5, 112 MB 36.8 -> 36.2, 114 MB 36.7 -> 38.1, 127 MB 38.6 -> 55.2.
//   * Two launches otherwise; ms of 30 iterations.  Rows of uneven lengths (the longest above 5/4 of the
//     mean: blocks finish apart), float 13/16 of L2: random 89 MB 1.12 -> 1.06, 117 MB 1.51 -> 1.40, 126 MB
//     1.53 -> 1.58, 132 MB 1.44 -> 1.59.  Double 7/4 (237 MB): Tet10 158 MB 4.35 -> 4.12, random 233 MB
//     3.28 -> 3.11, 347 MB 4.06 -> 4.14.
//   * Even rows, float 15/8 (254 MB): 129 MB 2.39 -> 2.06, 243 MB 3.75 -> 3.14, 251 MB 3.75 -> 3.76, 321 MB
//     4.21 -> 4.91.  Double 10 times L2: 642 MB 9.54 -> 8.89, 1280 MB 18.4 -> 17.7, 1696 MB 22.8 -> 23.7.
template <typename T>
bool plan_pcg_resident(int n_blocks, int64_t nnzb, ResidentRows row_lengths, ResidentPlan& plan)
{
    plan = ResidentPlan{};
    if (n_blocks <= 0 || nnzb <= 0) return false;
    const DeviceLimits d = device_limits();
    if (d.sms <= 0) return false;
    constexpr int64_t uneven16 = sizeof(T) == 4 ? 13 : 28, even16 = sizeof(T) == 4 ? 30 : 160;  // sixteenths of L2
    if (9 * (int64_t)sizeof(T) * nnzb > d.l2 / 16 * (row_lengths == ResidentRows::even ? even16 : uneven16)) return false;
    constexpr int max_threads = resident_threads<T>();
    // at least sixteen rows per block: fewer would only add sums to wait for (1,000 rows in double:
    // 7.4 us per iteration on 63, 76 or 125 blocks)
    const int64_t grid = std::min<int64_t>(std::min(d.sms, kMaxGrid), ((int64_t)n_blocks + 15) / 16);
    const int64_t rows = ((int64_t)n_blocks + grid - 1) / grid;
    // no block has more rows than 2 n / grid + 2 (block_first_row), rounded up to four in the kernel
    const int64_t rows_max = (2 * (int64_t)n_blocks / grid + 2 + 3) & ~(int64_t)3;
    const int64_t state = rows_max * (kStateValues * (int64_t)sizeof(T) + 4) + 64;
    const int64_t bitmap = ((int64_t)n_blocks + 31) / 32 * 8;
    if (state + bitmap + 64 > d.smem) return false;
    plan.grid = (int)grid;
    // rows of 80 blocks and more keep 16 lanes busy however many there are (double, ms of 30 iterations with
    // 4 lanes -> 16: 8,000 rows of 262 blocks 4.29 -> 3.09, of 104 1.46 -> 1.23, of 64 1.01 -> 1.05)
    plan.lanes_per_row = rows * 16 <= max_threads || nnzb >= 80 * (int64_t)n_blocks ? 16 : 4;
    // room for a quarter more rows than the mean: blocks at the mesh's boundary have more, shorter
    // rows, and a second round of the product for a few of them would hold up every block
    const int64_t lanes = (rows + rows / 4) * plan.lanes_per_row;
    plan.threads = (int)std::min<int64_t>(max_threads, std::max<int64_t>(256, (lanes + 31) / 32 * 32));
    plan.smem_bytes = d.smem;
    return true;
}

template <typename T>
void launch_pcg_resident(const PcgBuffers<T>& B, const ResidentPlan& plan, cudaStream_t s)
{
    // words that no tag matches: the sums' and, in the second direction buffer, z's
    cudaError_t e = cudaMemsetAsync(B.partials, 0, kSumBytes, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(B.p2, 0, 4 * sizeof(T) * (size_t)B.n_blocks, s);
    if (e != cudaSuccess) throw std::runtime_error(std::string("symx_gb300: memset: ") + cudaGetErrorString(e));
    PcgBuffers<T> arg = B;
    arg.staged.max_polls = wait_poll_limit();
    Word* zt = reinterpret_cast<Word*>(B.p2);
    int smem = plan.smem_bytes;
    void* args[] = {&arg, &zt, &smem};
    const void* fn = plan.lanes_per_row == 4 ? (const void*)k_pcg_resident<T, 4> : (const void*)k_pcg_resident<T, 16>;
    const cudaError_t l = cudaLaunchCooperativeKernel(fn, dim3(plan.grid), dim3(plan.threads), args, (size_t)smem, s);
    if (l != cudaSuccess)
        throw std::runtime_error(std::string("symx_gb300: cooperative launch of the resident PCG failed: ") +
                                 cudaGetErrorString(l));
    count_launch();
}

template bool plan_pcg_resident<float>(int, int64_t, ResidentRows, ResidentPlan&);
template bool plan_pcg_resident<double>(int, int64_t, ResidentRows, ResidentPlan&);
template void launch_pcg_resident<float>(const PcgBuffers<float>&, const ResidentPlan&, cudaStream_t);
template void launch_pcg_resident<double>(const PcgBuffers<double>&, const ResidentPlan&, cudaStream_t);

}  // namespace symxg
