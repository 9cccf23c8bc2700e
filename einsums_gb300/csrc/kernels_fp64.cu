// Plain FP64 kernels of the canonical contraction
//   C[b,m,n] = cp*C + ab * sum_k A[b,m,k] B[b,n,k]
// with every operand addressed through folded index maps, so permuted and
// strided operands are read in place (nothing is materialised).
//
//   k_elementwise   no summed modes: DIRECT / GER / broadcasts
//                   (replaces hipBLASVendor/src/direct_prod.hip:20-200, ger, and
//                    GPUTensorAlgebra.hpp:87-140)
//   k_dot_*         rank-0 C: deterministic reduction, no atomics, in one CTA for
//                   short sums, else in two passes
//                   (replaces GPULinearAlgebra.hpp:35-101 and GPUTensorAlgebra.hpp:146-198)
//   k_gemv          one of the M/N groups empty: one CTA or warp per output
//                   (replaces hipblasDgemv at GPULinearAlgebra.hpp:346-386)
//   k_contract_f64  general case: small-tile DFMA contraction, K cut over a cluster
//                   when the output has fewer tiles than the GPU has SMs
//                   (replaces hipblasDgemm_64 and the atomicAdd generic kernel
//                    GPUTensorAlgebra.hpp:28-82)
#include <algorithm>
#include <cmath>
#include <utility>

#include "common.cuh"
#include "f64_tile.cuh"
#include "ptx.cuh"

namespace eg {

int64_t mode_group_affine_stride(const ModeGroup &g, int comp);

namespace {

__device__ __forceinline__ double epilogue(double acc, double *cptr, double cp, double ab, bool zero) {
    const double v = ab * acc;
    if (zero && cp == 0.0) return v;
    return cp * (*cptr) + v;
}

// ----------------------------------------------------------- elementwise --
// One mode of stride 1 in all three (a DIRECT product of like-ordered tensors): pairs of
// 16 bytes, two pairs of a thread in flight.  Bound: memory, 24 bytes per element (32
// with C_prefactor), if the FP64 pipe is spared -- three operations an element took as
// long: a multiplication by ab = 1 and the sum with C are left out where they do nothing.
// 15e6 elements: 69 us (5.3 TB/s); mode by mode 81 us.  One element off alignment, or
// with a mode between, the kernel below takes it.
template <bool PLAIN, bool AB_ONE>
__global__ void __launch_bounds__(256) k_elementwise_contiguous(int64_t n, const double *__restrict__ A,
                                                                const double *__restrict__ B, double *C, double cp,
                                                                double ab) {
    auto one = [&](double a, double b, double c) {
        const double v = AB_ONE ? a * b : ab * (a * b);
        return PLAIN ? v : fma(cp, c, v);
    };
    const int64_t pairs = n / 2, stride = (int64_t)gridDim.x * blockDim.x;
    const double2 *A2 = (const double2 *)A, *B2 = (const double2 *)B;
    double2 *C2 = (double2 *)C;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < pairs; i += 2 * stride) {
        const int64_t j = i + stride;
        const bool two = j < pairs;
        const double2 a0 = __ldg(A2 + i), b0 = __ldg(B2 + i);
        const double2 a1 = two ? __ldg(A2 + j) : a0, b1 = two ? __ldg(B2 + j) : b0;
        double2 c0 = {0.0, 0.0}, c1 = {0.0, 0.0};
        if (!PLAIN) {
            c0 = C2[i];
            if (two) c1 = C2[j];
        }
        C2[i] = make_double2(one(a0.x, b0.x, c0.x), one(a0.y, b0.y, c0.y));
        if (two) C2[j] = make_double2(one(a1.x, b1.x, c1.x), one(a1.y, b1.y, c1.y));
    }
    if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) C[n - 1] = one(A[n - 1], B[n - 1], PLAIN ? 0.0 : C[n - 1]);
}

template <bool Wide>
__global__ void k_elementwise(ModeGroup g, const double *__restrict__ A, const double *__restrict__ B, double *C,
                              double cp, double ab, bool zero) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.total; i += stride) {
        int64_t oa, ob, oc;
        if (Wide)
            group_offsets(g, i, oa, ob, oc);
        else
            group_offsets32(g, (uint32_t)i, oa, ob, oc);
        C[oc] = epilogue(A[oa] * B[ob], C + oc, cp, ab, zero);
    }
}

// C = cp*C over every element of C (or C = 0 when cp == 0), walking C's own
// modes; the prologue the reference applies to the whole output before a
// generic contraction (BaseAlgebra.hpp:129-133), needed when C has repeated
// labels and the contraction itself visits only its diagonal.
template <bool Wide>
__global__ void k_scale(ModeGroup g, double *C, double cp) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.total; i += stride) {
        int64_t oa, ob, oc;
        if (Wide)
            group_offsets(g, i, oa, ob, oc);
        else
            group_offsets32(g, (uint32_t)i, oa, ob, oc);
        C[oc] = cp == 0.0 ? 0.0 : cp * C[oc];
    }
}

// ------------------------------------------------------ block reductions --
template <int THREADS>
__device__ __forceinline__ double block_sum(double v, double *smem) {
    // Fixed shuffle tree, then the warp sums in warp order: deterministic.
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    constexpr int W = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (W == 1) return v;
    __syncthreads();
    if (lane == 0) smem[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (warp == 0) {
        t = lane < W ? smem[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    return t; // valid in warp 0
}

// -------------------------------------------------------------------- dot --
// Four blocks per SM: the compensated sum over blocks, serial FP64 work on one SM, took
// 6 us of 54 with twice as many partials and threads.
constexpr int kDotThreads = 256, kDotBlocksPerSm = 4, kDotFinalThreads = 128;

template <bool Contig>
__global__ void __launch_bounds__(kDotThreads) k_dot_partial(ModeGroup k, const double *__restrict__ A,
                                                             const double *__restrict__ B, double *partial,
                                                             int64_t chunk) {
    __shared__ double smem[32];
    const int64_t begin = (int64_t)blockIdx.x * chunk;
    const int64_t end = min(begin + chunk, k.total);
    double acc0 = 0.0, acc1 = 0.0;
    if (Contig) {
        // 16-byte pairs where both operands allow (chunks are even), four pairs of each in
        // flight: 15e6 elements with the final sum 50 us, element by element 69 us
        int64_t i = begin + threadIdx.x;
        if ((((uintptr_t)A | (uintptr_t)B) & 15) == 0) {
            const double2 *A2 = (const double2 *)(A + begin), *B2 = (const double2 *)(B + begin);
            const int64_t pairs = (end - begin) / 2;
            double acc[4] = {};
            int64_t j = threadIdx.x;
            for (; j + 3 * kDotThreads < pairs; j += 4 * kDotThreads) {
                double2 x[4], y[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    x[q] = __ldg(A2 + j + q * kDotThreads);
                    y[q] = __ldg(B2 + j + q * kDotThreads);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) acc[q] = fma(x[q].y, y[q].y, fma(x[q].x, y[q].x, acc[q]));
            }
            for (; j < pairs; j += kDotThreads) {
                const double2 x = __ldg(A2 + j), y = __ldg(B2 + j);
                acc[0] = fma(x.y, y.y, fma(x.x, y.x, acc[0]));
            }
            acc0 = acc[0] + acc[1];
            acc1 = acc[2] + acc[3];
            i = begin + 2 * pairs + threadIdx.x; // the odd last element
        }
        for (; i + kDotThreads < end; i += 2 * kDotThreads) {
            acc0 = fma(__ldg(A + i), __ldg(B + i), acc0);
            acc1 = fma(__ldg(A + i + kDotThreads), __ldg(B + i + kDotThreads), acc1);
        }
        if (i < end) acc0 = fma(__ldg(A + i), __ldg(B + i), acc0);
    } else {
        for (int64_t i = begin + threadIdx.x; i < end; i += kDotThreads) {
            int64_t oa, ob, oc;
            group_offsets(k, i, oa, ob, oc);
            acc0 = fma(__ldg(A + oa), __ldg(B + ob), acc0);
        }
    }
    const double s = block_sum<kDotThreads>(acc0 + acc1, smem);
    if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// A short sum in one CTA and one launch: up to kDotSmall elements, eight of a thread in
// flight, each in a sum of its own: at most 4 + 3 + 9 additions lie on a path, against
// 8 + 1 + 8 before the compensated sum over blocks of the two launches of longer sums.
// Bound: latency.  10^4 elements: 6.2 us (10.0 us in two launches); above kDotSmall the
// CTA's one SM takes longer than a second launch.
constexpr int64_t kDotSmall = 16384;
constexpr int kDotSmallThreads = 512;
template <bool Contig>
__global__ void __launch_bounds__(kDotSmallThreads) k_dot_small(ModeGroup k, const double *__restrict__ A,
                                                                const double *__restrict__ B, double *C, double cp,
                                                                double ab, bool zero) {
    __shared__ double smem[32];
    constexpr int Q = 8;
    const int n = (int)k.total;
    double acc[Q] = {};
    for (int i = threadIdx.x; i < n; i += Q * kDotSmallThreads) {
        double x[Q], y[Q];
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int e = i + q * kDotSmallThreads;
            int64_t oa = e, ob = e, oc;
            if (!Contig && e < n) group_offsets32(k, (uint32_t)e, oa, ob, oc);
            x[q] = e < n ? __ldg(A + oa) : 0.0;
            y[q] = e < n ? __ldg(B + ob) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < Q; q++)
            if (i + q * kDotSmallThreads < n) acc[q] = fma(x[q], y[q], acc[q]);
    }
    const double mine = ((acc[0] + acc[1]) + (acc[2] + acc[3])) + ((acc[4] + acc[5]) + (acc[6] + acc[7]));
    const double sum = block_sum<kDotSmallThreads>(mine, smem);
    if (threadIdx.x == 0) *C = epilogue(sum, C, cp, ab, zero);
}

// Sums the per-block partials in a fixed order: Neumaier compensation within a
// thread, then a compensated tree across the block.
__global__ void __launch_bounds__(kDotFinalThreads) k_dot_final(const double *partial, int nparts, double *C, double cp,
                                                           double ab, bool zero) {
    __shared__ double sh_s[kDotFinalThreads / 32], sh_c[kDotFinalThreads / 32];
    double s = 0.0, c = 0.0;
    for (int i = threadIdx.x; i < nparts; i += kDotFinalThreads) {
        const double x = partial[i];
        const double t = s + x;
        c += (fabs(s) >= fabs(x)) ? (s - t) + x : (x - t) + s;
        s = t;
    }
    const double sum = block_sum_compensated<kDotFinalThreads>(s, c, sh_s, sh_c);
    if (threadIdx.x == 0) *C = epilogue(sum, C, cp, ab, zero);
}

// ------------------------------------------------------------------- gemv --
// Output positions are walked through `rows` (batch and the non-empty M or N
// group, offsets in A/B/C); every output sums over `k`.
// KContig: k is one mode of stride 1 in A and B.  Otherwise the offsets of
// every k in A and B come from tables (offk[0..K) for A, offk[K..2K) for B),
// or, when offk is null, from the mode decomposition.  Four independent
// accumulators keep four loads of each operand in flight per thread.
template <int TPR, bool KContig>
__global__ void __launch_bounds__(256) k_gemv(ModeGroup rows, ModeGroup k, const double *__restrict__ A,
                                              const double *__restrict__ B, double *C, double cp, double ab,
                                              bool zero, const int64_t *__restrict__ offk) {
    __shared__ double smem[32];
    constexpr int RPB = 256 / TPR; // rows per block
    const int sub = threadIdx.x / TPR, lane = threadIdx.x % TPR;
    const int64_t K = k.total;
    for (int64_t r = (int64_t)blockIdx.x * RPB + sub; r < rows.total; r += (int64_t)gridDim.x * RPB) {
        int64_t ra, rb, rc;
        group_offsets(rows, r, ra, rb, rc);
        const double *a = A + ra;
        const double *b = B + rb;
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
        int64_t i = lane;
        if (KContig && ((((uintptr_t)a) | ((uintptr_t)b)) & 15) == 0) {
            // 16-byte pairs: eight values of each operand in flight per thread
            const double2 *a2 = (const double2 *)a, *b2 = (const double2 *)b;
            const int64_t K2 = K / 2;
            int64_t j = lane;
            for (; j + 3 * TPR < K2; j += 4 * TPR) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const double2 x = __ldg(a2 + j + u * TPR), y = __ldg(b2 + j + u * TPR);
                    acc[u] = fma(x.x, y.x, acc[u]);
                    acc[u] = fma(x.y, y.y, acc[u]);
                }
            }
            for (; j < K2; j += TPR) {
                const double2 x = __ldg(a2 + j), y = __ldg(b2 + j);
                acc[0] = fma(x.x, y.x, acc[0]);
                acc[0] = fma(x.y, y.y, acc[0]);
            }
            if ((K & 1) && lane == 0) acc[1] = fma(__ldg(a + K - 1), __ldg(b + K - 1), acc[1]);
        } else if (KContig) {
            for (; i + 3 * TPR < K; i += 4 * TPR) {
#pragma unroll
                for (int u = 0; u < 4; u++) acc[u] = fma(__ldg(a + i + u * TPR), __ldg(b + i + u * TPR), acc[u]);
            }
            for (; i < K; i += TPR) acc[0] = fma(__ldg(a + i), __ldg(b + i), acc[0]);
        } else if (offk) {
            for (; i + 3 * TPR < K; i += 4 * TPR) {
#pragma unroll
                for (int u = 0; u < 4; u++)
                    acc[u] = fma(__ldg(a + __ldg(offk + i + u * TPR)), __ldg(b + __ldg(offk + K + i + u * TPR)), acc[u]);
            }
            for (; i < K; i += TPR) acc[0] = fma(__ldg(a + __ldg(offk + i)), __ldg(b + __ldg(offk + K + i)), acc[0]);
        } else {
            for (; i < K; i += TPR) {
                int64_t oa, ob, oc;
                group_offsets32(k, (uint32_t)i, oa, ob, oc);
                acc[0] = fma(__ldg(a + oa), __ldg(b + ob), acc[0]);
            }
        }
        double s = (acc[0] + acc[1]) + (acc[2] + acc[3]);
        if (TPR == 32) {
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        } else {
            s = block_sum<TPR>(s, smem);
        }
        if (lane == 0) C[rc] = epilogue(s, C + rc, cp, ab, zero);
        if (TPR != 32) __syncthreads();
    }
}

// Adds RB values of each lane over the warp: lane q < RB (spread over the lanes: the
// bits of a lane above the lowest log2(32 / RB)) ends up with the sum of value q.  Each
// step halves the values a lane holds, so four sums take 6 additions a lane, not 20 (the
// FP64 pipe bounds the kernel below).
template <int RB>
__device__ __forceinline__ double warp_sums(double (&v)[RB], int lane, int &which) {
    which = 0;
    int o = 16;
#pragma unroll
    for (int n = RB; n > 1; n /= 2, o /= 2) {
        const bool up = lane & o;
#pragma unroll
        for (int q = 0; q < n / 2; q++) {
            const double keep = up ? v[q + n / 2] : v[q], give = up ? v[q] : v[q + n / 2];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
        which = 2 * which + (up ? 1 : 0);
    }
    for (; o > 0; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

// Long k: one CTA takes RB outputs at a time, each k of B (the vector, shared
// by every output) is loaded once and used for RB rows of A, so the vector's L1 traffic
// is divided by RB.  Bound: the FP64 pipe at two FMAs per clock per SM, 8 bytes of A
// each (5 TB/s), ahead of memory.  10^4 rows of 10^4: one run 188 us, nested runs 203 us
// (208 us with a tree per row, 227 us with offset tables).  FORM 0: k is one mode of stride 1 in A and B, with
// 16-byte pairs when aligned; 1: two modes, the inner of stride 1 in both, walked by a
// running index (r, s) per thread; 2: offk[0..K) / offk[K..2K) hold the offsets of every
// k in A and B.
template <int RB, int FORM>
__global__ void __launch_bounds__(256) k_gemv_rows(ModeGroup rows, ModeGroup k, const double *__restrict__ A,
                                                   const double *__restrict__ B, double *C, double cp, double ab,
                                                   bool zero, const int64_t *__restrict__ offk) {
    __shared__ double red[8][RB];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t K = k.total;
    for (int64_t r0 = (int64_t)blockIdx.x * RB; r0 < rows.total; r0 += (int64_t)gridDim.x * RB) {
        const double *a[RB];
        const double *b = B;
        bool aligned = true;
#pragma unroll
        for (int q = 0; q < RB; q++) {
            const int64_t r = r0 + q < rows.total ? r0 + q : rows.total - 1; // tail rows repeat the last one
            int64_t ra, rb, oc;
            group_offsets(rows, r, ra, rb, oc);
            a[q] = A + ra;
            b = B + rb; // the same for every row: the rows run over A's modes only
            aligned &= (((uintptr_t)a[q]) & 15) == 0;
        }
        aligned &= (((uintptr_t)b) & 15) == 0;
        double acc[RB];
#pragma unroll
        for (int q = 0; q < RB; q++) acc[q] = 0.0;
        auto pair = [&](int64_t oa, int64_t ob) {
            const double2 y = __ldg((const double2 *)(b + ob));
            double2 x[RB];
#pragma unroll
            for (int q = 0; q < RB; q++) x[q] = __ldg((const double2 *)(a[q] + oa));
#pragma unroll
            for (int q = 0; q < RB; q++) acc[q] = fma(x[q].y, y.y, fma(x[q].x, y.x, acc[q]));
        };
        auto single = [&](int64_t oa, int64_t ob) {
            const double y = __ldg(b + ob);
#pragma unroll
            for (int q = 0; q < RB; q++) acc[q] = fma(__ldg(a[q] + oa), y, acc[q]);
        };
        if (FORM == 0 && aligned) {
            const int64_t K2 = K / 2;
            // CTAs start at different points of k so that concurrently read rows
            // (a fixed stride apart) do not hit the same memory channels in step
            const int64_t start = K2 > 4096 ? ((r0 / RB) * 1031 % (K2 / 256)) * 256 : 0;
#pragma unroll 2
            for (int64_t j = start + tid; j < K2; j += 256) pair(2 * j, 2 * j);
#pragma unroll 2
            for (int64_t j = tid; j < start; j += 256) pair(2 * j, 2 * j);
            if ((K & 1) && tid == 0) single(K - 1, K - 1);
        } else if (FORM == 0) {
#pragma unroll 2
            for (int64_t i = tid; i < K; i += 256) single(i, i);
        } else if (FORM == 1) {
            // the inner mode's pairs are aligned when its extent and all other strides are even
            const int64_t sa = k.s[0][0], sb = k.s[1][0];
            const bool pairs = aligned && k.ext[1] % 2 == 0 && sa % 2 == 0 && sb % 2 == 0;
            const int w = pairs ? 2 : 1;
            const uint32_t inner = (uint32_t)(k.ext[1] / w), n = (uint32_t)(K / w);
            const uint32_t dr = 256u / inner, ds = 256u - dr * inner;
            uint32_t r = (uint32_t)tid / inner, s = (uint32_t)tid - r * inner;
            int64_t oa = (int64_t)r * sa, ob = (int64_t)r * sb;
            auto walk = [&](auto &&use) {
#pragma unroll 2
                for (uint32_t i = tid; i < n; i += 256) {
                    use(oa + w * (int64_t)s, ob + w * (int64_t)s);
                    s += ds;
                    const uint32_t step = dr + (s >= inner ? 1u : 0u);
                    s -= s >= inner ? inner : 0u;
                    oa += (int64_t)step * sa;
                    ob += (int64_t)step * sb;
                }
            };
            if (pairs)
                walk(pair);
            else
                walk(single);
        } else {
            for (int64_t i = tid; i < K; i += 256) single(__ldg(offk + i), __ldg(offk + K + i));
        }
        // fixed-order reduction: warp trees, then the warps in order
        int which;
        const double v = warp_sums<RB>(acc, lane, which);
        if ((lane & (32 / RB - 1)) == 0) red[warp][which] = v;
        __syncthreads();
        if (tid < RB && r0 + tid < rows.total) {
            double t = 0.0;
            for (int w = 0; w < 8; w++) t += red[w][tid];
            int64_t ra, rb, oc;
            group_offsets(rows, r0 + tid, ra, rb, oc);
            C[oc] = epilogue(t, C + oc, cp, ab, zero);
        }
        __syncthreads();
    }
}

// Offsets of every k of a mode group in A (out[0..K)) and in B (out[K..2K)).
__global__ void k_k_offsets(ModeGroup k, int64_t *out) {
    const int64_t K = k.total;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < K; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t oa, ob, oc;
        group_offsets32(k, (uint32_t)i, oa, ob, oc);
        out[i] = oa;
        out[K + i] = ob;
    }
}

// ------------------------------------------------------ tiled contraction --
// Bound: the FP64 pipe, which retires two FMAs per clock per SM, so a 64-bit
// FMA of a warp takes 16 clocks of an SM while its two shared-memory reads take
// four: register tiles buy nothing, and what counts is that every SM has its
// share of the FMAs.  Tiles are therefore small (8, 16 or 32 square, picked by
// contract_plan), and when there are still fewer tiles than SMs a cluster of up
// to eight CTAs cuts K, its partial sums added over distributed shared memory
// in rank order (deterministic, no workspace, so the launch can be captured).
// 256 threads: KG groups along k times T*T outputs, R x R outputs per thread.
// Chunks of BK k come through a three-slot ring of 8-byte asynchronous copies
// (zero-filled past the edges), two chunks ahead of the FMAs.
// Measured against 64 x 64 tiles without a K cut: 40x60x50 92 -> 26 us a call
// (the call's host side), complex 300x170x257 (four launches) 1404 -> 156 us,
// 144x2304x2304 2.93 -> 1.31 ms, 2304^3 21.7 -> 20.1 ms (1.22 TFLOP/s, 97 % of
// the pipe).
using f64::kThreads;

struct F64Args {
    ModeGroup bg, mg, ng, kg;
    const double *A, *B;
    double *C;
    double cp, ab;
    int zero;
    int a_kfast, b_kfast;  // the operand is read along k (its smaller stride), else along its rows
    int64_t ka, kb;        // single k strides of A and B (0: none)
    int64_t mtiles, ntiles, total; // total = batches * mtiles * ntiles
    int cs;                // CTAs of a cluster, each taking a range of the k chunks
    // When set, the tiles are instead the parts of the blocks {batch, row, column}
    // listed there: 32 rows by the 16 columns from `column` and from 32, 64 and 96 further
    // on.  A part outside the output is skipped; with the parts of a block one after the
    // other some CTAs had only such ones (120000 x 75, K = 75, all listed: 2097 us, all
    // first parts first 1570).
    const int4 *list;
    int *count; // entries, the record of a wait that gave up, tiles handed out
    int *status;
    unsigned long long *magnitudes; // left zero for the next call
};

// All of C, by all threads of the grid: outputs that the tensor kernel did not finish must not
// pass for results.
__device__ __forceinline__ void fill_nan(const F64Args &p) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(p.status, 0, p.count[1]);
    const int64_t M = p.mg.total, N = p.ng.total, all = p.bg.total * M * N;
    for (int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x; i < all; i += (int64_t)gridDim.x * kThreads) {
        const int64_t q = i / N, b = q / M;
        int64_t oa, ob, oc, om, on;
        group_offsets(p.bg, b, oa, ob, oc);
        group_offsets(p.mg, q - b * M, oa, ob, om);
        group_offsets(p.ng, i - q * N, oa, ob, on);
        p.C[oc + om + on] = __longlong_as_double(0x7ff8000000000000ll);
    }
}

template <int T, bool LISTED>
__global__ void __launch_bounds__(kThreads, T == 32 && !LISTED ? 4 : 3) k_contract_f64(const __grid_constant__ F64Args p) {
    using Q = f64::Tile<T>;
    constexpr int R = Q::R, KG = Q::KG, BK = Q::BK, W = T / R;
    __shared__ f64::Buffers<T> chunk;
    __shared__ double part[T * T];
    const int tid = threadIdx.x;
    const int kgrp = tid / (W * W), tx = tid % W, ty = (tid / W) % W;
    const int rank = p.cs > 1 ? (int)ptx::cluster_ctarank() : 0;
    const int64_t M = p.mg.total, N = p.ng.total, K = p.kg.total;
    const int chunks = (int)((K + BK - 1) / BK);
    const int cbeg = (int)((int64_t)chunks * rank / p.cs), cend = (int)((int64_t)chunks * (rank + 1) / p.cs);
    const int64_t step = gridDim.x / p.cs;
    constexpr int ROWS = 32 / T, PARTS = ROWS * (64 / T); // of a listed block
    const uint32_t listed = LISTED ? (uint32_t)__ldg(p.count) : 0;
    if (LISTED && p.magnitudes && blockIdx.x == 0 && tid < kMagnitudeWords) p.magnitudes[tid] = 0;
    if (LISTED && __ldg(p.count + 1)) return fill_nan(p);
    const int64_t total = LISTED ? (int64_t)PARTS * listed : p.total;
    if (LISTED && blockIdx.x >= total) return;
    constexpr int gap = LISTED && T == 32 ? 16 : 0; // tile column j is column j + (j & gap) from the tile's first
    __shared__ uint32_t next; // listed tiles are handed out one by one
    uint32_t fetched = blockIdx.x;
    for (int64_t t = blockIdx.x / p.cs;; t += step) {
        if (LISTED) {
            if (tid == 0) {
                next = fetched;
                fetched = gridDim.x + atomicAdd((unsigned *)p.count + 2, 1u); // the one after, while this one runs
            }
            __syncthreads(); // and the chunks of the tile before are read
            t = next;
        }
        if (t >= total) break;
        int64_t b, m0, n0;
        if (LISTED) {
            const uint32_t part = (uint32_t)t / listed; // all first parts, then the second ones, ...
            const int4 e = p.list[(uint32_t)t - part * listed];
            const int col = part / ROWS * T;
            b = e.x;
            m0 = e.y + part % ROWS * T;
            n0 = e.z + (T == 32 ? 2 * col : 2 * col - col % 16);
            if (m0 >= M || n0 >= N) {
                __syncthreads();
                continue;
            }
        } else {
            const int64_t q = t / p.ntiles;
            b = q / p.mtiles;
            n0 = (t - q * p.ntiles) * T;
            m0 = (q - b * p.mtiles) * T;
        }
        int64_t ba, bb, bc;
        group_offsets(p.bg, b, ba, bb, bc);
        double acc[R][R] = {};
        f64::accumulate<T>(chunk, {p.mg, p.ng, p.kg, p.A + ba, p.B + bb, p.a_kfast, p.b_kfast, p.ka, p.kb}, m0, n0, gap,
                           cbeg, cend, acc);
        // the k groups of the CTA, then the CTAs of the cluster, added in order
        const bool reduce = KG > 1 || p.cs > 1;
        if (KG > 1) {
            static_assert(KG == 1 || (R == 1 && KG * T * T == kThreads), "one output per thread and k group");
            double *buf = &chunk.A[0][0][0];
            static_assert(KG == 1 || sizeof(chunk.A) >= KG * T * T * sizeof(double), "reduction buffer");
            __syncthreads();
            buf[tid] = acc[0][0];
            __syncthreads();
            if (kgrp == 0) {
                double v = buf[tid];
#pragma unroll
                for (int g = 1; g < KG; g++) v += buf[g * T * T + tid];
                acc[0][0] = v;
            }
        }
        if (p.cs > 1) {
            if (kgrp == 0) {
#pragma unroll
                for (int i = 0; i < R; i++)
#pragma unroll
                    for (int j = 0; j < R; j++) part[(ty + W * i) * T + tx + W * j] = acc[i][j];
            }
            ptx::cluster_sync();
            if (rank == 0 && kgrp == 0) {
#pragma unroll
                for (int i = 0; i < R; i++)
#pragma unroll
                    for (int j = 0; j < R; j++) {
                        const uint32_t at = ptx::smem_u32(&part[(ty + W * i) * T + tx + W * j]);
                        double v = acc[i][j];
                        for (int r = 1; r < p.cs; r++) v += ptx::ld_cluster_f64(ptx::mapa(at, (uint32_t)r));
                        acc[i][j] = v;
                    }
            }
        }
        if (rank == 0 && kgrp == 0) {
#pragma unroll
            for (int i = 0; i < R; i++) {
                const int64_t m = m0 + ty + W * i;
                if (m >= M) continue;
                int64_t ma, mb, mc;
                group_offsets32(p.mg, (uint32_t)m, ma, mb, mc);
#pragma unroll
                for (int j = 0; j < R; j++) {
                    const int64_t n = n0 + tx + W * j + ((tx + W * j) & gap);
                    if (n >= N) continue;
                    int64_t na, nb, nc;
                    group_offsets32(p.ng, (uint32_t)n, na, nb, nc);
                    double *cptr = p.C + bc + mc + nc;
                    *cptr = epilogue(acc[i][j], cptr, p.cp, p.ab, p.zero != 0);
                }
            }
        }
        if (p.cs > 1)
            ptx::cluster_sync(); // the peers' sums are read; the next tile may overwrite them
        else if (!LISTED && (reduce || t + step < total))
            __syncthreads();
    }
}

// Tile edge and cluster size of a contraction: the smallest of the estimated
// times of the busiest SM, its FMAs at two per clock plus a start-up of about
// 2000 clocks per resident round (prologue, first loads, stores) and 1500 for a
// cluster's exchange.  A smaller tile wins only where larger ones leave SMs
// idle: it issues more loads and index arithmetic per FMA (the factors).
double contract_plan(int64_t nb, int64_t M, int64_t N, int64_t K, int &T, int &cs, int most = 8) { // returns the clocks
    double best = -1.0;
    T = 32;
    cs = 1;
    for (int e : {32, 16, 8}) {
        const int bk = e == 32 ? 16 : 32;
        const double factor = e == 32 ? 1.0 : e == 16 ? 1.05 : 1.15;
        for (int c = 1; c <= most; c *= 2) {
            const int64_t chunks = (K + bk - 1) / bk;
            if (c > 1 && chunks < 2 * c) break;
            const double blocks = (double)nb * (double)((M + e - 1) / e) * (double)((N + e - 1) / e) * c;
            const double rounds = std::ceil(blocks / num_sms());
            const double fma = (double)e * e * (double)((chunks + c - 1) / c * bk) * 0.5 * factor;
            const double cost = rounds * fma + std::ceil(rounds / 4.0) * (2000.0 + (c > 1 ? 1500.0 : 0.0));
            if (best < 0.0 || cost < best * 0.98) {
                best = cost;
                T = e;
                cs = c;
            }
        }
    }
    return best;
}

template <int T, bool LISTED>
cudaError_t launch_f64_tiles(const F64Args &p, cudaStream_t s) {
    const int64_t clusters = LISTED ? 3 * num_sms() : std::min<int64_t>(p.total, int64_t(1) << 24);
    if (p.cs == 1) {
        k_contract_f64<T, LISTED><<<(unsigned)clusters, kThreads, 0, s>>>(p);
        return cudaGetLastError();
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * p.cs));
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)p.cs;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_contract_f64<T, LISTED>, p);
}

template <bool LISTED>
cudaError_t launch_f64_tiles(const F64Args &p, int T, cudaStream_t s) {
    return T == 32   ? launch_f64_tiles<32, LISTED>(p, s)
           : T == 16 ? launch_f64_tiles<16, LISTED>(p, s)
                     : launch_f64_tiles<8, LISTED>(p, s);
}

ModeGroup concat(std::initializer_list<const ModeGroup *> groups) {
    ModeGroup g;
    g.total = 1;
    for (const ModeGroup *x : groups)
        for (int d = 0; d < x->n; d++) {
            g.ext[g.n] = x->ext[d];
            for (int t = 0; t < 3; t++) g.s[t][g.n] = x->s[t][d];
            g.total *= x->ext[d];
            g.n++;
        }
    return g;
}

bool fits32(const ModeGroup &g) { return g.total < (int64_t(1) << 31); }

int grid_for(int64_t work, int per_block) {
    int64_t blocks = (work + per_block - 1) / per_block;
    const int64_t cap = (int64_t)num_sms() * 32;
    if (blocks > cap) blocks = cap;
    return (int)(blocks < 1 ? 1 : blocks);
}

} // namespace

eg_status launch_elementwise(const Contraction &c, cudaStream_t s) {
    ModeGroup g = concat({&c.batch, &c.m, &c.n});
    if (g.total == 0) return EG_SUCCESS;
    const int grid = grid_for(g.total, 256);
    // modes that follow one another in all three are one (the groups' folds keep them
    // apart when they lie in different groups)
    bool contiguous = true;
    int64_t span = 1;
    for (int d = g.n - 1; d >= 0 && contiguous; d--) {
        for (int t = 0; t < 3; t++) contiguous = contiguous && g.s[t][d] == span;
        span *= g.ext[d];
    }
    if (contiguous && (((uintptr_t)c.A | (uintptr_t)c.B | (uintptr_t)c.C) & 15) == 0) {
        {
            LaunchScope ls_("k_elementwise", s);
            const int cgrid = grid_for(g.total, 1024);
            const bool plain = c.zero_when_cp_zero && c.cp == 0.0;
            auto go = plain ? (c.ab == 1.0 ? k_elementwise_contiguous<true, true> : k_elementwise_contiguous<true, false>)
                            : (c.ab == 1.0 ? k_elementwise_contiguous<false, true> : k_elementwise_contiguous<false, false>);
            go<<<cgrid, 256, 0, s>>>(g.total, c.A, c.B, c.C, c.cp, c.ab);
        }
        EG_CHECK_LAUNCH("k_elementwise");
        return EG_SUCCESS;
    }
    if (fits32(g))
        { LaunchScope ls_("k_elementwise", s);
        k_elementwise<false><<<grid, 256, 0, s>>>(g, c.A, c.B, c.C, c.cp, c.ab, c.zero_when_cp_zero);
        }
    else
        { LaunchScope ls_("k_elementwise", s);
        k_elementwise<true><<<grid, 256, 0, s>>>(g, c.A, c.B, c.C, c.cp, c.ab, c.zero_when_cp_zero);
        }
    EG_CHECK_LAUNCH("k_elementwise");
    return EG_SUCCESS;
}

eg_status launch_scale(const ModeGroup &g, double *C, double cp, cudaStream_t s) {
    if (g.total == 0) return EG_SUCCESS;
    const int grid = grid_for(g.total, 256);
    {
        LaunchScope ls_("k_scale", s);
        if (fits32(g))
            k_scale<false><<<grid, 256, 0, s>>>(g, C, cp);
        else
            k_scale<true><<<grid, 256, 0, s>>>(g, C, cp);
    }
    EG_CHECK_LAUNCH("k_scale");
    return EG_SUCCESS;
}

eg_status launch_dot(const Contraction &c, cudaStream_t s) {
    const ModeGroup &k = c.k;
    if (k.total <= kDotSmall) {
        const bool contig = k.n == 1 && k.s[0][0] == 1 && k.s[1][0] == 1;
        {
            LaunchScope ls_("k_dot_small", s);
            if (contig)
                k_dot_small<true><<<1, kDotSmallThreads, 0, s>>>(k, c.A, c.B, c.C, c.cp, c.ab, c.zero_when_cp_zero);
            else
                k_dot_small<false><<<1, kDotSmallThreads, 0, s>>>(k, c.A, c.B, c.C, c.cp, c.ab, c.zero_when_cp_zero);
        }
        EG_CHECK_LAUNCH("k_dot_small");
        return EG_SUCCESS;
    }
    const int64_t per_block_min = 4096;
    int64_t nblocks = (k.total + per_block_min - 1) / per_block_min;
    const int64_t cap = (int64_t)num_sms() * kDotBlocksPerSm;
    if (nblocks > cap) nblocks = cap;
    if (nblocks < 1) nblocks = 1;
    const int64_t chunk = ((k.total + nblocks - 1) / nblocks + 1) & ~int64_t(1); // even: pairs stay aligned
    nblocks = std::max<int64_t>(1, (k.total + chunk - 1) / chunk);
    void *ws = nullptr;
    eg_status st = workspace(s, (size_t)nblocks * sizeof(double), &ws);
    if (st != EG_SUCCESS) return st;
    double *partial = (double *)ws;
    const bool contig = k.n == 1 && k.s[0][0] == 1 && k.s[1][0] == 1;
    if (contig)
        { LaunchScope ls_("k_dot_partial", s);
        k_dot_partial<true><<<(int)nblocks, kDotThreads, 0, s>>>(k, c.A, c.B, partial, chunk);
        }
    else
        { LaunchScope ls_("k_dot_partial", s);
        k_dot_partial<false><<<(int)nblocks, kDotThreads, 0, s>>>(k, c.A, c.B, partial, chunk);
        }
    EG_CHECK_LAUNCH("k_dot_partial");
    { LaunchScope ls_("k_dot_final", s);
    k_dot_final<<<1, kDotFinalThreads, 0, s>>>(partial, (int)nblocks, c.C, c.cp, c.ab, c.zero_when_cp_zero);
    }
    EG_CHECK_LAUNCH("k_dot_final");
    return EG_SUCCESS;
}

eg_status launch_gemv(const Contraction &c, cudaStream_t s) {
    ModeGroup rows = concat({&c.batch, &c.m, &c.n});
    ModeGroup k = c.k;
    if (!fits32(k)) return fail(EG_ERROR_NOT_SUPPORTED, "gemv: summed extent exceeds 2^31");
    const bool contig = k.n == 1 && k.s[0][0] == 1 && k.s[1][0] == 1;
    // Long k, unbatched, one free group: the operand without free modes is a
    // vector shared by every output, and k_gemv_rows reuses it for RB rows.  It
    // takes the rows from its first operand, so when they run over B's modes
    // (M empty) the operands and their stride components are swapped.
    const bool rows_kernel = k.total >= 2048 && c.batch.n == 0 && (c.m.n == 0) != (c.n.n == 0);
    const double *X = c.A, *Y = c.B;
    if (rows_kernel && c.m.n == 0) {
        for (int d = 0; d < rows.n; d++) std::swap(rows.s[0][d], rows.s[1][d]);
        for (int d = 0; d < k.n; d++) std::swap(k.s[0][d], k.s[1][d]);
        std::swap(X, Y);
    }
    const bool nested = k.n == 2 && k.s[0][1] == 1 && k.s[1][1] == 1;
    // offset tables for a strided k, built once and shared by every output
    int64_t *offk = nullptr;
    if (!contig && !(rows_kernel && nested) && k.total <= (int64_t(1) << 24) && rows.total > 1) {
        void *ws = nullptr;
        eg_status st = workspace(s, (size_t)k.total * 2 * sizeof(int64_t), &ws);
        if (st != EG_SUCCESS) return st;
        offk = (int64_t *)ws;
        {
            LaunchScope ls_("k_k_offsets", s);
            k_k_offsets<<<(int)std::min<int64_t>((k.total + 255) / 256, (int64_t)num_sms() * 8), 256, 0, s>>>(k, offk);
        }
        EG_CHECK_LAUNCH("k_k_offsets");
    }
    if (rows_kernel && (contig || nested || offk)) {
        constexpr int RB = 4;
        // one unit of RB rows per CTA, handed out by the hardware: persistent CTAs (4 to 8
        // per SM) took 193 to 246 us where these take 188 (n = 100, 10^4 rows of 10^4)
        const int grid = grid_for(rows.total, RB);
        LaunchScope ls_("k_gemv", s);
        if (contig)
            k_gemv_rows<RB, 0><<<grid, 256, 0, s>>>(rows, k, X, Y, c.C, c.cp, c.ab, c.zero_when_cp_zero, nullptr);
        else if (nested)
            k_gemv_rows<RB, 1><<<grid, 256, 0, s>>>(rows, k, X, Y, c.C, c.cp, c.ab, c.zero_when_cp_zero, nullptr);
        else
            k_gemv_rows<RB, 2><<<grid, 256, 0, s>>>(rows, k, X, Y, c.C, c.cp, c.ab, c.zero_when_cp_zero, offk);
    } else if (k.total >= 2048) {
        const int grid = grid_for(rows.total, 1);
        LaunchScope ls_("k_gemv", s);
        if (contig)
            k_gemv<256, true><<<grid, 256, 0, s>>>(rows, k, X, Y, c.C, c.cp, c.ab, c.zero_when_cp_zero, nullptr);
        else
            k_gemv<256, false><<<grid, 256, 0, s>>>(rows, k, X, Y, c.C, c.cp, c.ab, c.zero_when_cp_zero, offk);
    } else {
        const int grid = grid_for(rows.total, 8);
        LaunchScope ls_("k_gemv", s);
        if (contig)
            k_gemv<32, true><<<grid, 256, 0, s>>>(rows, k, X, Y, c.C, c.cp, c.ab, c.zero_when_cp_zero, nullptr);
        else
            k_gemv<32, false><<<grid, 256, 0, s>>>(rows, k, X, Y, c.C, c.cp, c.ab, c.zero_when_cp_zero, offk);
    }
    EG_CHECK_LAUNCH("k_gemv");
    return EG_SUCCESS;
}

namespace {
F64Args f64_args(const Contraction &c) {
    F64Args p{};
    p.bg = c.batch;
    p.mg = c.m;
    p.ng = c.n;
    p.kg = c.k;
    p.A = c.A;
    p.B = c.B;
    p.C = c.C;
    p.cp = c.cp;
    p.ab = c.ab;
    p.zero = c.zero_when_cp_zero ? 1 : 0;
    // read each operand along the smaller of its fastest k and row strides
    auto kfast = [](const ModeGroup &k, const ModeGroup &r, int comp) {
        if (k.n == 0) return 0;
        return r.n == 0 || k.s[comp][k.n - 1] < r.s[comp][r.n - 1] ? 1 : 0;
    };
    p.a_kfast = kfast(c.k, c.m, 0);
    p.b_kfast = kfast(c.k, c.n, 1);
    p.ka = mode_group_affine_stride(c.k, 0);
    p.kb = mode_group_affine_stride(c.k, 1);
    p.cs = 1;
    return p;
}
} // namespace

eg_status launch_contract_f64(const Contraction &c, cudaStream_t s) {
    if (!fits32(c.m) || !fits32(c.n) || !fits32(c.k))
        return fail(EG_ERROR_NOT_SUPPORTED, "contraction: a mode group exceeds 2^31 elements");
    if (c.m.total > int64_t(65535) * 64) return fail(EG_ERROR_NOT_SUPPORTED, "contraction: too many row tiles");
    F64Args p = f64_args(c);
    int T = 32;
    contract_plan(c.batch.total, c.m.total, c.n.total, c.k.total, T, p.cs);
    p.mtiles = (c.m.total + T - 1) / T;
    p.ntiles = (c.n.total + T - 1) / T;
    p.total = c.batch.total * p.mtiles * p.ntiles;
    if (p.total == 0) return EG_SUCCESS;
    {
        LaunchScope ls_("k_contract_f64", s);
        const cudaError_t err = launch_f64_tiles<false>(p, T, s);
        if (err != cudaSuccess) return cuda_fail(err, "k_contract_f64");
    }
    EG_CHECK_LAUNCH("k_contract_f64");
    return EG_SUCCESS;
}

double contract_f64_seconds(const Contraction &c) {
    int T = 0, cs = 0;
    return contract_plan(c.batch.total, c.m.total, c.n.total, c.k.total, T, cs) / 2.0e9;
}

eg_status launch_contract_f64_listed(const Contraction &c, const int4 *list, int *count, int *status,
                                     unsigned long long *magnitudes, cudaStream_t s) {
    // Tiles as if the whole output were listed (K in one piece: launching clusters takes 2 us
    // more, mostly for nothing), but for outputs of six rounds of 32 x 32 tiles or more, where
    // those are faster although the last round is not full (1024^3, all listed, dealt in turn:
    // 2.19 ms, 2.33 with 16 x 16; handed out one by one 1.97).
    F64Args p = f64_args(c);
    int T = 32;
    if (c.batch.total * ((c.m.total + 31) / 32) * ((c.n.total + 31) / 32) < 6 * num_sms())
        contract_plan(c.batch.total, c.m.total, c.n.total, c.k.total, T, p.cs, 1);
    p.list = list;
    p.count = count;
    p.status = status;
    p.magnitudes = magnitudes;
    {
        LaunchScope ls_("k_contract_f64_listed", s);
        const cudaError_t err = launch_f64_tiles<true>(p, T, s);
        if (err != cudaSuccess) return cuda_fail(err, "k_contract_f64_listed");
    }
    EG_CHECK_LAUNCH("k_contract_f64_listed");
    return EG_SUCCESS;
}

} // namespace eg
