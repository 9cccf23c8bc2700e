// Grouped execution of many independent contractions that share one index
// pattern but not their extents (the reference's list einsum,
// Backends/Dispatch.hpp:1264-1286, and block-sparse blocks).
//
// A plan lowers every item to the canonical contraction, builds a device-side
// work list of output tiles (largest first), and captures the whole batch as
// a CUDA graph that later calls replay:
//   * FP64, when it pays (f64_tensor_plan_pays): as split-BF16 with eight slices and
//     the accuracy check of split.cu's launch_f64_tensor, then one launch of the FMA
//     kernel over the blocks that failed it;
//   * FP64 otherwise: one persistent launch of k_grouped_f64 over the work list; each
//     entry computes a 32x32 or 64x64 tile with the DFMA core, the tile size
//     chosen per shape bucket by the autotuner (autotune.cu);
//   * split-BF16: one digit-splitting launch over every operand of every item, then
//     one persistent launch of the tcgen05 GEMM over the work list
//     (k_tc_split_gemm<true>).
#include <algorithm>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <numeric>
#include <queue>
#include <string>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>

#include "f64_tile.cuh"
#include "grouped.cuh"
#include "ptx.cuh"
#include "split.cuh"

namespace eg {
int64_t mode_group_affine_stride(const ModeGroup &g, int comp);
eg_status encode_planes_extent(CUtensorMap *map, void *base, int64_t K, int64_t rows, int64_t planes, int64_t Kp,
                               int64_t Rp);
void set_capture_mode(bool on);
void count_launches(uint64_t n);
} // namespace eg

namespace eg::grouped {

namespace {

// ------------------------------------------------------------ FP64 tiles --
struct F64Item {
    const double *A, *B;
    double *C;
    ModeGroup b, m, n, k;
    int a_kfast, b_kfast;
    int64_t ka, kb; // single k strides of A and B (0: none)
};

constexpr int BK = 16, THREADS = 256, LD = 65;

template <int T>
__device__ __forceinline__ void f64_tile(const F64Item &it, int64_t bidx, int64_t m0, int64_t n0, double cp, double ab,
                                         bool zero, double (*As)[LD], double (*Bs)[LD]) {
    constexpr int R = T / 16; // outputs per thread per dimension, and loads per thread per operand
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int64_t M = it.m.total, N = it.n.total, K = it.k.total;
    int64_t ba, bb, bc;
    group_offsets(it.b, bidx, ba, bb, bc);
    int lm[R], lk[R], ln[R], lkb[R];
    int64_t offA[R], offB[R];
    bool okA[R], okB[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int e = tid + THREADS * i;
        lm[i] = it.a_kfast ? e / BK : e % T;
        lk[i] = it.a_kfast ? e % BK : e / T;
        ln[i] = it.b_kfast ? e / BK : e % T;
        lkb[i] = it.b_kfast ? e % BK : e / T;
        int64_t oa, ob, oc;
        okA[i] = m0 + lm[i] < M;
        group_offsets32(it.m, (uint32_t)(okA[i] ? m0 + lm[i] : 0), oa, ob, oc);
        offA[i] = ba + oa;
        okB[i] = n0 + ln[i] < N;
        group_offsets32(it.n, (uint32_t)(okB[i] ? n0 + ln[i] : 0), oa, ob, oc);
        offB[i] = bb + ob;
    }
    double acc[R][R];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < R; j++) acc[i][j] = 0.0;
    for (int64_t k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < R; i++) {
            const int64_t ka = k0 + lk[i];
            double va = 0.0;
            if (okA[i] && ka < K) {
                int64_t oa, ob, oc;
                group_offsets32(it.k, (uint32_t)ka, oa, ob, oc);
                va = __ldg(it.A + offA[i] + oa);
            }
            As[lk[i]][lm[i]] = va;
            const int64_t kb = k0 + lkb[i];
            double vb = 0.0;
            if (okB[i] && kb < K) {
                int64_t oa, ob, oc;
                group_offsets32(it.k, (uint32_t)kb, oa, ob, oc);
                vb = __ldg(it.B + offB[i] + ob);
            }
            Bs[lkb[i]][ln[i]] = vb;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            double a[R], b[R];
#pragma unroll
            for (int i = 0; i < R; i++) a[i] = As[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < R; j++) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < R; i++)
#pragma unroll
                for (int j = 0; j < R; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int64_t m = m0 + ty + 16 * i;
        if (m >= M) continue;
        int64_t ma, mb, mc;
        group_offsets32(it.m, (uint32_t)m, ma, mb, mc);
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int64_t n = n0 + tx + 16 * j;
            if (n >= N) continue;
            int64_t na, nb, nc;
            group_offsets32(it.n, (uint32_t)n, na, nb, nc);
            double *cptr = it.C + bc + mc + nc;
            const double v = ab * acc[i][j];
            *cptr = (zero && cp == 0.0) ? v : cp * (*cptr) + v;
        }
    }
}

// Work entry: {item, batch index, mt, nt}; tile size per item in `tiles`.
__global__ void __launch_bounds__(THREADS) k_grouped_f64(const F64Item *items, const int *tiles, const int4 *work,
                                                          int nwork, double cp, double ab, int zero) {
    __shared__ double As[BK][LD];
    __shared__ double Bs[BK][LD];
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int4 e = work[w];
        const F64Item &it = items[e.x];
        if (tiles[e.x] == 64)
            f64_tile<64>(it, e.y, int64_t(64) * e.z, int64_t(64) * e.w, cp, ab, zero != 0, As, Bs);
        else
            f64_tile<32>(it, e.y, int64_t(32) * e.z, int64_t(32) * e.w, cp, ab, zero != 0, As, Bs);
    }
}

// All outputs of all items (work: {item, batch index, mt, nt} of every 128 x 128 tile): what the
// tensor kernel did not finish must not pass for results.
__device__ __noinline__ void fill_nan(const F64Item *items, const int4 *work, int nwork, int *const *status_at, int lost) {
    if (blockIdx.x == 0 && threadIdx.x == 0) split::report_lost(status_at, nullptr, lost);
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const int4 e = work[w];
        const F64Item &it = items[e.x];
        const int64_t m0 = (int64_t)e.z * split::kBM, n0 = (int64_t)e.w * split::kBN;
        const int64_t rows = min((int64_t)split::kBM, it.m.total - m0), cols = min((int64_t)split::kBN, it.n.total - n0);
        int64_t oa, ob, oc, om, on;
        group_offsets(it.b, e.y, oa, ob, oc);
        for (int64_t i = threadIdx.x; i < rows * cols; i += blockDim.x) {
            group_offsets(it.m, m0 + i / cols, oa, ob, om);
            group_offsets(it.n, n0 + i % cols, oa, ob, on);
            it.C[oc + om + on] = __longlong_as_double(0x7ff8000000000000ll);
        }
    }
}

// The blocks of outputs that the FP64 form on the tensor cores left out, *count of them:
// {item, batch index, row, column}, 32 rows by the 16 columns from `column` and from 32,
// 64 and 96 further on.  A list that fails the check everywhere must not take longer than
// as a plan for the FP64 pipe, so: tiles of 16 x 16, as items of lists are small, those
// outside the output skipped, handed out one by one (count[1], cleared like the count), all
// first tiles of the blocks first.  512 uneven items (4-32 x 4-32 summed, 20-120 x 20-120), all
// graded: 876 us in all, in tiles of 32 x 32 dealt in turn 2691; as a plan for the FP64 pipe
// 825 to 940.  2048 items: 2.97 ms, 8.11, 3.28.
__global__ void __launch_bounds__(f64::kThreads) k_grouped_f64_listed(const F64Item *items, const int4 *list, int *count,
                                                                      double cp, double ab, int zero,
                                                                      int *const *status_at, const int4 *work, int nwork) {
    constexpr int T = 16;
    __shared__ f64::Buffers<T> chunk;
    __shared__ uint32_t next;
    const int tx = threadIdx.x % T, ty = threadIdx.x / T;
    const uint32_t listed = (uint32_t)__ldg(count), total = 8 * listed;
    const int lost = __ldg(count + 2);
    if (lost) return fill_nan(items, work, nwork, status_at, lost);
    uint32_t fetched = blockIdx.x;
    while (true) {
        if (threadIdx.x == 0) {
            next = fetched;
            fetched = gridDim.x + atomicAdd((unsigned *)count + 1, 1u); // the one after, while this one runs
        }
        __syncthreads(); // and the chunks of the tile before are read
        const uint32_t u = next;
        if (u >= total) return;
        const uint32_t part = u / listed;
        const int4 e = list[u - part * listed];
        const F64Item &it = items[e.x];
        const int64_t m0 = e.z + part % 2 * T, n0 = e.w + part / 2 * 2 * T;
        if (m0 >= it.m.total || n0 >= it.n.total) {
            __syncthreads();
            continue;
        }
        int64_t ba, bb, bc, oa, ob, oc;
        group_offsets(it.b, e.y, ba, bb, bc);
        double acc[1][1] = {};
        constexpr int CK = f64::Tile<T>::BK;
        f64::accumulate<T>(chunk, {it.m, it.n, it.k, it.A + ba, it.B + bb, it.a_kfast, it.b_kfast, it.ka, it.kb}, m0, n0, 0,
                           0, (int)((it.k.total + CK - 1) / CK), acc);
        if (m0 + ty < it.m.total && n0 + tx < it.n.total) {
            group_offsets32(it.m, (uint32_t)(m0 + ty), oa, ob, oc);
            bc += oc;
            group_offsets32(it.n, (uint32_t)(n0 + tx), oa, ob, oc);
            double *cptr = it.C + bc + oc;
            const double v = ab * acc[0][0];
            *cptr = (zero && cp == 0.0) ? v : cp * (*cptr) + v;
        }
    }
}

// --------------------------------------------------- grouped digit split --
struct GOp {
    const double *X;
    ModeGroup bg, rg, kg;
    int comp;             // 0: A, 1: B
    int row_fast;         // operand contiguous along rows
    int nbatch;
    int64_t rows, Rp, K, Kp;
    int64_t rowbase;      // first entry in the row-max / exponent arrays
    int64_t plane0;       // element offset of the first digit plane
    int64_t pitch, pstride; // elements between rows and between planes (16-byte multiples)
    int64_t rtab, ktab;   // first entries of this operand's row and K offsets in the plan's offset table
    int64_t sr, sk;       // the single element stride of the rows / of K when the modes nest (else 0: tables)
};

__host__ __device__ __forceinline__ int64_t pick(int comp, int64_t oa, int64_t ob) { return comp == 0 ? oa : ob; }

// One work unit = 32 rows of one operand of one item (and batch index): the
// rows' maxima (the operand is read once along its contiguous direction), their
// exponents, then the digit planes of those rows, written K-major in BF16 pairs
// through a 32 x 64 shared tile when the operand is contiguous along its rows.
// Only the real rows and K are written: the planes and exponents of padded rows
// and of K beyond the item's extent are zeroed once when the plan is built and
// never written after.
constexpr int kGU = 32, kGK = 64, kGThreads = 256, kGWarps = kGThreads / 32;

template <int S>
__global__ void __launch_bounds__(kGThreads, 4) k_grouped_split(const GOp *ops, const int4 *units, int nunits,
                                                             const long long *__restrict__ offs, int *rexpA,
                                                             int *rexpB, __nv_bfloat16 *planesA,
                                                             __nv_bfloat16 *planesB) {
    __shared__ double tile[kGU][kGK + 1];
    __shared__ unsigned long long red[kGWarps][kGU];
    __shared__ int ex[kGU];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int u = blockIdx.x; u < nunits; u += gridDim.x) {
        const int4 un = units[u];
        const GOp &g = ops[un.x];
        const int64_t b = un.y, r0 = un.z;
        const int64_t K = g.K;
        const int nr = (int)(g.rows - r0 < kGU ? g.rows - r0 : kGU);
        const long long *koff = offs + g.ktab; // element offset of each k in this operand
        const int64_t sk = g.sk;
        auto kofs = [&](int64_t k) -> int64_t { return sk ? k * sk : (int64_t)__ldg(koff + k); };
        const double *X = g.X;
        int64_t oa, ob, oc;
        group_offsets(g.bg, b, oa, ob, oc);
        const int64_t obase = pick(g.comp, oa, ob);
        const bool row_fast = g.row_fast != 0;
        // row offsets: the lane's row (rows contiguous) or the warp's rows w + 8j (K contiguous)
        int64_t orow[kGU / kGWarps];
#pragma unroll
        for (int j = 0; j < kGU / kGWarps; j++) {
            const int rr = row_fast ? lane : w + kGWarps * j;
            orow[j] = (rr < nr && (j == 0 || !row_fast))
                          ? obase + (g.sr ? (r0 + rr) * g.sr : (int64_t)__ldg(offs + g.rtab + r0 + rr))
                          : 0;
        }
        // phase 1: row maxima of |x| as IEEE bit patterns
        if (row_fast) {
            unsigned long long mx = 0;
            if (lane < nr) {
#pragma unroll 8
                for (int64_t k = w; k < K; k += kGWarps)
                    mx = max(mx, split::abs_bits(__ldg(X + orow[0] + kofs(k))));
            }
            red[w][lane] = mx;
        } else {
#pragma unroll
            for (int j = 0; j < kGU / kGWarps; j++) {
                const int rr = w + kGWarps * j;
                unsigned long long mx = 0;
                if (rr < nr) {
#pragma unroll 4
                    for (int64_t k = lane; k < K; k += 32)
                        mx = max(mx, split::abs_bits(__ldg(X + orow[j] + kofs(k))));
                }
                for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                if (lane == 0) {
                    red[0][rr] = mx;
                    for (int q = 1; q < kGWarps; q++) red[q][rr] = 0;
                }
            }
        }
        __syncthreads();
        if (w == 0) {
            unsigned long long mx = red[0][lane];
            for (int q = 1; q < kGWarps; q++) mx = max(mx, red[q][lane]);
            const double m = __longlong_as_double((long long)mx);
            int e = 0;
            if (!isfinite(m))
                e = INT_MIN;
            else if (m > 0.0)
                frexp(m, &e);
            ex[lane] = e;
            if (lane < nr) (g.comp ? rexpB : rexpA)[g.rowbase + b * g.Rp + r0 + lane] = e;
        }
        __syncthreads();
        // phase 2: digit planes, 64 K at a time
        __nv_bfloat16 *planes = g.comp ? planesB : planesA;
        for (int64_t k0 = 0; k0 < K; k0 += kGK) {
            if (row_fast) {
#pragma unroll
                for (int kk = w; kk < kGK; kk += kGWarps) {
                    const int64_t k = k0 + kk;
                    tile[lane][kk] = (k < K && lane < nr) ? __ldg(X + orow[0] + kofs(k)) : 0.0;
                }
            } else {
#pragma unroll
                for (int j = 0; j < kGU / kGWarps; j++) {
                    const int rr = w + kGWarps * j;
#pragma unroll
                    for (int h = 0; h < kGK / 32; h++) {
                        const int64_t k = k0 + lane + 32 * h;
                        tile[rr][lane + 32 * h] = (rr < nr && k < K) ? __ldg(X + orow[j] + kofs(k)) : 0.0;
                    }
                }
            }
            __syncthreads();
            const int64_t k = k0 + 2 * lane;
#pragma unroll
            for (int j = 0; j < kGU / kGWarps; j++) {
                const int rr = w + kGWarps * j;
                if (rr < nr && k < K) {
                    uint32_t pk[S];
                    const int e = ex[rr];
                    if (e == INT_MIN) {
#pragma unroll
                        for (int q = 0; q < S; q++) pk[q] = 0u;
                    } else {
                        split::digits_bf16x2<S>(tile[rr][2 * lane], tile[rr][2 * lane + 1], e, pk);
                    }
#pragma unroll
                    for (int q = 0; q < S; q++)
                        *reinterpret_cast<uint32_t *>(planes + g.plane0 + (b * S + q) * g.pstride + (r0 + rr) * g.pitch + k) = pk[q];
                }
            }
            __syncthreads();
        }
    }
}

// The same when every item's K is short (kRowsMaxK): a unit is 32 rows or fewer (a power
// of two), as many as keep it within 32 KB of shared memory, so that every element is read
// once, all of a unit's loads in flight at once while the unit before is converted, and
// the maxima and digits are taken from shared memory.  Bound: latency and integer
// instructions; the unit above read each element twice, a few loads per thread at a time.
// What a unit needs to be known stands in one record, itself fetched three units ahead:
// looked up through the operand's, its loads waited for three chains of loads first
// (2048 items of 4-32 x 4-32 summed, 20-120 x 20-120, S = 5: 286 us, now 241).
constexpr int64_t kRowsElems = 4096, kRowsMaxK = 1152;

struct alignas(16) RowsUnit {
    const double *X;       // the operand at this batch index (and at the first row, when sr)
    __nv_bfloat16 *planes; // the first row's leading digits
    int *rexp;             // the rows' exponents
    unsigned long long *magnitudes; // FP64 form: the operand's sum over all rows (TcGemmParams)
    int64_t sr, sk;        // strides of the rows and of k, 0: the tables at rtab (first row), ktab
    int64_t rtab, ktab;
    int64_t pitch, pstride;
    int K, R, rows; // rows: of the R, those that exist
    int flags;      // 1: contiguous along the rows
};
constexpr int kUnitSlots = 4;
static_assert(sizeof(RowsUnit) % 16 == 0 && sizeof(RowsUnit) / 16 <= 32, "fetched by one warp, 16 bytes a lane");

__host__ __device__ inline int rows_ld(int64_t K) { return (int)((K + 15) / 16 * 16 + 2); }

template <int S, bool CHECK>
__global__ void __launch_bounds__(kGThreads, 3) k_grouped_rows(const RowsUnit *units, int nunits,
                                                               const long long *__restrict__ offs, int tile_elems) {
    extern __shared__ __align__(16) double tiles[]; // two of [rows of the unit][rows_ld(K)]
    __shared__ RowsUnit slots[kUnitSlots];
    __shared__ int ex[32];
    constexpr int P = S + (CHECK ? 2 : 0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto fetch = [&](int64_t u, int n) { // the record of this CTA's n-th unit
        if (u < nunits && threadIdx.x < sizeof(RowsUnit) / 16)
            ptx::cp_async16((double *)&slots[n % kUnitSlots] + 2 * threadIdx.x, (const double *)(units + u) + 2 * threadIdx.x);
    };
    auto load = [&](int64_t u, int n, double *tile) {
        if (u < nunits) {
            const RowsUnit &g = slots[n % kUnitSlots];
            const int R = g.R, K = g.K, ld = rows_ld(K), kw = (K + 3) & ~3, nr = g.rows;
            const int64_t sr = g.sr, sk = g.sk, rtab = g.rtab, ktab = g.ktab;
            const double *X = g.X;
            // (a single k stride is added up: the loop is two copies for it)
            auto row_copy = [&](int r, int k, int step) { // k, k + step, ... of row r
                const double *x = X + (sr ? r * sr : (int64_t)__ldg(offs + rtab + r));
                double *t = tile + r * ld;
                if (sk) {
                    const int64_t inc = (int64_t)step * sk;
                    x += (int64_t)k * sk;
#pragma unroll 4
                    for (; k < K; k += step, x += inc) ptx::cp_async8(t + k, x);
                } else {
#pragma unroll 4
                    for (; k < K; k += step) ptx::cp_async8(t + k, x + __ldg(offs + ktab + k));
                }
                for (; k < kw; k += step) t[k] = 0.0;
            };
            if (g.flags & 1) {
                const int r = lane & (R - 1), per = 32 / R;
                if (r < nr) row_copy(r, warp * per + lane / R, kGWarps * per);
            } else {
                for (int r = warp; r < nr; r += kGWarps) row_copy(r, lane, 32);
            }
        }
    };
    const int64_t u0 = blockIdx.x, step = gridDim.x;
    for (int n = 0; n < 3; n++) fetch(u0 + n * step, n);
    ptx::cp_async_commit();
    ptx::cp_async_wait<0>();
    __syncthreads();
    load(u0, 0, tiles);
    ptx::cp_async_commit();
    int n = 0, buf = 0;
    for (int64_t u = u0; u < nunits; u += step, n++) {
        load(u + step, n + 1, tiles + (buf ^ 1) * tile_elems);
        fetch(u + 3 * step, n + 3); // has landed two units on: its slot was read up to the unit before
        ptx::cp_async_commit();
        ptx::cp_async_wait<1>();
        __syncthreads();
        const double *tile = tiles + buf * tile_elems;
        const RowsUnit &g = slots[n % kUnitSlots];
        const int K = g.K, ld = rows_ld(K), kw = (K + 3) & ~3, nr = g.rows;
        const int64_t pstride = g.pstride, pitch = g.pitch;
        // the rows' exponents, a warp to a row, then the digits, four k a thread and the rows
        // one after the other, so that rows of few k keep all lanes busy
        __nv_bfloat16 *const planes = g.planes;
        int *const rexp = g.rexp;
        unsigned long long *const magnitudes = g.magnitudes;
        float leading = 0.0f; // whole numbers below 2^24
        for (int r = warp; r < nr; r += kGWarps) {
            const int e = split::row_exponent(split::row_max_bits(tile + r * ld, kw, lane));
            if (lane == 0) ex[r] = rexp[r] = e;
        }
        __syncthreads();
        const int quads = kw / 4, dr = kGThreads / quads, dk = kGThreads - dr * quads;
        int r = threadIdx.x / quads, k = threadIdx.x - r * quads;
        for (int i = threadIdx.x; i < nr * quads; i += kGThreads) {
            const double *x = tile + r * ld + 4 * k;
            const double2 v0 = *(const double2 *)x, v1 = *(const double2 *)(x + 2);
            uint32_t p0[P], p1[P];
            const int e = ex[r];
            if (e == INT_MIN) {
#pragma unroll
                for (int s = 0; s < P; s++) p0[s] = p1[s] = 0u;
            } else {
                split::digits_bf16x2<S>(v0.x, v0.y, e, p0);
                split::digits_bf16x2<S>(v1.x, v1.y, e, p1);
                if constexpr (CHECK) {
                    p0[S] = split::check_magnitude(p0[0]);
                    p1[S] = split::check_magnitude(p1[0]);
                }
            }
            if constexpr (CHECK) {
                leading += split::pair_sum(p0[S]) + split::pair_sum(p1[S]);
                p0[S + 1] = split::check_mark(v0.x, v0.y);
                p1[S + 1] = split::check_mark(v1.x, v1.y);
            }
            __nv_bfloat16 *row = planes + r * pitch + 4 * k;
#pragma unroll
            for (int s = 0; s < P; s++) *(uint2 *)(row + s * pstride) = make_uint2(p0[s], p1[s]);
            r += dr;
            k += dk;
            if (k >= quads) {
                k -= quads;
                r++;
            }
        }
        if constexpr (CHECK) {
            const unsigned sum = __reduce_add_sync(0xffffffffu, (unsigned)leading);
            if (lane == 0) atomicAdd(magnitudes, (unsigned long long)sum);
        }
        __syncthreads(); // the tile is read before the loads of the unit after next replace it
        buf ^= 1;
    }
}

// f(std::integral_constant<int, S>, std::bool_constant<FP64 form>) for a run-time form.
template <typename F>
auto with_slices(int S, bool f64, F f) {
    using std::integral_constant;
    if (f64) return f(integral_constant<int, split::kF64Slices>{}, std::true_type{});
    switch (S) {
    case 2: return f(integral_constant<int, 2>{}, std::false_type{});
    case 3: return f(integral_constant<int, 3>{}, std::false_type{});
    case 4: return f(integral_constant<int, 4>{}, std::false_type{});
    case 5: return f(integral_constant<int, 5>{}, std::false_type{});
    default: return f(integral_constant<int, 6>{}, std::false_type{});
    }
}

// Outside any capture, before launch_grouped_rows is captured.
cudaError_t allow_grouped_rows(int S, bool f64) {
    return with_slices(S, f64, [](auto slices, auto check) {
        return cudaFuncSetAttribute(k_grouped_rows<decltype(slices)::value, decltype(check)::value>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, 76 * 1024);
    });
}

eg_status launch_grouped_rows(int S, bool f64, const RowsUnit *units, int nunits, const long long *offs, size_t smem,
                              cudaStream_t s) {
    const int per_sm = std::max(1, std::min<int>(8, (int)(220 * 1024 / (smem + 1024))));
    const int grid = std::min(std::max(nunits, 1), num_sms() * per_sm);
    with_slices(S, f64, [&](auto slices, auto check) {
        k_grouped_rows<decltype(slices)::value, decltype(check)::value>
            <<<grid, kGThreads, smem, s>>>(units, nunits, offs, (int)(smem / 16));
        return 0;
    });
    EG_CHECK_LAUNCH("k_grouped_rows");
    return EG_SUCCESS;
}

eg_status launch_grouped_split(int S, const GOp *ops, const int4 *units, int nunits, const long long *offs, int *eA,
                               int *eB, __nv_bfloat16 *pA, __nv_bfloat16 *pB, cudaStream_t s) {
    const int grid = (int)std::min<int64_t>(std::max(nunits, 1), (int64_t)num_sms() * 8);
    with_slices(S, false, [&](auto slices, auto) {
        k_grouped_split<decltype(slices)::value><<<grid, kGThreads, 0, s>>>(ops, units, nunits, offs, eA, eB, pA, pB);
        return 0;
    });
    EG_CHECK_LAUNCH("grouped digit splitting");
    return EG_SUCCESS;
}

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

bool fast_along(const ModeGroup &g, int comp) { return g.n > 0 && g.s[comp][g.n - 1] == 1; }

} // namespace

// ------------------------------------------------------------------ plan --

namespace {

eg_status dev_copy(Plan &plan, const void *host, size_t bytes, void **dev) {
    void *p = nullptr;
    eg_status st = tracked_malloc(bytes ? bytes : 16, &p, !plan.optional);
    if (st != EG_SUCCESS) return st;
    plan.owned.push_back(p);
    if (bytes) EG_CUDA(cudaMemcpy(p, host, bytes, cudaMemcpyHostToDevice));
    *dev = p;
    return EG_SUCCESS;
}

eg_status dev_alloc(Plan &plan, size_t bytes, void **dev) {
    void *p = nullptr;
    eg_status st = tracked_malloc(bytes ? bytes : 16, &p, !plan.optional);
    if (st != EG_SUCCESS) return st;
    plan.owned.push_back(p);
    *dev = p;
    return EG_SUCCESS;
}

struct CaptureGuard {
    CaptureGuard() { set_capture_mode(true); }
    ~CaptureGuard() { set_capture_mode(false); }
};

// Issues the FP64 grouped launch on `s` (captured by the caller).
eg_status issue_f64(const F64Item *items, const int *tiles, const int4 *work, int nwork, double cp, double ab,
                    int zero, cudaStream_t s) {
    if (nwork <= 0) return EG_SUCCESS;
    const int grid = std::min(nwork, num_sms() * 8);
    {
        LaunchScope ls_("k_grouped_f64", s);
        k_grouped_f64<<<grid, THREADS, 0, s>>>(items, tiles, work, nwork, cp, ab, zero);
    }
    EG_CHECK_LAUNCH("k_grouped_f64");
    return EG_SUCCESS;
}

// Cost-ordered work list (largest K first) of tiles of size tile[item].
std::vector<int4> f64_work(const std::vector<Contraction> &cs, const std::vector<int> &tiles) {
    std::vector<std::pair<int64_t, int4>> w;
    for (size_t i = 0; i < cs.size(); i++) {
        const int T = tiles[i];
        const int64_t mt = (cs[i].m.total + T - 1) / T, nt = (cs[i].n.total + T - 1) / T;
        for (int64_t b = 0; b < cs[i].batch.total; b++)
            for (int64_t x = 0; x < mt; x++)
                for (int64_t y = 0; y < nt; y++)
                    w.push_back({cs[i].k.total * T * T, make_int4((int)i, (int)b, (int)x, (int)y)});
    }
    std::stable_sort(w.begin(), w.end(), [](auto &a, auto &b) { return a.first > b.first; });
    std::vector<int4> out;
    out.reserve(w.size());
    for (auto &e : w) out.push_back(e.second);
    return out;
}

F64Item f64_item(const Contraction &c) {
    F64Item it;
    it.A = c.A;
    it.B = c.B;
    it.C = c.C;
    it.b = c.batch;
    it.m = c.m;
    it.n = c.n;
    it.k = c.k;
    it.a_kfast = c.k.n > 0 && c.k.s[0][c.k.n - 1] == 1 && !(c.m.n > 0 && c.m.s[0][c.m.n - 1] == 1);
    it.b_kfast = c.k.n > 0 && c.k.s[1][c.k.n - 1] == 1 && !(c.n.n > 0 && c.n.s[1][c.n.n - 1] == 1);
    it.ka = mode_group_affine_stride(c.k, 0);
    it.kb = mode_group_affine_stride(c.k, 1);
    return it;
}

// Times a FP64 grouped launch of `items` with tile size T into scratch outputs.
eg_status time_f64(const std::vector<Contraction> &bucket, int T, cudaStream_t s, float *ms) {
    // outputs redirected to compact scratch so user data is untouched
    std::vector<Contraction> cs = bucket;
    size_t total = 0;
    for (auto &c : cs) total += (size_t)(c.batch.total * c.m.total * c.n.total);
    Plan tmp;
    void *scratch = nullptr;
    eg_status st = dev_alloc(tmp, total * sizeof(double), &scratch);
    if (st != EG_SUCCESS) return st;
    size_t off = 0;
    std::vector<F64Item> items;
    for (auto &c : cs) {
        c.C = (double *)scratch + off;
        // compact C strides: batch, m, n row-major
        int64_t stride = 1;
        for (int d = c.n.n - 1; d >= 0; d--) {
            c.n.s[2][d] = stride;
            stride *= c.n.ext[d];
        }
        for (int d = c.m.n - 1; d >= 0; d--) {
            c.m.s[2][d] = stride;
            stride *= c.m.ext[d];
        }
        for (int d = c.batch.n - 1; d >= 0; d--) {
            c.batch.s[2][d] = stride;
            stride *= c.batch.ext[d];
        }
        off += (size_t)(c.batch.total * c.m.total * c.n.total);
        items.push_back(f64_item(c));
    }
    std::vector<int> tiles(cs.size(), T);
    auto work = f64_work(cs, tiles);
    void *d_items, *d_tiles, *d_work;
    if ((st = dev_copy(tmp, items.data(), items.size() * sizeof(F64Item), &d_items)) != EG_SUCCESS) return st;
    if ((st = dev_copy(tmp, tiles.data(), tiles.size() * sizeof(int), &d_tiles)) != EG_SUCCESS) return st;
    if ((st = dev_copy(tmp, work.data(), work.size() * sizeof(int4), &d_work)) != EG_SUCCESS) return st;
    cudaEvent_t e0, e1;
    EG_CUDA(cudaEventCreate(&e0));
    EG_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    for (int rep = 0; rep < 3; rep++) {
        EG_CUDA(cudaEventRecord(e0, s));
        st = issue_f64((F64Item *)d_items, (int *)d_tiles, (int4 *)d_work, (int)work.size(), 0.0, 1.0, 1, s);
        if (st != EG_SUCCESS) break;
        EG_CUDA(cudaEventRecord(e1, s));
        EG_CUDA(cudaEventSynchronize(e1));
        float t = 0.f;
        EG_CUDA(cudaEventElapsedTime(&t, e0, e1));
        if (rep > 0) best = std::min(best, t);
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *ms = best;
    return st;
}

} // namespace

// Chooses the FP64 tile size of every item: per shape bucket from the tuning
// cache, timing both sizes on the bucket's items when the cache has no entry.
eg_status choose_f64_tiles(const std::vector<Contraction> &cs, cudaStream_t s, std::vector<int> &tiles) {
    tiles.assign(cs.size(), 64);
    std::map<std::string, std::vector<size_t>> buckets;
    for (size_t i = 0; i < cs.size(); i++)
        buckets[autotune::bucket_key("f64", cs[i].m.total, cs[i].n.total, cs[i].k.total)].push_back(i);
    for (auto &kv : buckets) {
        int choice = 0;
        if (!autotune::lookup(kv.first, &choice)) {
            if (autotune::enabled()) {
                std::vector<Contraction> sample;
                for (size_t j = 0; j < kv.second.size() && j < 256; j++) sample.push_back(cs[kv.second[j]]);
                float t32 = 0, t64 = 0;
                eg_status st = time_f64(sample, 32, s, &t32);
                if (st != EG_SUCCESS) return st;
                if ((st = time_f64(sample, 64, s, &t64)) != EG_SUCCESS) return st;
                choice = t32 < t64 ? 32 : 64;
                autotune::store(kv.first, choice);
            } else {
                const Contraction &c = cs[kv.second[0]];
                choice = (c.m.total <= 48 || c.n.total <= 48) ? 32 : 64;
            }
        }
        for (size_t i : kv.second) tiles[i] = choice;
    }
    return EG_SUCCESS;
}

// Builds and captures the FP64 plan.
eg_status build_f64_plan(Plan &plan, const std::vector<Contraction> &cs, cudaStream_t s) {
    std::vector<int> tiles;
    eg_status st = choose_f64_tiles(cs, s, tiles);
    if (st != EG_SUCCESS) return st;
    std::vector<F64Item> items;
    for (auto &c : cs) items.push_back(f64_item(c));
    auto work = f64_work(cs, tiles);
    void *d_items, *d_tiles, *d_work;
    if ((st = dev_copy(plan, items.data(), items.size() * sizeof(F64Item), &d_items)) != EG_SUCCESS) return st;
    if ((st = dev_copy(plan, tiles.data(), tiles.size() * sizeof(int), &d_tiles)) != EG_SUCCESS) return st;
    if ((st = dev_copy(plan, work.data(), work.size() * sizeof(int4), &d_work)) != EG_SUCCESS) return st;
    const Contraction &c0 = cs[0];
    EG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    {
        CaptureGuard g;
        st = issue_f64((F64Item *)d_items, (int *)d_tiles, (int4 *)d_work, (int)work.size(), c0.cp, c0.ab,
                       c0.zero_when_cp_zero ? 1 : 0, s);
    }
    cudaGraph_t graph = nullptr;
    cudaError_t err = cudaStreamEndCapture(s, &graph);
    if (st != EG_SUCCESS) {
        if (graph) cudaGraphDestroy(graph);
        return st;
    }
    if (err != cudaSuccess) return cuda_fail(err, "cudaStreamEndCapture");
    plan.graph = graph;
    EG_CUDA(cudaGraphInstantiate(&plan.exec, graph, 0));
    plan.kernels = work.empty() ? 0 : 1;
    return EG_SUCCESS;
}

// Whether an FP64 list is worth the tensor cores (the FP64 form of split.cu's
// launch_f64_tensor, every item a tile or a few): from estimates of both times, the
// FMAs of 32 x 32 tiles at the FP64 pipe's rate against 30 us of launches, the splitting
// (28 bytes per element) and the tiles, each at least its chain of loads.  The digit
// planes stay below 1 GB; items with K below 8 or beyond the row-wise splitting keep the
// list on the FMA kernel.
bool f64_tensor_plan_pays(const std::vector<Contraction> &cs) {
    double fma = 0.0, bytes = 0.0, clocks = 0.0, planes = 0.0;
    for (const Contraction &c : cs) {
        const double nb = (double)c.batch.total, M = (double)c.m.total, N = (double)c.n.total, K = (double)c.k.total;
        if (c.k.total < 8 || c.k.total > kRowsMaxK || c.m.total >= (1ll << 31) || c.n.total >= (1ll << 31)) return false;
        fma += nb * std::ceil(M / 32) * std::ceil(N / 32) * 1024.0 * K;
        bytes += nb * (M + N) * K * 28.0;
        planes += nb * (M + N) * (K + 16) * 2.0 * (split::kF64Slices + 2);
        clocks += nb * std::ceil(M / 128) * std::ceil(N / 128) * (std::ceil(K / 64) * 38 * 420 + 16000);
    }
    const double sms = num_sms();
    const double t_fma = 1.1 * fma / (2.0 * sms * 1.9e9);
    const double t_tensor = 30e-6 + bytes / 2.2e12 + std::max(clocks / sms, 60000.0) / 1.9e9;
    return planes < 1e9 && t_tensor < 0.8 * t_fma;
}

// C = B A instead of A B, for an item whose tiles then end sooner: a tile's time is its
// epilogue's, that of the columns of one warp of each lane quadrant, whether or not its
// rows fill the four quadrants (30 x 100: 64 columns a warp, 100 x 30: 16).  The sums are
// exact either way, so the results are the same bits.  2048 uneven items in five
// slices: 557 -> 523 us, 512 in FP64: 328 -> 319.
int64_t warp_columns(int64_t n) { return n / 32 * 16 + std::min<int64_t>(n % 32, 16); }
Contraction better_side_first(const Contraction &c) {
    using namespace split;
    auto cost = [&](int64_t m, int64_t n) { return (m + kBM - 1) / kBM * warp_columns(n); };
    if (cost(c.n.total, c.m.total) >= cost(c.m.total, c.n.total)) return c;
    Contraction t = c;
    std::swap(t.A, t.B);
    std::swap(t.m, t.n);
    for (ModeGroup *g : {&t.batch, &t.m, &t.n, &t.k})
        for (int d = 0; d < g->n; d++) std::swap(g->s[0][d], g->s[1][d]);
    return t;
}

// Builds and captures the split-BF16 plan, or (f64) the FP64 one on the tensor cores;
// returns EG_ERROR_NOT_SUPPORTED when an item's K needs more than one exact pass (the
// caller then runs items one by one).
eg_status build_split_plan(Plan &plan, const std::vector<Contraction> &given, int slices, cudaStream_t s, bool f64) {
    using namespace split;
    std::vector<Contraction> cs;
    for (auto &c : given) cs.push_back(better_side_first(c));
    const int S = f64 ? kF64Slices : slices ? slices : 5, P = f64 ? S + 2 : S;
    if (!f64 && (S < 2 || S > kMaxSlices)) return fail(EG_ERROR_INVALID_ARGUMENT, "split form: slices must be in 2..6");
    plan.optional = f64; // (the FMA plan)
    const int64_t kmax = f64 ? kRowsMaxK : max_k_per_pass(S);
    int64_t elemsA = 0, elemsB = 0, rowsA = 0, rowsB = 0;
    for (auto &c : cs) {
        if (c.k.total > kmax) return fail(EG_ERROR_NOT_SUPPORTED, "grouped split: K above one exact pass");
        if (c.k.total <= 0) return fail(EG_ERROR_NOT_SUPPORTED, "grouped split: an item sums over no index");
        if (c.m.total >= (1ll << 31) || c.n.total >= (1ll << 31) || c.k.total >= (1ll << 31))
            return fail(EG_ERROR_NOT_SUPPORTED, "grouped split: extent above 2^31");
    }
    std::vector<GOp> opsA, opsB;
    std::vector<TcItem> items;
    std::vector<std::pair<int64_t, int4>> work;
    std::vector<int4> units; // (operand, batch index, first row); operands A then B of every item
    for (size_t i = 0; i < cs.size(); i++) {
        const Contraction &c = cs[i];
        const int64_t nb = c.batch.total, M = c.m.total, N = c.n.total, K = c.k.total;
        const int64_t Kp = round_up(K, kBK), Mp = round_up(M, kBM), Np = round_up(N, kBN);
        GOp a{};
        a.X = c.A;
        a.bg = c.batch;
        a.rg = c.m;
        a.kg = c.k;
        a.comp = 0;
        a.row_fast = !fast_along(c.k, 0) && fast_along(c.m, 0);
        a.nbatch = (int)nb;
        a.rows = M;
        a.Rp = Mp;
        a.K = K;
        a.Kp = Kp;
        a.rowbase = rowsA;
        // an item's planes are packed: its own rows, at a pitch of 32-byte multiples
        a.pitch = round_up(K, 16);
        a.pstride = M * a.pitch;
        a.plane0 = elemsA;
        a.sr = mode_group_affine_stride(c.m, 0);
        a.sk = mode_group_affine_stride(c.k, 0);
        GOp b = a;
        b.X = c.B;
        b.rg = c.n;
        b.comp = 1;
        b.row_fast = !fast_along(c.k, 1) && fast_along(c.n, 1);
        b.rows = N;
        b.Rp = Np;
        b.rowbase = rowsB;
        b.pstride = N * b.pitch;
        b.plane0 = elemsB;
        b.sr = mode_group_affine_stride(c.n, 1);
        b.sk = mode_group_affine_stride(c.k, 1);
        opsA.push_back(a);
        opsB.push_back(b);
        TcItem it{};
        it.C = c.C;
        it.M = M;
        it.N = N;
        it.nkb = (int)(Kp / kBK);
        it.eAoff = (int)rowsA;
        it.eBoff = (int)rowsB;
        it.Mp = (int)Mp;
        it.Np = (int)Np;
        it.bg = c.batch;
        it.mg = c.m;
        it.ng = c.n;
        it.tried = kTriedMean * (float)nb * (float)nb * (float)M * (float)N * (float)K * (float)K;
        items.push_back(it);
        for (int64_t bb = 0; bb < nb; bb++)
            for (int64_t x = 0; x < Mp / kBM; x++)
                for (int64_t y = 0; y < Np / kBN; y++)
                    work.push_back({Kp / kBK * 256 * (S * (S + 1) / 2) + 6000 +
                                        (f64 ? 700 : 350) * warp_columns(std::min<int64_t>(N - y * kBN, kBN)),
                                    make_int4((int)i, (int)bb, (int)x, (int)y)});
        rowsA += nb * Mp;
        rowsB += nb * Np;
        elemsA += round_up(nb * P * a.pstride, 64);
        elemsB += round_up(nb * P * b.pstride, 64);
    }
    if (rowsA >= (1ll << 31) || rowsB >= (1ll << 31))
        return fail(EG_ERROR_NOT_SUPPORTED, "grouped split: batch too large");
    std::stable_sort(work.begin(), work.end(), [](auto &x, auto &y) { return x.first > y.first; });
    // the tiles, the longest first, each to the CTA with the least to do (first: estimated
    // clocks of the MMAs and of the epilogue).  512 uneven items in FP64, dealt round in
    // that order: 222 us, of which the CTA with the longest first item took twice the mean;
    // 160 us so.
    const int grid = (int)std::min<size_t>(work.size(), (size_t)num_sms());
    std::vector<std::vector<int4>> of_cta(grid);
    std::priority_queue<std::pair<int64_t, int>, std::vector<std::pair<int64_t, int>>, std::greater<>> least;
    for (int c = 0; c < grid; c++) least.push({0, c});
    for (auto &w : work) {
        const auto [load, c] = least.top();
        least.pop();
        of_cta[c].push_back(w.second);
        least.push({load + w.first, c});
    }
    std::vector<int4> wl;
    std::vector<int> ranges(1, 0);
    for (auto &l : of_cta) {
        wl.insert(wl.end(), l.begin(), l.end());
        ranges.push_back((int)wl.size());
    }
    // one splitting unit per 32 real rows of every operand (and batch index)
    std::vector<GOp> ops(opsA);
    ops.insert(ops.end(), opsB.begin(), opsB.end());
    // row and K element offsets of every operand, fixed by the strides: built once here
    std::vector<long long> offs;
    for (auto &op : ops) {
        int64_t oa, ob, oc;
        op.rtab = (int64_t)offs.size();
        for (int64_t r = 0; r < op.rows && !op.sr; r++) { // (none where one stride serves)
            group_offsets(op.rg, r, oa, ob, oc);
            offs.push_back(op.comp ? ob : oa);
        }
        op.ktab = (int64_t)offs.size();
        for (int64_t k = 0; k < op.K && !op.sk; k++) {
            group_offsets(op.kg, k, oa, ob, oc);
            offs.push_back(op.comp ? ob : oa);
        }
    }
    int64_t Kmax = 0;
    for (const auto &op : ops) Kmax = std::max(Kmax, op.K);
    const bool by_rows = Kmax <= kRowsMaxK;
    size_t rows_smem = 0;
    for (size_t i = 0; i < ops.size(); i++) {
        int R = 32;
        if (by_rows) {
            while (R > 4 && (int64_t)R * ops[i].K > kRowsElems) R /= 2;
            rows_smem = std::max(rows_smem, (size_t)R * rows_ld(ops[i].K) * 16); // two tiles
        }
        for (int64_t bb = 0; bb < ops[i].nbatch; bb++)
            for (int64_t r0 = 0; r0 < ops[i].rows; r0 += R) units.push_back(make_int4((int)i, (int)bb, (int)r0, R));
    }
    if (units.size() >= (size_t)INT_MAX) return fail(EG_ERROR_NOT_SUPPORTED, "grouped split: batch too large");

    void *planesA, *planesB, *eA, *eB, *d_ops, *d_units, *d_offs, *d_items, *d_work, *rbuf;
    eg_status st;
    if ((st = dev_alloc(plan, rbuf_bytes(f64 ? 3 : 1), &rbuf)) != EG_SUCCESS) return st;
    const size_t pbytesA = (size_t)elemsA * 2, pbytesB = (size_t)elemsB * 2;
    if ((st = dev_alloc(plan, pbytesA, &planesA)) != EG_SUCCESS) return st;
    if ((st = dev_alloc(plan, pbytesB, &planesB)) != EG_SUCCESS) return st;
    if ((st = dev_alloc(plan, (size_t)rowsA * 4, &eA)) != EG_SUCCESS) return st;
    if ((st = dev_alloc(plan, (size_t)rowsB * 4, &eB)) != EG_SUCCESS) return st;
    // the exponents of padded rows are never written: zero them once
    EG_CUDA(cudaMemsetAsync(eA, 0, (size_t)rowsA * 4, s));
    EG_CUDA(cudaMemsetAsync(eB, 0, (size_t)rowsB * 4, s));
    if ((st = dev_copy(plan, ops.data(), ops.size() * sizeof(GOp), &d_ops)) != EG_SUCCESS) return st;
    // cleared by every replay: the counts of the blocks left out and of their tiles handed out,
    // the record of a wait that gave up, and in the FP64 form from byte 16 on two sums an item
    void *redo_count = nullptr;
    const size_t counts = 16 + (f64 ? items.size() * 16 : 0);
    if ((st = dev_alloc(plan, counts, &redo_count)) != EG_SUCCESS) return st;
    unsigned long long *magnitudes = f64 ? (unsigned long long *)redo_count + 2 : nullptr;
    if (by_rows) {
        std::vector<RowsUnit> rows;
        rows.reserve(units.size());
        for (const int4 &u : units) {
            const GOp &g = ops[u.x];
            int64_t oa, ob, oc;
            group_offsets(g.bg, u.y, oa, ob, oc);
            const int64_t r0 = u.z;
            RowsUnit x{};
            x.X = g.X + pick(g.comp, oa, ob) + (g.sr ? r0 * g.sr : 0);
            x.planes = (__nv_bfloat16 *)(g.comp ? planesB : planesA) + g.plane0 + u.y * P * g.pstride + r0 * g.pitch;
            x.rexp = (int *)(g.comp ? eB : eA) + g.rowbase + u.y * g.Rp + r0;
            if (f64) x.magnitudes = magnitudes + (size_t)u.x % items.size() * 2 + (g.comp ? 1 : 0);
            x.sr = g.sr;
            x.sk = g.sk;
            x.rtab = g.rtab + r0;
            x.ktab = g.ktab;
            x.pitch = g.pitch;
            x.pstride = g.pstride;
            x.K = (int)g.K;
            x.R = u.w;
            x.rows = (int)std::min<int64_t>(g.rows - r0, u.w);
            x.flags = g.row_fast ? 1 : 0;
            rows.push_back(x);
        }
        st = dev_copy(plan, rows.data(), rows.size() * sizeof(RowsUnit), &d_units);
    } else {
        st = dev_copy(plan, units.data(), units.size() * sizeof(int4), &d_units);
    }
    if (st != EG_SUCCESS) return st;
    if ((st = dev_copy(plan, offs.data(), offs.size() * sizeof(long long), &d_offs)) != EG_SUCCESS) return st;
    if ((st = dev_copy(plan, items.data(), items.size() * sizeof(TcItem), &d_items)) != EG_SUCCESS) return st;
    if ((st = dev_copy(plan, wl.data(), wl.size() * sizeof(int4), &d_work)) != EG_SUCCESS) return st;
    void *d_ranges = nullptr;
    if ((st = dev_copy(plan, ranges.data(), ranges.size() * sizeof(int), &d_ranges)) != EG_SUCCESS) return st;

    // per-item maps: each item's planes with its own M (N) and K as the extents
    std::vector<CUtensorMap> maps(2 * items.size());
    for (size_t i = 0; i < items.size(); i++) {
        const TcItem &it = items[i];
        const Contraction &c = cs[i];
        if (it.M == 0 || it.N == 0 || c.batch.total == 0) continue; // no tiles: the maps are never used
        const int64_t planes = c.batch.total * P, K = c.k.total;
        if ((st = encode_planes_extent(&maps[2 * i], (__nv_bfloat16 *)planesA + opsA[i].plane0, K, it.M, planes,
                                       opsA[i].pitch, it.M)) != EG_SUCCESS)
            return st;
        if ((st = encode_planes_extent(&maps[2 * i + 1], (__nv_bfloat16 *)planesB + opsB[i].plane0, K, it.N, planes,
                                       opsB[i].pitch, it.N)) != EG_SUCCESS)
            return st;
    }
    void *d_maps = nullptr;
    if ((st = dev_copy(plan, maps.data(), maps.size() * sizeof(CUtensorMap), &d_maps)) != EG_SUCCESS) return st;
    if ((st = status_word(s, &plan.status_on)) != EG_SUCCESS) return st;
    void *status_at = nullptr;
    if ((st = dev_copy(plan, &plan.status_on, sizeof(int *), &status_at)) != EG_SUCCESS) return st;
    plan.status_at = (int **)status_at;

    const Contraction &c0 = cs[0];
    TcGemmParams p{};
    p.S = S;
    p.planes = P;
    p.nbatch = 1;
    p.cp = c0.cp;
    p.ab = c0.ab;
    p.zero = c0.zero_when_cp_zero ? 1 : 0;
    p.eA = (int *)eA;
    p.eB = (int *)eB;
    p.shift_const = -2 * kTopBits - kBits * (S - 1);
    {
        int k = 0;
        const double f = std::frexp(std::fabs(c0.ab), &k);
        p.ab_pow2 = (f == 0.5) ? 1 : 0;
        p.ab_neg = (p.ab_pow2 && c0.ab < 0) ? 1 : 0;
        if (p.ab_pow2) p.shift_const += k - 1;
    }
    p.status_at = plan.status_at;
    p.lost = (int *)redo_count + 2;
    p.timeout_ns = 2000ull * 1000 * 1000;
    p.d0 = 0; // every slice group in one launch (K fits one exact pass)
    p.d1 = S;
    p.t0 = INT_MAX; // no K slicing in grouped launches
    p.ksplit = 1;
    p.kslice = 0;
    p.item_maps = (const CUtensorMap *)d_maps;
    p.ranges = (const int *)d_ranges;
    p.rbuf = (long long *)rbuf;
    static const bool prof_on = std::getenv("EINSUMS_GB300_TC_PROFILE") != nullptr;
    if (prof_on) {
        // per-role cycle counters summed over the plan's replays, printed when it is destroyed
        void *prof = nullptr;
        const size_t pbytes = (size_t)num_sms() * 8 * sizeof(unsigned long long);
        if ((st = dev_alloc(plan, pbytes, &prof)) != EG_SUCCESS) return st;
        EG_CUDA(cudaMemsetAsync(prof, 0, pbytes, s));
        p.prof = (unsigned long long *)prof;
        plan.prof = p.prof;
    }

    if ((st = ensure_tc_attributes()) != EG_SUCCESS) return st;
    if (by_rows) EG_CUDA(allow_grouped_rows(S, f64));
    void *d_fma = nullptr, *redo = nullptr;
    if (f64) {
        std::vector<F64Item> fma;
        for (auto &c : cs) fma.push_back(f64_item(c));
        if ((st = dev_copy(plan, fma.data(), fma.size() * sizeof(F64Item), &d_fma)) != EG_SUCCESS) return st;
        if ((st = dev_alloc(plan, wl.size() * kTileRegions * sizeof(int4), &redo)) != EG_SUCCESS) return st;
        p.hid = kF64High;
        p.redo = (int4 *)redo;
        p.redo_count = (int *)redo_count;
        p.magnitudes = magnitudes;
    }
    EG_CUDA(cudaEventCreateWithFlags(&plan.last, cudaEventDisableTiming));
    EG_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    {
        CaptureGuard g;
        auto issue = [&]() -> eg_status {
            EG_CUDA(cudaMemsetAsync(redo_count, 0, counts, s));
            eg_status is = inject_lost(p.lost, s);
            if (is != EG_SUCCESS) return is;
            is =
                by_rows ? launch_grouped_rows(S, f64, (const RowsUnit *)d_units, (int)units.size(),
                                              (const long long *)d_offs, rows_smem, s)
                        : launch_grouped_split(S, (const GOp *)d_ops, (const int4 *)d_units, (int)units.size(),
                                               (const long long *)d_offs, (int *)eA, (int *)eB, (__nv_bfloat16 *)planesA,
                                               (__nv_bfloat16 *)planesB, s);
            if (is != EG_SUCCESS) return is;
            is = launch_tc_gemm_grouped(maps[0], maps[1], p, (TcItem *)d_items, (int4 *)d_work, grid, s);
            if (is != EG_SUCCESS || !f64) return is;
            k_grouped_f64_listed<<<num_sms() * 8, f64::kThreads, 0, s>>>((const F64Item *)d_fma, (const int4 *)redo,
                                                                   (int *)redo_count, c0.cp, c0.ab, p.zero, p.status_at,
                                                                   (const int4 *)d_work, (int)wl.size());
            EG_CHECK_LAUNCH("k_grouped_f64_listed");
            return EG_SUCCESS;
        };
        st = issue();
    }
    cudaGraph_t graph = nullptr;
    cudaError_t err = cudaStreamEndCapture(s, &graph);
    if (st != EG_SUCCESS) {
        if (graph) cudaGraphDestroy(graph);
        return st;
    }
    if (err != cudaSuccess) return cuda_fail(err, "cudaStreamEndCapture");
    plan.graph = graph;
    EG_CUDA(cudaGraphInstantiate(&plan.exec, graph, 0));
    plan.kernels = f64 ? 3 : 2;
    if (!f64) plan.report = eg_split_report{S, S * (S + 1) / 2, kBits, error_bound(S)};
    return EG_SUCCESS;
}

} // namespace eg::grouped
