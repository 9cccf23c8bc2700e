// Host orchestration of the split-BF16 form, of plain FP64 on the tensor cores
// (launch_f64_tensor) and of their digit-splitting kernels.
//
//   k_split_rows     row maxima, exponents and digit planes of both operands in one
//                    launch that reads every element once, for K up to about 25000;
//                    beyond, passes over each operand:
//   k_split_rowmax   max |x| of every operand row (atomicMax on the bit
//                    pattern of |x|, which orders like the value; deterministic)
//   k_split_exponent row exponent e with |x| < 2^e (INT_MIN for a row holding
//                    Inf/NaN, whose outputs are written as NaN)
//   k_split_digits   32x64 tiles staged through shared memory (double-buffered
//                    asynchronous copies) so the operand is read along its
//                    contiguous mode and the digit planes are written along k;
//                    padding rows/columns are written as 0
// then the tcgen05 GEMM (tc_gemm.cu) over the digit planes.  The operands'
// index permutation is folded into the address maps of these kernels and of
// the GEMM epilogue: nothing but the BF16 digit planes is materialised.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "ptx.cuh"
#include "split.cuh"

namespace eg {
void set_split_report(const eg_split_report &r);
}

namespace eg::split {

namespace {

// Operand view for the splitting kernels: rows (batch x row group) and k.
struct OperandMap {
    ModeGroup bg, rg, kg;
    int comp;          // stride component: 0 for A, 1 for B
    int64_t rows, Rp;  // logical and padded rows per batch
    int64_t K, Kp;
    int nbatch;
    // Element offsets of every row and every k (filled by k_operand_offsets),
    // or null: then each offset is decomposed mode by mode, which costs integer
    // divisions per element and made these kernels ALU-bound.
    const int64_t *offr = nullptr, *offk = nullptr;
    // When a group walks memory with a single stride (the usual case: its modes
    // are nested like a row-major block), that stride; the offset is then
    // index * stride, with no table load in the dependency chain.  0 otherwise.
    int64_t sr = 0, sk = 0;
    // First batch index and row of the panel being split (rows, nbatch count from there).
    int64_t b0 = 0, row0 = 0;
};

__device__ __forceinline__ int64_t comp_of(int comp, int64_t oa, int64_t ob) { return comp == 0 ? oa : ob; }

__device__ __forceinline__ int64_t off_b(const OperandMap &m, int64_t b) {
    if (m.bg.n == 0) return 0;
    int64_t oa, ob, oc;
    group_offsets(m.bg, m.b0 + b, oa, ob, oc);
    return comp_of(m.comp, oa, ob);
}
__device__ __forceinline__ int64_t decompose_r(const OperandMap &m, int64_t r) {
    int64_t oa, ob, oc;
    group_offsets32(m.rg, (uint32_t)(m.row0 + r), oa, ob, oc);
    return comp_of(m.comp, oa, ob);
}
__device__ __forceinline__ int64_t decompose_k(const OperandMap &m, int64_t k) {
    int64_t oa, ob, oc;
    group_offsets32(m.kg, (uint32_t)k, oa, ob, oc);
    return comp_of(m.comp, oa, ob);
}
__device__ __forceinline__ int64_t off_r(const OperandMap &m, int64_t r) {
    if (m.sr) return (m.row0 + r) * m.sr;
    return m.offr ? __ldg(m.offr + r) : decompose_r(m, r);
}
__device__ __forceinline__ int64_t off_k(const OperandMap &m, int64_t k) {
    if (m.sk) return k * m.sk;
    return m.offk ? __ldg(m.offk + k) : decompose_k(m, k);
}

// Fills the row and k offset tables of an operand.
__global__ void k_operand_offsets(OperandMap m, int64_t *offr, int64_t *offk) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m.rows; i += stride) offr[i] = decompose_r(m, i);
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m.K; i += stride) offk[i] = decompose_k(m, i);
}

constexpr int T = 32, TR = 8;

// Splits a work index w = (b * n1 + i1) * n0 + i0 into its parts, in 32-bit
// arithmetic when the work count fits (`narrow`): a 64-bit division is a long
// subroutine, and the splitting kernels pay this once per work unit.
__device__ __forceinline__ void split_unit(int64_t w, int64_t n0, int64_t n1, bool narrow, int64_t &i0, int64_t &i1,
                                           int64_t &b) {
    if (narrow) {
        const uint32_t x = (uint32_t)w, a = (uint32_t)n0, c = (uint32_t)n1;
        const uint32_t q = x / a, q2 = q / c;
        i0 = x - q * a;
        i1 = q - q2 * c;
        b = q2;
    } else {
        const int64_t q = w / n0, q2 = q / n1;
        i0 = w - q * n0;
        i1 = q - q2 * n1;
        b = q2;
    }
}

// Row maxima over work units of rows x kchunk k (kchunk a multiple of T), the
// k loop inside the unit so that the unit's decomposition, batch offset and
// row offsets are paid once per unit; one atomicMax per row per unit.
//
// row_fast (the operand is contiguous along rows): a unit is 256 rows, one per
// thread, each thread walking all k of the chunk for its row with 8 loads in
// flight.  A CTA's eight warps read 2 KB contiguous at each k, and consecutive
// units are consecutive row blocks at the same k range; no reduction between
// threads is needed.  Otherwise (contiguous along k): a unit is 32 rows, lanes
// walk k and each warp reduces its 4 rows with shuffles at the unit's end.
constexpr int kRowFastBatch = 8;   // loads a thread keeps in flight when it walks one row
constexpr int kRowFastRows = T * TR; // rows of a unit when the operand is contiguous along rows
__global__ void __launch_bounds__(T *TR, 5) k_split_rowmax(OperandMap m, const double *__restrict__ X,
                                                        unsigned long long *rowmax, int row_fast, int kchunk) {
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t rows_per_unit = row_fast ? kRowFastRows : T;
    const int64_t rt = (m.rows + rows_per_unit - 1) / rows_per_unit, kcs = (m.K + kchunk - 1) / kchunk;
    const int64_t units = (int64_t)m.nbatch * rt * kcs;
    const bool narrow = units < INT_MAX;
    for (int64_t u = blockIdx.x; u < units; u += gridDim.x) {
        int64_t i0, i1, b;
        split_unit(u, row_fast ? rt : kcs, row_fast ? kcs : rt, narrow, i0, i1, b);
        const int64_t kc = row_fast ? i1 : i0, rtile = row_fast ? i0 : i1;
        const int64_t ob = off_b(m, b);
        const int64_t r0 = rtile * rows_per_unit;
        const int64_t kbeg = kc * kchunk, kend = min(m.K, kbeg + kchunk);
        if (row_fast) {
            const int64_t r = r0 + ty * T + tx;
            if (r < m.rows) {
                const double *xr = X + ob + off_r(m, r);
                unsigned long long mx = 0;
                int64_t k = kbeg;
                for (; k + kRowFastBatch <= kend; k += kRowFastBatch) {
                    unsigned long long v[kRowFastBatch];
#pragma unroll
                    for (int i = 0; i < kRowFastBatch; i++) v[i] = abs_bits(__ldg(xr + off_k(m, k + i)));
#pragma unroll
                    for (int i = 0; i < kRowFastBatch; i++) mx = max(mx, v[i]);
                }
                for (; k < kend; k++) mx = max(mx, abs_bits(__ldg(xr + off_k(m, k))));
                if (mx) atomicMax(rowmax + b * m.Rp + r, mx);
            }
        } else {
            // thread (tx, ty): rows r0+ty, +8, ...; k = kbeg+tx, +32, ...; warp reduce along k
            constexpr int RPT = T / TR;
            const double *xr[RPT];
            unsigned long long mx[RPT];
#pragma unroll
            for (int j = 0; j < RPT; j++) {
                const int64_t r = r0 + ty + TR * j;
                xr[j] = r < m.rows ? X + ob + off_r(m, r) : nullptr;
                mx[j] = 0;
            }
#pragma unroll 2
            for (int64_t k = kbeg + tx; k < kend; k += T) {
                const int64_t okk = off_k(m, k);
#pragma unroll
                for (int j = 0; j < RPT; j++)
                    if (xr[j]) mx[j] = max(mx[j], abs_bits(__ldg(xr[j] + okk)));
            }
#pragma unroll
            for (int j = 0; j < RPT; j++) {
                unsigned long long v = mx[j];
                for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
                const int64_t r = r0 + ty + TR * j;
                if (tx == 0 && r < m.rows && v) atomicMax(rowmax + b * m.Rp + r, v);
            }
        }
    }
}

__global__ void k_split_exponent(const unsigned long long *rowmax, int *e, int64_t n) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        e[i] = row_exponent(rowmax[i]);
}

// Tiles of 32 rows x 64 k staged through shared memory so that the operand is
// read along its contiguous mode; each thread then converts two consecutive k
// of a row and writes them as one BF16 pair per digit plane (a warp stores 128
// contiguous bytes per plane).  Padding rows and columns are written as 0.
//
// A work unit is a strip of up to kDigitStrip k tiles of one 32-row tile, so
// that the unit's decomposition, exponents and row offsets are paid per strip.
// Consecutive units walk the operand's contiguous mode: k strips of one row
// tile, or (row_fast) row tiles of one k strip.  Within a strip the tiles are
// double-buffered: asynchronous copies (cp.async, zero-filled outside the
// operand) bring tile t+1 into shared memory while tile t is converted.
constexpr int TK = 2 * T;
constexpr int64_t kDigitStrip = 8; // k tiles per work unit
template <int S, bool CHECK>
__global__ void __launch_bounds__(T *TR) k_split_digits(OperandMap m, const double *__restrict__ X, const int *rexp,
                                                        __nv_bfloat16 *planes, int row_fast) {
    __shared__ double tile[2][T][TK + 1];
    __shared__ int ex[T];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int64_t rt = m.Rp / T, kt = m.Kp / TK, segs = (kt + kDigitStrip - 1) / kDigitStrip;
    const int64_t work = (int64_t)m.nbatch * rt * segs;
    const bool narrow = work < INT_MAX;
    const int64_t plane = m.Rp * m.Kp;
    constexpr int RPT = T / TR;
    for (int64_t w = blockIdx.x; w < work; w += gridDim.x) {
        int64_t i0, i1, b;
        split_unit(w, row_fast ? rt : segs, row_fast ? segs : rt, narrow, i0, i1, b);
        const int64_t sg = row_fast ? i1 : i0, rtile = row_fast ? i0 : i1;
        const int64_t ob = off_b(m, b);
        const int64_t r0 = rtile * T;
        __syncthreads(); // the previous strip's last reads of ex[] and of the tiles are done
        if (ty == 0) ex[tx] = (r0 + tx < m.rows) ? rexp[b * m.Rp + r0 + tx] : 0;
        const double *xr[RPT]; // row_fast: row r0+tx in xr[0]; else rows r0+ty+8j
#pragma unroll
        for (int j = 0; j < RPT; j++) {
            const int64_t r = row_fast ? (j == 0 ? r0 + tx : m.rows) : r0 + ty + TR * j;
            xr[j] = r < m.rows ? X + ob + off_r(m, r) : nullptr;
        }
        auto load_tile = [&](int buf, int64_t k0) {
            if (row_fast) {
#pragma unroll
                for (int j = ty; j < TK; j += TR) {
                    const int64_t k = k0 + j;
                    const bool ok = xr[0] && k < m.K;
                    ptx::cp_async8(&tile[buf][tx][j], ok ? xr[0] + off_k(m, k) : X, ok);
                }
            } else {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int64_t k = k0 + h * T + tx;
                    const bool kin = k < m.K;
                    const int64_t okk = kin ? off_k(m, k) : 0;
#pragma unroll
                    for (int j = 0; j < RPT; j++) {
                        const bool ok = xr[j] && kin;
                        ptx::cp_async8(&tile[buf][ty + TR * j][h * T + tx], ok ? xr[j] + okk : X, ok);
                    }
                }
            }
            ptx::cp_async_commit();
        };
        const int64_t kt_beg = sg * kDigitStrip, kt_end = min(kt, (sg + 1) * kDigitStrip);
        load_tile(0, kt_beg * TK);
        for (int64_t ktile = kt_beg; ktile < kt_end; ktile++) {
            const int cur = (int)((ktile - kt_beg) & 1);
            const int64_t k0 = ktile * TK;
            if (ktile + 1 < kt_end) {
                load_tile(cur ^ 1, k0 + TK);
                ptx::cp_async_wait<1>();
            } else {
                ptx::cp_async_wait<0>();
            }
            __syncthreads();
            // write: thread tx converts k0 + 2tx and k0 + 2tx + 1 of each of its rows
#pragma unroll
            for (int j = ty; j < T; j += TR) {
                const int64_t r = r0 + j;
                constexpr int P = S + (CHECK ? 2 : 0);
                uint32_t pk[P];
                const int e = ex[j];
                const double x0 = tile[cur][j][2 * tx], x1 = tile[cur][j][2 * tx + 1];
                if (e == INT_MIN) {
#pragma unroll
                    for (int s = 0; s < P; s++) pk[s] = 0u;
                } else {
                    digits_bf16x2<S>(x0, x1, e, pk);
                    if constexpr (CHECK) pk[S] = check_magnitude(pk[0]);
                }
                if constexpr (CHECK) pk[S + 1] = check_mark(x0, x1);
                uint32_t *out = (uint32_t *)(planes + ((int64_t)b * P) * plane + r * m.Kp + k0) + tx;
#pragma unroll
                for (int s = 0; s < P; s++) out[(int64_t)s * (plane / 2)] = pk[s];
            }
            __syncthreads();
        }
    }
}

// Row maxima, exponents and digit planes of both operands in one launch that reads
// every element once: a cluster of C CTAs takes R rows, each CTA a range of kc of
// the K elements, which it holds in shared memory (asynchronous 8-byte copies, all
// in flight at once); the CTAs' row maxima meet over distributed shared memory, and
// each writes its range of the digit planes.  Bound: memory, 8 bytes read and 2 per
// plane written per element.  Against the passes above (memset, maxima, exponents,
// digits for each operand, with every element read twice): see split_both.
struct SplitJob {
    OperandMap m;
    const double *X;
    int *rexp;
    __nv_bfloat16 *planes;
    int row_fast;  // consecutive lanes walk rows (the smaller stride), else k
    int pairs;     // (k, k + 1) with even k are neighbours on a 16-byte boundary in every row
    int64_t tiles; // batches x R-row tiles
    int sample;    // every so-manieth tile's magnitudes are added up
};

constexpr int kFusedThreads = 256;

template <int S, bool CHECK, int R>
__global__ void __launch_bounds__(kFusedThreads) k_split_rows(const __grid_constant__ SplitJob ja,
                                                              const __grid_constant__ SplitJob jb, int kc, int ld,
                                                              int C, int *clear, unsigned long long *magnitudes) {
    extern __shared__ __align__(16) double tile[]; // [R][ld], then the tables
    int64_t *koff = (int64_t *)(tile + (size_t)R * ld);
    int64_t *roff = koff + kc;
    unsigned long long *pmax = (unsigned long long *)(roff + R);
    int *ex = (int *)(pmax + R);
    constexpr int W = kFusedThreads / 32, P = S + (CHECK ? 2 : 0);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (clear && blockIdx.x == 0 && tid < kListWords) clear[tid] = 0; // words of the kernels that follow
    const int64_t id = blockIdx.x / C;
    const int rank = C > 1 ? (int)ptx::cluster_ctarank() : 0;
    const bool second = id >= ja.tiles;
    const SplitJob &jj = second ? jb : ja;
    const OperandMap &m = jj.m;
    const int64_t t = second ? id - ja.tiles : id, rt = m.Rp / R;
    const int64_t b = t / rt, r0 = (t - b * rt) * R;
    const int64_t k0 = (int64_t)rank * kc;
    const int nk = (int)max((int64_t)0, min((int64_t)kc, m.K - k0)); // real elements of this CTA's range
    const int64_t ob = off_b(m, b);
    if (!m.sk)
        for (int k = tid; k < nk; k += kFusedThreads) koff[k] = off_k(m, k0 + k);
    if (tid < R) roff[tid] = r0 + tid < m.rows ? ob + off_r(m, r0 + tid) : -1;
    __syncthreads();
    // k, k + step, ... of row r: copies of the real elements, then zeros (a single k
    // stride is added up: the loop is two copies for it)
    auto row_copy = [&](int r, int k, int step) {
        const int64_t ro = roff[r];
        double *t = tile + r * ld;
        if (ro >= 0) {
            const double *x = jj.X + ro;
            if (m.sk) {
                const int64_t inc = (int64_t)step * m.sk;
                x += (k0 + k) * m.sk;
#pragma unroll 4
                for (; k < nk; k += step, x += inc) ptx::cp_async8(t + k, x);
            } else {
#pragma unroll 4
                for (; k < nk; k += step) ptx::cp_async8(t + k, x + koff[k]);
            }
        }
        for (; k < kc; k += step) t[k] = 0.0;
    };
    if (jj.row_fast) {
        constexpr int KP = 32 / R; // k a warp takes at a time
        row_copy(lane % R, warp * KP + lane / R, W * KP);
    } else if (jj.pairs) {
        for (int r = warp; r < R; r += W) {
            const int64_t ro = roff[r];
            double *t = tile + r * ld;
            int k = 2 * lane; // the real elements are even in number
            if (ro >= 0) {
                const double *x = jj.X + ro;
#pragma unroll 4
                for (; k < nk; k += 64) ptx::cp_async16(t + k, x + (m.sk ? k0 + k : koff[k]));
            }
            for (; k < kc; k += 64) t[k] = t[k + 1] = 0.0;
        }
    } else {
        for (int r = warp; r < R; r += W) row_copy(r, lane, 32);
    }
    ptx::cp_async_commit();
    ptx::cp_async_wait<0>();
    __syncthreads();
    for (int r = warp; r < R; r += W) {
        const unsigned long long mx = row_max_bits(tile + r * ld, kc, lane);
        if (lane == 0) pmax[r] = mx;
    }
    if (C > 1)
        ptx::cluster_sync();
    else
        __syncthreads();
    if (tid < R) {
        unsigned long long mx = pmax[tid];
        for (int c = 1; c < C; c++) {
            const int peer = rank + c < C ? rank + c : rank + c - C;
            mx = max(mx, ptx::ld_cluster_u64(ptx::mapa(ptx::smem_u32(&pmax[tid]), (uint32_t)peer)));
        }
        const int e = row_exponent(mx);
        ex[tid] = e;
        if (rank == 0) jj.rexp[b * m.Rp + r0 + tid] = e;
    }
    if (C > 1)
        ptx::cluster_sync(); // the peers have read this CTA's maxima
    else
        __syncthreads();
    if constexpr (CHECK) {
        // The magnitudes of eight rows of some 32 tiles of each operand are added up, from the bits
        // and apart from the digits.  (Of all rows, from the digits: 64 registers instead of 40,
        // and n = 75 transformations 3560 us, not 3410.)
        if (magnitudes && (uint32_t)t % (uint32_t)jj.sample == 0) {
            unsigned leading = 0, nonzero = 0;
            const int e = ex[warp];
#pragma unroll 2
            for (int k = lane; k < nk && e != INT_MIN; k += 32) {
                const uint32_t hi = (uint32_t)(abs_bits(tile[warp * ld + k]) >> 32);
                const int down = e + 1022 - (int)(hi >> 20); // of the leading bit, below the row's bound
                leading += down <= 6 ? max((int)((0x100000u | (hi & 0xFFFFFu)) >> (14 + down)), 1) - 1 : 0;
                nonzero += hi != 0 ? 1 : 0;
            }
            leading = __reduce_add_sync(0xffffffffu, leading);
            nonzero = __reduce_add_sync(0xffffffffu, nonzero);
            if (lane < 2) atomicAdd(magnitudes + (second ? 2 : 0) + lane, (unsigned long long)(lane ? nonzero : leading));
        }
    }
    const int64_t plane = m.Rp * m.Kp;
    const int kw = (int)max((int64_t)0, min((int64_t)kc, m.Kp - k0)); // range written, a multiple of 4
    // four elements a thread, rows one after the other: a warp runs across the ends of rows,
    // so that rows of few elements keep all lanes busy (a row to a warp at a time left 12 of
    // 32 idle at K = 75)
    const int quads = kw / 4;
    __nv_bfloat16 *const first = jj.planes + (int64_t)b * P * plane + r0 * m.Kp + k0;
    int r = tid / max(quads, 1), k = tid - r * quads;
    const int dr = kFusedThreads / max(quads, 1), dk = kFusedThreads - dr * quads;
    for (int i = tid; i < R * quads; i += kFusedThreads) {
        const double *x = tile + r * ld + 4 * k;
        const double2 v0 = *(const double2 *)x, v1 = *(const double2 *)(x + 2);
        uint32_t p0[P], p1[P];
        const int e = ex[r];
        if (e == INT_MIN) {
#pragma unroll
            for (int s = 0; s < P; s++) p0[s] = p1[s] = 0u;
        } else {
            digits_bf16x2<S>(v0.x, v0.y, e, p0);
            digits_bf16x2<S>(v1.x, v1.y, e, p1);
            if constexpr (CHECK) {
                p0[S] = check_magnitude(p0[0]);
                p1[S] = check_magnitude(p1[0]);
            }
        }
        if constexpr (CHECK) {
            p0[S + 1] = check_mark(v0.x, v0.y);
            p1[S + 1] = check_mark(v1.x, v1.y);
        }
        __nv_bfloat16 *row = first + r * m.Kp + 4 * k;
#pragma unroll
        for (int s = 0; s < P; s++) *(uint2 *)(row + s * plane) = make_uint2(p0[s], p1[s]);
        r += dr;
        k += dk;
        if (k >= quads) {
            k -= quads;
            r++;
        }
    }
}

// CTAs of `kernel` (256 threads, static shared memory) that fit on the GPU at
// once: the splitting kernels launch exactly one wave of them and loop over
// their work units, so no partial second wave trails the launch.
template <typename F>
int resident_grid(F kernel) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, T * TR, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
    return per_sm * num_sms();
}

// K chunk (a multiple of `gran`) for `row_units` row blocks: among splits into
// about one to four units per resident CTA, the one whose last wave of units is
// fullest (the fewest units when two are about as full).
int balanced_chunk(int64_t row_units, int64_t K, int64_t resident, int gran) {
    const int64_t ktiles = std::max<int64_t>(1, (K + gran - 1) / gran);
    row_units = std::max<int64_t>(1, row_units);
    int64_t best_tiles = ktiles;
    double best_eff = -1.0;
    for (int per = 1; per <= 4; per++) {
        const int64_t want = std::min(ktiles, std::max<int64_t>(1, resident * per / row_units));
        const int64_t tiles = (ktiles + want - 1) / want; // tiles of `gran` k per chunk
        const int64_t units = row_units * ((ktiles + tiles - 1) / tiles);
        const int64_t waves = (units + resident - 1) / resident;
        const double eff = (double)units / (double)(waves * resident);
        if (eff > best_eff + 0.02) {
            best_eff = eff;
            best_tiles = tiles;
        }
    }
    return (int)(best_tiles * gran);
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

// 3-D map over [planes][rows][Kp] BF16 (zeros beyond Kp), box 64 (k) x box_rows rows x 1, 128-byte swizzle.
eg_status encode_planes(CUtensorMap *map, void *base, int64_t Kp, int64_t rows, int64_t planes, int box_rows = kBM) {
    auto fn = encode_fn();
    if (!fn) return fail(EG_ERROR_CUDA, "cuTensorMapEncodeTiled is unavailable");
    cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)(Kp * 2), (cuuint64_t)(Kp * 2 * rows)};
    cuuint32_t box[3] = {(cuuint32_t)kBK, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(EG_ERROR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return EG_SUCCESS;
}

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

bool is_fast(const ModeGroup &g, int comp) { return g.n > 0 && g.s[comp][g.n - 1] == 1; }

// The single stride of a group whose modes (extent-1 modes ignored) nest like a
// row-major block in operand `comp`, else 0.
int64_t affine_stride(const ModeGroup &g, int comp) {
    int64_t stride = 0, span = 0; // stride of the fastest mode seen, and stride * extents so far
    for (int d = g.n - 1; d >= 0; d--) {
        if (g.ext[d] == 1) continue;
        const int64_t sd = g.s[comp][d];
        if (stride == 0) {
            if (sd == 0) return 0;
            stride = sd;
            span = sd * g.ext[d];
        } else {
            if (sd != span) return 0;
            span = sd * g.ext[d];
        }
    }
    return stride == 0 ? 1 : stride; // no mode of extent > 1: the group has one index, offset 0
}

eg_status split_operand(OperandMap om, const double *X, unsigned long long *rowmax, int *rexp,
                        __nv_bfloat16 *planes, int S, cudaStream_t s, int64_t *offr, int64_t *offk,
                        bool f64 = false) {
    const bool k_fast = is_fast(om.kg, om.comp);
    om.sr = affine_stride(om.rg, om.comp);
    om.sk = affine_stride(om.kg, om.comp);
    if (om.sr && om.sk) offr = offk = nullptr; // no tables needed
    if (offr && offk) {
        const int64_t n = std::max(om.rows, om.K);
        {
            LaunchScope ls_("k_operand_offsets", s);
            k_operand_offsets<<<(int)std::min<int64_t>((n + 255) / 256, (int64_t)num_sms() * 8), 256, 0, s>>>(om, offr,
                                                                                                            offk);
        }
        EG_CHECK_LAUNCH("k_operand_offsets");
        om.offr = offr;
        om.offk = offk;
    }
    const bool r_fast = !k_fast && is_fast(om.rg, om.comp);
    EG_CUDA(cudaMemsetAsync(rowmax, 0, (size_t)om.nbatch * om.Rp * sizeof(unsigned long long), s));
    const int cap = num_sms() * 8;
    {
        static PerDevice<int> grids;
        const int resident = grids.get(current_device(), [] { return resident_grid(k_split_rowmax); });
        const int64_t unit_rows = r_fast ? kRowFastRows : T;
        const int64_t rows_units = (int64_t)om.nbatch * ((om.rows + unit_rows - 1) / unit_rows);
        const int kchunk = balanced_chunk(rows_units, om.K, resident, r_fast ? kRowFastBatch : T);
        const int64_t work = rows_units * ((om.K + kchunk - 1) / kchunk);
        const int grid = (int)(work < resident ? (work < 1 ? 1 : work) : resident);
        LaunchScope ls_("k_split_rowmax", s);
        k_split_rowmax<<<grid, dim3(T, TR), 0, s>>>(om, X, rowmax, r_fast ? 1 : 0, kchunk);
    }
    EG_CHECK_LAUNCH("k_split_rowmax");
    {
        const int64_t n = (int64_t)om.nbatch * om.Rp;
        LaunchScope ls_("k_split_exponent", s);
        k_split_exponent<<<(int)std::min<int64_t>((n + 255) / 256, cap), 256, 0, s>>>(rowmax, rexp, n);
    }
    EG_CHECK_LAUNCH("k_split_exponent");
    {
        const int64_t work = (int64_t)om.nbatch * (om.Rp / T) * ((om.Kp / TK + kDigitStrip - 1) / kDigitStrip);
        static PerDevice<int> grids, grids_f64; // (the S variants share a register budget)
        const int cta = f64 ? grids_f64.get(current_device(), [] { return resident_grid(k_split_digits<kF64Slices, true>); })
                            : grids.get(current_device(), [] { return resident_grid(k_split_digits<5, false>); });
        const int grid = (int)(work < cta ? work : cta);
        LaunchScope ls_("k_split_digits", s);
        const int rf = r_fast ? 1 : 0;
        if (f64)
            k_split_digits<kF64Slices, true><<<grid, dim3(T, TR), 0, s>>>(om, X, rexp, planes, rf);
        else switch (S) {
        case 2: k_split_digits<2, false><<<grid, dim3(T, TR), 0, s>>>(om, X, rexp, planes, rf); break;
        case 3: k_split_digits<3, false><<<grid, dim3(T, TR), 0, s>>>(om, X, rexp, planes, rf); break;
        case 4: k_split_digits<4, false><<<grid, dim3(T, TR), 0, s>>>(om, X, rexp, planes, rf); break;
        case 5: k_split_digits<5, false><<<grid, dim3(T, TR), 0, s>>>(om, X, rexp, planes, rf); break;
        default: k_split_digits<6, false><<<grid, dim3(T, TR), 0, s>>>(om, X, rexp, planes, rf); break;
        }
    }
    EG_CHECK_LAUNCH("k_split_digits");
    return EG_SUCCESS;
}

template <int S, bool CHECK, int R>
cudaError_t launch_split_rows(const SplitJob &a, const SplitJob &b, int kc, int ld, int C, size_t smem, int *clear,
                              unsigned long long *magnitudes, cudaStream_t s) {
    static PerDevice<cudaError_t> attributes;
    const cudaError_t attr = attributes.get(current_device(), [] {
        return cudaFuncSetAttribute(k_split_rows<S, CHECK, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    });
    if (attr != cudaSuccess) return attr;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((a.tiles + b.tiles) * C));
    cfg.blockDim = dim3(kFusedThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute la;
    la.id = cudaLaunchAttributeClusterDimension;
    la.val.clusterDim.x = (unsigned)C;
    la.val.clusterDim.y = 1;
    la.val.clusterDim.z = 1;
    cfg.attrs = &la;
    cfg.numAttrs = C > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_split_rows<S, CHECK, R>, a, b, kc, ld, C, clear, magnitudes);
}

// Elements from row to row of the digit planes: K in whole blocks of 64, or for a short K
// of which those would be an eighth padding or more, in 32-byte sectors (the tensor maps
// fill the rest of the last block with zeros; only the fused launch writes such rows).
// 421875 x 75: 68 MB a plane instead of 108; with ten of them the splitting takes 222 us
// instead of 228, and 180 with the rows' elements spread over all lanes (k_split_rows).
int64_t plane_pitch(int64_t K) {
    const int64_t sectors = round_up(K, 16), blocks = round_up(K, kBK);
    return K <= 512 && 8 * sectors <= 7 * blocks ? sectors : blocks;
}

// Splits the operands of a contraction (an operand without rows is left out), and sets
// the kListWords words at clear to zero (unless null).  *magnitudes, zero before, receive
// TcGemmParams::magnitudes (FP64 form, unless null; null afterwards where they do not).  The
// fused launch when a range of K fits shared memory (K to about 25000); beyond, the
// passes over each operand, with tables of offsets at tab (rows and K of each operand;
// may be null).  Fused against passes, device time: both operands of 2304^3 in FP64
// 165 -> 68 us, the six splits of a ring contraction with adjoints at o = 24, v = 96
// 515 -> 211 us, the four of n = 75 quarter transformations 1.90 -> 0.72 ms (0.9 GB
// each: 5.2 TB/s).
eg_status split_both(OperandMap oa, const double *A, int *eA, __nv_bfloat16 *pA, OperandMap ob, const double *B, int *eB,
                     __nv_bfloat16 *pB, unsigned long long *maxima, int64_t *tab, int S, bool f64, int *clear,
                     unsigned long long **magnitudes, cudaStream_t s) {
    for (OperandMap *o : {&oa, &ob}) {
        o->sr = affine_stride(o->rg, o->comp);
        o->sk = affine_stride(o->kg, o->comp);
    }
    const int64_t Kp = oa.Kp;
    int R = 32, C = 1;
    int64_t kc = 0;
    size_t smem = 0;
    auto fits = [&](int r, int c, size_t limit) {
        const int64_t k = round_up((Kp + c - 1) / c, 4), ld = round_up(k, 16) + 2;
        const size_t bytes = (size_t)r * ld * 8 + (size_t)k * 8 + (size_t)r * 20;
        if (bytes > limit) return false;
        R = r;
        C = c;
        kc = k;
        smem = bytes;
        return true;
    };
    bool ok = false;
    // 32 rows, then 8, and up to eight CTAs along K, such that three CTAs fit an SM and,
    // where K allows, there are a few for every SM; the longest K takes an SM per CTA
    for (int r : {32, 8})
        for (int c = 1; c <= 8 && !ok; c *= 2)
            if (fits(r, c, 75 * 1024)) {
                const int64_t tiles = (oa.nbatch * oa.Rp + ob.nbatch * ob.Rp) / r;
                ok = tiles * c >= (r == 32 ? 2 : 4) * num_sms() || c == 8 || Kp / (2 * c) < 128;
            }
    if (!ok) ok = fits(8, 8, 227 * 1024);
    const int64_t tiles = (oa.rows ? oa.nbatch * oa.Rp / R : 0) + (ob.rows ? ob.nbatch * ob.Rp / R : 0);
    if (ok && tiles * C < (int64_t(1) << 31)) {
        auto job = [&](const OperandMap &o, const double *X, int *e, __nv_bfloat16 *pl) {
            const int64_t kstride = o.kg.n ? o.kg.s[o.comp][o.kg.n - 1] : 0, rstride = o.rg.n ? o.rg.s[o.comp][o.rg.n - 1] : 0;
            SplitJob j{o, X, e, pl, rstride > 0 && (kstride == 0 || rstride < kstride) ? 1 : 0,
                       0, o.rows ? o.nbatch * o.Rp / R : 0, 1};
            j.sample = (int)std::max<int64_t>(1, j.tiles / 32);
            bool even = !j.row_fast && kstride == 1 && o.kg.ext[o.kg.n - 1] % 2 == 0 && ((uintptr_t)X & 15) == 0;
            for (const ModeGroup *g : {&o.bg, &o.rg, &o.kg})
                for (int d = 0; d < g->n - (g == &o.kg ? 1 : 0); d++) even = even && g->s[o.comp][d] % 2 == 0;
            j.pairs = even ? 1 : 0;
            return j;
        };
        const SplitJob ja = job(oa, A, eA, pA), jb = job(ob, B, eB, pB);
        const int ld = (int)round_up(kc, 16) + 2;
        cudaError_t err;
        {
            LaunchScope ls_("k_split_rows", s);
            auto go = [&](auto slices, auto check) {
                constexpr int SL = decltype(slices)::value;
                constexpr bool CH = decltype(check)::value;
                return R == 32 ? launch_split_rows<SL, CH, 32>(ja, jb, (int)kc, ld, C, smem, clear, *magnitudes, s)
                               : launch_split_rows<SL, CH, 8>(ja, jb, (int)kc, ld, C, smem, clear, *magnitudes, s);
            };
            using std::integral_constant;
            if (f64)
                err = go(integral_constant<int, kF64Slices>{}, std::true_type{});
            else
                switch (S) {
                case 2: err = go(integral_constant<int, 2>{}, std::false_type{}); break;
                case 3: err = go(integral_constant<int, 3>{}, std::false_type{}); break;
                case 4: err = go(integral_constant<int, 4>{}, std::false_type{}); break;
                case 5: err = go(integral_constant<int, 5>{}, std::false_type{}); break;
                default: err = go(integral_constant<int, 6>{}, std::false_type{}); break;
                }
        }
        if (err != cudaSuccess) return cuda_fail(err, "k_split_rows");
        EG_CHECK_LAUNCH("k_split_rows");
        return EG_SUCCESS;
    }
    *magnitudes = nullptr; // (the passes do not add them up)
    if (clear) EG_CUDA(cudaMemsetAsync(clear, 0, kListWords * sizeof(int), s));
    unsigned long long *maxA = maxima, *maxB = maxima + (int64_t)oa.nbatch * oa.Rp;
    eg_status st;
    if (oa.rows && (st = split_operand(oa, A, maxA, eA, pA, S, s, tab, tab ? tab + oa.rows : nullptr, f64)) != EG_SUCCESS)
        return st;
    int64_t *tabB = tab ? tab + oa.rows + oa.K : nullptr;
    if (ob.rows && (st = split_operand(ob, B, maxB, eB, pB, S, s, tabB, tab ? tabB + ob.rows : nullptr, f64)) != EG_SUCCESS)
        return st;
    return EG_SUCCESS;
}

} // namespace

} // namespace eg::split

namespace eg {

int64_t mode_group_affine_stride(const ModeGroup &g, int comp) { return split::affine_stride(g, comp); }

// A tiled map over an FP64 tensor of rank 2..5: dims[0] is the contiguous mode,
// strides_bytes[i] the byte stride of mode i + 1, no swizzle, zero fill.
eg_status encode_tiled_f64(CUtensorMap *map, const void *base, int rank, const uint64_t *dims,
                           const uint64_t *strides_bytes, const uint32_t *box) {
    auto fn = split::encode_fn();
    if (!fn) return fail(EG_ERROR_CUDA, "cuTensorMapEncodeTiled is unavailable");
    cuuint64_t d[5], st[4];
    cuuint32_t b[5], es[5];
    for (int i = 0; i < rank; i++) {
        d[i] = dims[i];
        b[i] = box[i];
        es[i] = 1;
        if (i + 1 < rank) st[i] = strides_bytes[i];
    }
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, (cuuint32_t)rank, const_cast<void *>(base), d, st, b, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(EG_ERROR_NOT_SUPPORTED, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return EG_SUCCESS;
}

// A map over `planes` planes of `rows` x `K` BF16 digits laid out with row
// stride Kp and plane stride Rp * Kp elements (the extents may be below the
// padded layout: TMA then fills the rest of a box with zeros).
eg_status encode_planes_extent(CUtensorMap *map, void *base, int64_t K, int64_t rows, int64_t planes, int64_t Kp,
                               int64_t Rp) {
    auto fn = split::encode_fn();
    if (!fn) return fail(EG_ERROR_CUDA, "cuTensorMapEncodeTiled is unavailable");
    cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)(Kp * 2), (cuuint64_t)(Kp * 2 * Rp)};
    cuuint32_t box[3] = {(cuuint32_t)split::kBK, (cuuint32_t)split::kBM, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(EG_ERROR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
    return EG_SUCCESS;
}

// Whether |ab| is a power of two: it then joins the exponent instead of costing
// an FP64 multiplication per output.
static void set_ab(split::TcGemmParams &p, double ab) {
    int k = 0;
    const double f = std::frexp(std::fabs(ab), &k); // |ab| = f 2^k
    p.ab = ab;
    p.ab_pow2 = (f == 0.5) ? 1 : 0;
    p.ab_neg = (p.ab_pow2 && ab < 0) ? 1 : 0;
    if (p.ab_pow2) p.shift_const += k - 1;
}

// Single CTAs or CTA pairs, which tiles of a launch are cut along K, and how often:
// the whole rounds of the CTAs run whole tiles; the tiles left over for the last
// round -- 20 of 324 on 152 SMs, a third of the time -- are cut into as many slices
// of K blocks as give the smallest estimated time.  The estimate counts
// clocks: 360 per K block of a slice pair (320 on CTA pairs, which need two row
// tiles), 6000 for a tile's epilogue, and where tiles are cut 8000 for the launch that
// adds the slices up and 100 per plane of a slice's sums to write and read it.  At most
// max_slices tiles' sums are kept.  Returns the clocks.
static double choose_schedule(split::TcGemmParams &p, int64_t nb, int64_t mtiles, int64_t ntiles, int pairs, int planes,
                              int64_t max_slices) {
    using namespace split;
    double best = -1.0;
    const int clusters = mtiles >= 2 ? tc_pair_clusters() : 0;
    for (int cl = clusters > 0 && tc_pairs_forced() ? 2 : 1; cl <= (clusters > 0 ? 2 : 1); cl++) {
        const int64_t units = nb * ((mtiles + cl - 1) / cl) * ntiles, workers = cl == 2 ? clusters : num_sms();
        auto entry = [&](int64_t kb) { return (cl == 2 ? 320.0 : 360.0) * pairs * (double)kb + 6000.0; };
        const int64_t rounds = units / workers, rem = units - rounds * workers;
        const double whole = (double)rounds * entry(p.nkb);
        auto offer = [&](double t, int64_t t0, int64_t ks, int64_t slice, double margin) {
            if (best >= 0.0 && t >= margin * best) return;
            best = t;
            p.pair = cl - 1;
            p.t0 = (int)t0;
            p.ksplit = (int)ks;
            p.kslice = (int)slice;
        };
        offer(whole + (rem ? entry(p.nkb) : 0.0), units, 1, p.nkb, 1.0);
        if (rem == 0) continue;
        int64_t last = 0;
        for (int64_t ks = 2; ks <= std::min<int64_t>(p.nkb, 64); ks++) {
            const int64_t slice = (p.nkb + ks - 1) / ks;
            const int64_t n = (p.nkb + slice - 1) / slice; // slices actually used
            if (n == last) continue;
            last = n;
            if (rem * n * cl > max_slices) break;
            const int64_t r = (rem * n + workers - 1) / workers;
            offer(whole + (double)r * entry(slice) + 8000.0 + 100.0 * (double)(rem * n * cl * planes), rounds * workers, n,
                  slice, 0.98);
        }
    }
    return best;
}

// Scratch for the slices of tiles cut along K, in tiles of sums: as many as a schedule of
// `tiles` tiles of nkb K blocks may use, at most two per SM.
static int64_t slice_room(int64_t tiles, int64_t nkb) {
    return std::min<int64_t>(2 * tiles * std::min<int64_t>(nkb, 64), 2 * num_sms());
}

eg_status launch_split_contract(const Contraction &c, int slices, cudaStream_t s, eg_split_report *rep) {
    using namespace split;
    const int S = slices ? slices : 5;
    if (S < 2 || S > kMaxSlices) return fail(EG_ERROR_INVALID_ARGUMENT, "split form: slices must be in 2..6");
    const int64_t nb = c.batch.total, M = c.m.total, N = c.n.total, K = c.k.total;
    if (M >= (int64_t(1) << 31) || N >= (int64_t(1) << 31) || K >= (int64_t(1) << 31) || nb * S >= (int64_t(1) << 31))
        return fail(EG_ERROR_NOT_SUPPORTED, "split form: a mode group exceeds 2^31 elements");
    const int64_t Kp = plane_pitch(K), Mp = round_up(M, kBM), Np = round_up(N, kBN);
    const int64_t nkb_total = (K + kBK - 1) / kBK;

    // workspace: digit planes of A and B, row maxima, exponents, status word
    const size_t bytesA = (size_t)nb * S * Mp * Kp * 2, bytesB = (size_t)nb * S * Np * Kp * 2;
    const size_t offB = round_up((int64_t)bytesA, 1024);
    const size_t offMaxA = offB + round_up((int64_t)bytesB, 1024);
    const size_t offEA = offMaxA + round_up(nb * (Mp + Np) * 8, 256);
    const size_t offEB = offEA + round_up(nb * Mp * 4, 256);
    const size_t offR = offEB + round_up(nb * Np * 4, 256);
    // offset tables (rows and k of each operand) unless they would be large
    const bool tables = M + K <= (int64_t(1) << 25) && N + K <= (int64_t(1) << 25);
    const size_t offLost = offR + rbuf_bytes(), offTab = offLost + 256;
    const size_t tabBytes = tables ? (size_t)(M + N + 2 * K) * 8 : 0;
    const int64_t tiles = nb * (Mp / kBM) * (Np / kBN);
    const size_t offRacc = round_up((int64_t)(offTab + tabBytes), 256);
    int64_t slices_max = slice_room(tiles, nkb_total); // tiles cut along K
    const size_t raccBytes = (size_t)slices_max * kBM * kBN * 8;
    size_t total = offRacc + raccBytes;
    void *ws = nullptr;
    eg_status st = workspace(s, total, &ws);
    if (st == EG_ERROR_OUT_OF_MEMORY) { // without tiles cut along K
        set_error("");
        slices_max = 0;
        st = workspace(s, total = offRacc, &ws);
    }
    if (st != EG_SUCCESS) return st;
    char *base = (char *)ws;
    __nv_bfloat16 *planesA = (__nv_bfloat16 *)base, *planesB = (__nv_bfloat16 *)(base + offB);
    unsigned long long *maxA = (unsigned long long *)(base + offMaxA);
    int *eA = (int *)(base + offEA), *eB = (int *)(base + offEB);
    int *status = nullptr, *lost = (int *)(base + offLost); // kListWords, the second this call's record
    if ((st = status_word(s, &status)) != EG_SUCCESS) return st;

    unsigned long long *no_sums = nullptr;
    OperandMap oa{c.batch, c.m, c.k, 0, M, Mp, K, Kp, (int)nb};
    OperandMap ob{c.batch, c.n, c.k, 1, N, Np, K, Kp, (int)nb};
    int64_t *tab = tables ? (int64_t *)(base + offTab) : nullptr;
    if ((st = split_both(oa, c.A, eA, planesA, ob, c.B, eB, planesB, maxA, tab, S, false, lost, &no_sums, s)) != EG_SUCCESS) return st;
    if ((st = inject_lost(lost + 1, s)) != EG_SUCCESS) return st;

    CUtensorMap tmA, tmB, tmBh;
    if ((st = encode_planes(&tmA, planesA, Kp, Mp, nb * S)) != EG_SUCCESS) return st;
    if ((st = encode_planes(&tmB, planesB, Kp, Np, nb * S)) != EG_SUCCESS) return st;
    if ((st = encode_planes(&tmBh, planesB, Kp, Np, nb * S, kBN / 2)) != EG_SUCCESS) return st;

    TcGemmParams p{};
    p.S = S;
    p.planes = S;
    p.mtiles = (int)(Mp / kBM);
    p.ntiles = (int)(Np / kBN);
    p.nbatch = (int)nb;
    p.M = M;
    p.N = N;
    p.Mp = (int)Mp;
    p.Np = (int)Np;
    p.bg = c.batch;
    p.mg = c.m;
    p.ng = c.n;
    p.C = c.C;
    p.eA = eA;
    p.eB = eB;
    p.shift_const = -2 * kTopBits - kBits * (S - 1);
    set_ab(p, c.ab);
    p.status = status;
    p.lost = lost + 1;
    p.timeout_ns = 2000ull * 1000 * 1000;
    p.rbuf = (long long *)(base + offR);
    p.parts = (long long *)(base + offRacc);

    // Launches: when all slice groups' exact sum fits int64 over the whole K (up to
    // 65024 for S = 5), one.  Otherwise the slice groups are cut into ranges whose
    // own exact sums fit (S = 6 with K = 16384: groups 0-4 and 5), each range added
    // into C in FP64 by its own launch -- one extra rounding per range instead of a
    // launch (and a read and write of C) per 128 of K; a range that still cannot
    // take the whole K runs K passes.
    std::vector<std::pair<int, int>> ranges;
    for (int d0 = 0; d0 < S;) {
        int d1 = d0 + 1;
        while (d1 < S && max_k_per_pass_groups(d0, d1 + 1) >= Kp) d1++;
        ranges.push_back({d0, d1});
        d0 = d1;
    }
    const int shift_base = p.shift_const;
    bool first_launch = true;
    for (const auto &range : ranges) {
        p.d0 = range.first;
        p.d1 = range.second;
        p.shift_const = shift_base + kBits * (S - p.d1);
        const int64_t kb_per_pass = max_k_per_pass_groups(p.d0, p.d1) / kBK;
        if (kb_per_pass < 1) return fail(EG_ERROR_NOT_SUPPORTED, "split form: slice count too large for exact accumulation");
        for (int64_t kb0 = 0; kb0 < nkb_total || kb0 == 0; kb0 += kb_per_pass) {
            p.kb0 = (int)kb0;
            p.nkb = (int)std::min<int64_t>(kb_per_pass, nkb_total - kb0);
            int pairs = 0;
            for (int d = p.d0; d < p.d1; d++) pairs += d + 1;
            choose_schedule(p, nb, p.mtiles, p.ntiles, pairs, 1, slices_max);
            const bool first = first_launch;
            first_launch = false;
            p.cp = first ? c.cp : 1.0;
            p.zero = first ? (c.zero_when_cp_zero ? 1 : 0) : 0;
            if (p.nkb <= 0) break;
            static const bool prof_on = std::getenv("EINSUMS_GB300_TC_PROFILE") != nullptr;
            unsigned long long *prof = nullptr;
            if (prof_on) {
                EG_CUDA(cudaMalloc(&prof, (size_t)num_sms() * 8 * sizeof(unsigned long long)));
                EG_CUDA(cudaMemsetAsync(prof, 0, (size_t)num_sms() * 8 * sizeof(unsigned long long), s));
            }
            p.prof = prof;
            if ((st = launch_tc_gemm(tmA, tmB, tmBh, p, s)) != EG_SUCCESS) return st;
            if (prof) {
                // Per-role wait/busy cycles summed over CTAs (a tracing aid, off by default).
                std::vector<unsigned long long> h((size_t)num_sms() * 8);
                EG_CUDA(cudaMemcpyAsync(h.data(), prof, h.size() * 8, cudaMemcpyDeviceToHost, s));
                EG_CUDA(cudaStreamSynchronize(s));
                cudaFree(prof);
                double tot[8] = {0};
                int ran = 0; // CTAs of the launch (its grid may be below the SM count)
                for (size_t i = 0; i < h.size(); i++) tot[i % 8] += (double)h[i];
                for (size_t i = 6; i < h.size(); i += 8) ran += h[i] > 0 ? 1 : 0;
                std::fprintf(stderr,
                             "[tc profile] M=%lld N=%lld K=%lld tiles=%d: total %.3g cyc/CTA | producer wait empty %.1f%% | "
                             "mma wait full %.1f%% | mma wait acc %.1f%% | epi wait acc %.1f%% | epi flush %.1f%% | "
                             "epi final %.1f%%\n",
                             (long long)M, (long long)N, (long long)K, p.mtiles * p.ntiles * p.nbatch,
                             tot[6] / (ran > 0 ? ran : 1), 100 * tot[0] / tot[6], 100 * tot[1] / tot[6], 100 * tot[2] / tot[6],
                             100 * tot[3] / tot[6], 100 * tot[4] / tot[6], 100 * tot[5] / tot[6]);
            }
        }
    }
    if (rep) {
        rep->slices = S;
        rep->slice_pairs = S * (S + 1) / 2;
        rep->bits_per_slice = kBits;
        rep->error_bound = error_bound(S);
    }
    return EG_SUCCESS;
}

// The plain FP64 contraction on the tensor cores.
//
// This GPU's FP64 pipe retires two FMAs per clock per SM; the tensor cores run
// the 36 BF16 slice products of an eight-slice split (63 bits below the power of
// two above each row's largest element) an order of magnitude faster.  What the
// split leaves out is bounded for every output before it is written:
//
//   |C - C_exact| <= 9.04 2^-64 N max|A_i| max|B_j|     N: the k where both are nonzero
//
// (7.03 from the slice pairs dropped, 2 from the digits, with max| | the power of
// two above the row's largest element).  The check planes give, in two more slice
// products and exactly where it decides, M = sum_k p_a p_b with p <= 128 |x| / max, and N; where
//   M >= 20 N   (M >= 20 N + 256 for N < 8)
// the error is at most 4 2^-53 sum_k |A_ik| |B_jk| -- four roundings' worth, where
// the bound of a chain of K FMAs is K of them; with two products, half a rounding.
// A single product (N = 1), which an FMA rounds once and exactly, always fails; sums of
// no products are zero and pass.  Random sums that just pass, against FMA chains in exact
// arithmetic: rms error 0.82 of the chain's at N = 2, 0.65 at 4, 0.5 at 8, 0.25 at 32.
// A region of a tile in which the check fails anywhere (rows graded against each other,
// infinities, NaN) is not written but listed, and k_contract_f64 computes it from C as it
// was.  Inputs that fail everywhere so take the FP64 pipe's time and a little more; where the
// operands' magnitudes say so, nothing is tried (all_left_out in tc_gemm.cu).  The
// sums of all 36 products are exact in two int64 words and rounded once.  Neither they
// nor the check depend on how tiles are cut along K or shared by CTAs.
//
// The digit planes live in scratch of the device's pool (ScratchLease), bounded by
// kF64ScratchCap; larger operands are cut into panels of rows.  When the scratch or the
// stream's status word cannot be had (a memory budget, a full device) or the stream is
// being captured (a graph must not hold the scratch), EG_ERROR_NOT_SUPPORTED comes back
// with nothing launched and the FMA kernel runs instead.
constexpr size_t kF64ScratchCap = size_t(2) << 30;

eg_status launch_f64_tensor(Contraction c, cudaStream_t s, size_t front,
                            const std::function<eg_status(Contraction &, void *)> &fill) {
    using namespace split;
    constexpr int S = kF64Slices, P = S + 2;
    const int64_t nb = c.batch.total, M = c.m.total, N = c.n.total, K = c.k.total;
    const int64_t Kp = plane_pitch(K), nkb = (K + kBK - 1) / kBK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    EG_CUDA(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone) return EG_ERROR_NOT_SUPPORTED;
    RelaxedCapture relaxed; // another thread's capture neither stops nor suffers from the scratch
    // panels: all rows of both operands when they fit, else whole 128-row blocks of
    // each (and, with batches, as many batch indices as fit)
    const int64_t row_bytes = P * Kp * 2 + 32, Mp_all = round_up(M, kBM), Np_all = round_up(N, kBN);
    const int64_t budget = (int64_t)kF64ScratchCap / row_bytes / kBM * kBM;
    int64_t mb = Mp_all, nbk = Np_all, bb = 1;
    if (mb + nbk > budget) {
        const int64_t half = budget / 2 / kBM * kBM;
        if (half < kBM) return EG_ERROR_NOT_SUPPORTED;
        if (nbk <= half)
            mb = budget - nbk;
        else if (mb <= half)
            nbk = budget - mb;
        else
            mb = nbk = half;
    } else {
        bb = std::max<int64_t>(1, std::min<int64_t>(nb, budget / (mb + nbk)));
        bb = std::min<int64_t>(bb, (int64_t(1) << 20) / P);
    }
    const int64_t tiles = bb * (mb / kBM) * (nbk / kBN);
    const int64_t slices_max = slice_room(tiles, nkb); // tiles cut along K
    const int64_t all_tiles = nb * (Mp_all / kBM) * (Np_all / kBN);
    const bool tables = M + K <= (int64_t(1) << 22) && N + K <= (int64_t(1) << 22);
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 1023) & ~size_t(1023);
        return o;
    };
    const size_t oFront = take(front);
    const size_t oPA = take((size_t)bb * P * mb * Kp * 2), oPB = take((size_t)bb * P * nbk * Kp * 2);
    const size_t oMax = take((size_t)bb * (mb + nbk) * 8);
    const size_t oCheck = take((size_t)slices_max * kBM * kBN * sizeof(int));
    const size_t oParts = take((size_t)slices_max * 2 * kBM * kBN * 8);
    const size_t oExp = take((size_t)bb * (mb + nbk) * 4);
    const size_t oTab = take(tables ? (size_t)(M + N + 2 * K) * 8 : 0);
    const size_t oR = take(rbuf_bytes(3));
    const size_t oRedoN = take(kListWords * sizeof(int)), oRedo = take((size_t)all_tiles * kTileRegions * sizeof(int4));
    ScratchLease lease(s, at);
    if (!lease.ptr()) return EG_ERROR_NOT_SUPPORTED;
    int *status = nullptr;
    eg_status st = status_word(s, &status);
    if (st != EG_SUCCESS) {
        set_error("");
        return EG_ERROR_NOT_SUPPORTED;
    }
    char *base = (char *)lease.ptr();
    if (fill && (st = fill(c, base + oFront)) != EG_SUCCESS) return st;
    __nv_bfloat16 *planesA = (__nv_bfloat16 *)(base + oPA), *planesB = (__nv_bfloat16 *)(base + oPB);
    int *eA = (int *)(base + oExp), *eB = eA + bb * mb;
    int64_t *tab = tables ? (int64_t *)(base + oTab) : nullptr;

    TcGemmParams p{};
    p.S = S;
    p.planes = P;
    p.bg = c.batch;
    p.mg = c.m;
    p.ng = c.n;
    p.C = c.C;
    p.cp = c.cp;
    p.zero = c.zero_when_cp_zero ? 1 : 0;
    p.eA = eA;
    p.eB = eB;
    p.shift_const = -2 * kTopBits - kBits * (S - 1);
    set_ab(p, c.ab);
    p.status = status;
    p.timeout_ns = 2000ull * 1000 * 1000;
    p.rbuf = (long long *)(base + oR);
    p.parts = (long long *)(base + oParts);
    p.parts_check = (int *)(base + oCheck);
    p.d0 = 0;
    p.d1 = S;
    p.hid = kF64High;
    p.redo = (int4 *)(base + oRedo);
    p.redo_count = (int *)(base + oRedoN);
    p.lost = p.redo_count + 1;
    bool first = true; // the first splitting launch clears redo_count and the record
    // whether the data are worth a try is looked at where one panel holds all of them
    unsigned long long *const header = (unsigned long long *)lease.header();
    unsigned long long *magnitudes = bb >= nb && mb >= Mp_all && nbk >= Np_all ? header : nullptr;

    for (int64_t b0 = 0; b0 < nb; b0 += bb) {
        const int64_t nbc = std::min(bb, nb - b0);
        for (int64_t m0 = 0; m0 < M; m0 += mb) {
            const int64_t mc = std::min(mb, M - m0), Mp = round_up(mc, kBM);
            for (int64_t n0 = 0; n0 < N; n0 += nbk) {
                const int64_t nc = std::min(nbk, N - n0), Np = round_up(nc, kBN);
                p.nkb = (int)nkb;
                choose_schedule(p, nbc, Mp / kBM, Np / kBN, S * (S + 1) / 2 + 2, 2, slices_max);
                OperandMap oa{c.batch, c.m, c.k, 0, mc, Mp, K, Kp, (int)nbc};
                oa.b0 = b0;
                oa.row0 = m0;
                OperandMap ob{c.batch, c.n, c.k, 1, nc, Np, K, Kp, (int)nbc};
                ob.b0 = b0;
                ob.row0 = n0;
                // a panel's planes stay while the other operand's panels go by
                if (n0 > 0) oa.rows = 0;
                if (nbk >= Np_all && m0 > 0) ob.rows = 0;
                if ((st = split_both(oa, c.A, eA, planesA, ob, c.B, eB, planesB, (unsigned long long *)(base + oMax), tab,
                                     S, true, first ? p.redo_count : nullptr, &magnitudes, s)) != EG_SUCCESS)
                    return st;
                if (first && (st = inject_lost(p.lost, s)) != EG_SUCCESS) return st;
                first = false;
                CUtensorMap tmA, tmB, tmBh;
                if ((st = encode_planes(&tmA, planesA, Kp, Mp, nbc * P)) != EG_SUCCESS) return st;
                if ((st = encode_planes(&tmB, planesB, Kp, Np, nbc * P)) != EG_SUCCESS) return st;
                if ((st = encode_planes(&tmBh, planesB, Kp, Np, nbc * P, kBN / 2)) != EG_SUCCESS) return st;
                p.magnitudes = magnitudes;
                p.b0 = b0;
                p.m0 = m0;
                p.n0 = n0;
                p.M = mc;
                p.N = nc;
                p.Mp = (int)Mp;
                p.Np = (int)Np;
                p.mtiles = (int)(Mp / kBM);
                p.ntiles = (int)(Np / kBN);
                p.nbatch = (int)nbc;
                if ((st = launch_tc_gemm(tmA, tmB, tmBh, p, s)) != EG_SUCCESS) return st;
            }
        }
    }
    return launch_contract_f64_listed(c, p.redo, p.redo_count, status, magnitudes, s);
}

// Whether an FP64 contraction is worth its detour over the tensor cores, from
// estimates of both times: the FMA kernel's own, against 30 us of launches, the
// splitting of both operands (36 bytes moved per element) and the tensor kernel's
// schedule.  K below 32 is left to the FMA kernel, whose own error is then as small
// as the check's bound; above 65536 the sums would need more bits.
bool f64_tensor_pays(const Contraction &c) {
    using namespace split;
    const int64_t nb = c.batch.total, M = c.m.total, N = c.n.total, K = c.k.total;
    if (K < 32 || K > 65536 || M < 8 || N < 8) return false;
    if (M > int64_t(65535) * 64 || N > int64_t(65535) * 64 || nb > (int64_t(1) << 24)) return false;
    const double fma = contract_f64_seconds(c);
    if (fma < 40e-6) return false;
    TcGemmParams p{};
    p.nkb = (int)(round_up(K, kBK) / kBK);
    const int64_t mtiles = round_up(M, kBM) / kBM, ntiles = round_up(N, kBN) / kBN;
    if (nb * mtiles * ntiles > (int64_t(1) << 30)) return false;
    const double clocks = choose_schedule(p, nb, mtiles, ntiles, kF64Slices * (kF64Slices + 1) / 2 + 2, 2,
                                           slice_room(nb * mtiles * ntiles, p.nkb));
    const double tensor = 30e-6 + (double)nb * (double)(M + N) * (double)K * 36.0 / 3e12 + clocks / 1.9e9;
    return tensor < 0.9 * fma;
}

} // namespace eg
