// tcgen05 GEMM of the split-BF16 form (see split.cuh for the arithmetic).
//
// One persistent CTA per SM, or a pair of CTAs on two SMs (cta_group::2), 384
// threads in three roles:
//   warps 0, 2  TMA producers: stream 128 x 64 BF16 tiles of the A and of the B digit
//               planes (128-byte swizzle) into a ring of six slots, a slot holding
//               one K block of one A slice and one B slice;
//   warp 1      MMA issuer: allocates 512 TMEM columns and issues tcgen05.mma
//               kind::f16 (N = 256: two slice groups at once, step_of below) into
//               one of two FP32 accumulators of 256 columns, committing each slot
//               and each chunk of at most 1024 products per accumulated sum;
//   warps 4-11  epilogue (two warps per TMEM lane quadrant, 64 columns each in turns of 16): after
//               every chunk convert the exact FP32 sums to integers and add them to
//               int64 sums in registers (128 of them; setmaxnreg moves registers
//               from the other warps); a finished tile's sums wait in a scratch and
//               are scaled by 2^(eA+eB-...) and applied, C = cp*C + ab*v in FP64
//               through the output's index map, between the chunks of the next tile.
// Bound: the tensor pipe (64 clocks per 128 x 128 x 16 product and SM).  What kept
// it idle before was the issue loop, not operand delivery (see the issuer).
// Every mbarrier wait is bounded (split.cuh, ptx.cuh): on a timeout the CTA
// records an error code (report_lost), raises its abort flag, waits for its own
// TMA loads and MMAs to land, frees TMEM and returns.  The launches after it then
// add up no slices, and in the FP64 form write NaN to all of C.
#include <climits>
#include <cstdlib>

#include "ptx.cuh"
#include "split.cuh"

namespace eg::split {

namespace {

constexpr int kSlots = 6;                  // ring slots: one K block of one A slice and one B slice
constexpr int TILE_BYTES = kBM * kBK * 2;  // a 128 x 64 BF16 tile
constexpr int kEpiWarps = 8;               // two per TMEM lane quadrant
constexpr int THREADS = 128 + 32 * kEpiWarps; // warps 0 and 2 TMA, warp 1 MMA, warps 4..11 epilogue (3 idle)
constexpr uint32_t TMEM_COLS = 512;
constexpr int AUX_BYTES = 256;
constexpr int kFin = 8;      // columns finished at a time
constexpr int FIN_T = 33;    // padded row count of a warp's transposition buffer
constexpr int kCols = kBN / (kEpiWarps / 4); // columns of an epilogue warp
static_assert(kTileRegions == kEpiWarps, "a region per epilogue warp");
// per epilogue warp: its column offsets and (of two tiles) exponents, the
// transposition buffer of one batch, and its 32 rows' addresses
constexpr int EPI_WARP_BYTES = kCols * (8 + 2 * 4) + kFin * FIN_T * 8 + 33 * 8;
constexpr int SMEM_BYTES = 1024 + 2 * kSlots * TILE_BYTES + AUX_BYTES + kEpiWarps * EPI_WARP_BYTES + 64;
static_assert(SMEM_BYTES <= 232448, "shared memory per CTA");
// setmaxnreg: the epilogue warps' sums take 128 registers; what they hold beyond the
// launch's 168 a thread, the four other warps give up.  No role may spill: a local load
// that misses the few KB of L1 left beside the ring waits some 4000 clocks behind the
// tiles in flight (25600 x 25600, K = 1024: 16.0 ms with 60 bytes of spills a thread,
// 12.9 without).
constexpr int kRegsIssue = 56, kRegsEpilogue = 224;
static_assert(128 * kRegsIssue + 32 * kEpiWarps * kRegsEpilogue <= THREADS * 168, "registers of the launch");
constexpr int GROUP_M = 16; // tile rasterisation: groups of 16 row tiles share B tiles in L2
constexpr unsigned long long DRAIN_NS = 200ull * 1000 * 1000;
constexpr unsigned long long ODD_DRAIN_NS = 10ull * 1000 * 1000; // longer than any load takes

// Optional cycle counters per CTA (TcGemmParams::prof, 8 slots per CTA).
enum { kProfProducerWaitEmpty, kProfMmaWaitFull, kProfMmaWaitAcc, kProfEpiWaitAcc, kProfEpiFlush, kProfEpiFinal,
       kProfTotal, kProfSlots = 8 };

__device__ __forceinline__ void prof_add(const TcGemmParams &p, int slot, long long cycles) {
    if (p.prof) atomicAdd(p.prof + blockIdx.x * kProfSlots + slot, (unsigned long long)cycles);
}

// Output tile t of the schedule in units of CL row tiles (a CTA pair takes two
// vertically adjacent 128-row tiles); mt counts those units.
template <int CL>
__device__ __forceinline__ void tile_coords(const TcGemmParams &p, int t, int &b, int &mt, int &nt) {
    const int mtiles = (p.mtiles + CL - 1) / CL, gm = GROUP_M / CL;
    const int per_batch = mtiles * p.ntiles;
    b = t / per_batch;
    t -= b * per_batch;
    const int per_group = gm * p.ntiles;
    const int g = t / per_group;
    const int first_m = g * gm;
    const int gsize = min(mtiles - first_m, gm);
    const int r = t - g * per_group;
    mt = first_m + r % gsize;
    nt = r / gsize;
}

// Column of a tile that is an epilogue warp's column i: the two warps of a lane quadrant
// take turns of 16 columns, so that a narrow tile (N = 57: 32 and 25 columns, not 57 and
// none) keeps both busy.  421875 x 75, K = 75 in FP64: 673 us, with the columns in two
// runs of 64 793 us.
__device__ __forceinline__ int tile_col(int half, int i) { return (i >> 4) * 32 + half * 16 + (i & 15); }

// Everything one role needs about a tile, for both the single-contraction and
// the grouped form.
struct TileJob {
    int mt, nt;
    int zA, zB;  // digit plane of slice 0 for A / B
    int kbeg;    // first K block (of this pass) of the K slice
    int nkb;     // K blocks
    int part;    // a K slice of a tile: where its sums go (-1: a whole tile); -2: rows past
                 // the last tile (the odd half of a CTA pair's tile), nothing to store
    int64_t M, N;
    const ModeGroup *mg, *ng;
    const int *eA, *eB; // exponents of rows / columns of this (item, batch)
    double *C;          // output base of this (item, batch)
    int b;              // batch index
    int item;           // item of a grouped launch
    const CUtensorMap *mapA, *mapB; // per-item maps (grouped launches), else null
};

// Tile t of the schedule, as seen by CTA `rank` of its pair (0 when CL = 1).
template <bool GROUPED, int CL>
__device__ __forceinline__ TileJob resolve(const TcGemmParams &p, const TcItem *items, const int4 *work, int t,
                                           int rank) {
    TileJob j;
    if (!GROUPED) {
        int b, mu, ks = 0;
        const bool split = t >= p.t0;
        j.part = split ? (t - p.t0) * CL + rank : -1;
        if (split) {
            const int e = t - p.t0, q = e / p.ksplit;
            ks = e - q * p.ksplit;
            t = p.t0 + q;
        }
        tile_coords<CL>(p, t, b, mu, j.nt);
        j.mt = mu * CL + rank;
        j.zA = b * p.planes;
        j.zB = b * p.planes;
        j.kbeg = ks * p.kslice;
        j.nkb = split ? min(p.kslice, p.nkb - j.kbeg) : p.nkb;
        if (j.mt >= p.mtiles) j.part = -2;
        j.M = p.M;
        j.N = p.N;
        j.mg = &p.mg;
        j.ng = &p.ng;
        j.eA = p.eA + (int64_t)b * p.Mp;
        j.eB = p.eB + (int64_t)b * p.Np;
        int64_t oa, ob, oc;
        group_offsets(p.bg, p.b0 + b, oa, ob, oc);
        j.C = p.C + oc;
        j.b = (int)(p.b0 + b);
        j.mapA = j.mapB = nullptr;
    } else {
        const int4 w = work[t];
        const TcItem &it = items[w.x];
        const int b = w.y;
        j.mt = w.z;
        j.nt = w.w;
        j.mapA = p.item_maps + 2 * w.x;
        j.mapB = j.mapA + 1;
        j.zA = j.zB = b * p.planes; // planes are numbered within the item
        j.item = w.x;
        j.kbeg = 0;
        j.nkb = it.nkb;
        j.part = -1;
        j.M = it.M;
        j.N = it.N;
        j.mg = &it.mg;
        j.ng = &it.ng;
        j.eA = p.eA + it.eAoff + (int64_t)b * it.Mp;
        j.eB = p.eB + it.eBoff + (int64_t)b * it.Np;
        int64_t oa, ob, oc;
        group_offsets(it.bg, b, oa, ob, oc);
        j.C = it.C + oc;
        j.b = b;
    }
    return j;
}

// The slice groups (anti-diagonals s + t = d of the digit pairs) run two at a
// time, a step q covering groups d and d + 1 -- or group d alone: first, when their
// number is odd -- because both read the same slices: per K block the ring takes
// A_j and B_{hi-j} for j = 0 .. hi (hi the higher group), A_j meets B_{hi-j} in group
// hi and B_{hi-1-j}, the next slot's, in group hi - 1, in one MMA of N = 256.  The
// FP64 form starts with step -1, the two plane pairs of its accuracy check (planes S
// and S + 1), each a product of its own slot's tiles in an accumulator of its own.
struct Step {
    int hi;     // the higher group
    int slots;  // ring slots per K block
    bool two;   // groups hi - 1 and hi
    // K blocks of a chunk: at most 16 tile products per accumulator, 1024 digit products.
    // The check's sums (of whole numbers, none negative) run over all of K: N stays below
    // 2^24, and M is exact up to there, far above where it decides.
    int kbc;
};
__device__ __forceinline__ int step_count(const TcGemmParams &p) { return (p.d1 - p.d0 + 1) / 2; }
__device__ __forceinline__ Step step_of(const TcGemmParams &p, int q) {
    Step s;
    if (q < 0) {
        s.hi = p.S;
        s.slots = 2;
        s.two = false;
        s.kbc = INT_MAX;
    } else {
        const int odd = (p.d1 - p.d0) & 1;
        s.two = !(odd && q == 0);
        s.hi = p.d0 + 2 * q + 1 - odd;
        s.slots = s.hi + 1;
        s.kbc = kChunkKB / s.slots;
    }
    return s;
}
__device__ __forceinline__ int slot_a(const TcGemmParams &p, int q, int j) { return q < 0 ? p.S + j : j; }
__device__ __forceinline__ int slot_b(const TcGemmParams &p, int q, const Step &st, int j) {
    return q < 0 ? p.S + j : st.hi - j;
}

// K blocks of schedule entry t.
template <bool GROUPED>
__device__ __forceinline__ int entry_nkb(const TcGemmParams &p, const TcItem *items, const int4 *work, int t) {
    if (GROUPED) return items[work[t].x].nkb;
    if (t < p.t0) return p.nkb;
    const int kbeg = ((t - p.t0) % p.ksplit) * p.kslice;
    return min(p.kslice, p.nkb - kbeg);
}

// FP64 form: whether entry t's item of a list, or the whole of a single contraction, is left to
// the FMA kernel without being tried.  The splitting kernel adds up the check's magnitudes over
// each operand; where their means (over the elements that are not zero, in lists over all)
// multiply to less than 32, outputs with 20 N are few or none, and the FMA kernel would have to
// compute (nearly) all of it after the tensor cores did.  The kernel before wrote the sums, so
// all roles decide alike.  (It saves such a list the 160 us that the tensor kernel takes for 512
// uneven items, and costs an ordinary one 4.)
template <bool GROUPED, bool F64>
__device__ __forceinline__ bool left_out(const TcGemmParams &p, const TcItem *items, const int4 *work, int t) {
    if constexpr (GROUPED && F64) {
        const int i = work[t].x;
        const ulonglong2 s = __ldg((const ulonglong2 *)p.magnitudes + i);
        return (float)s.x * (float)s.y < items[i].tried;
    }
    return false;
}
template <bool F64>
__device__ __forceinline__ bool all_left_out(const TcGemmParams &p) {
    if (!F64 || !p.magnitudes) return false;
    const ulonglong2 a = __ldg((const ulonglong2 *)p.magnitudes), b = __ldg((const ulonglong2 *)p.magnitudes + 1);
    return (float)a.x * (float)b.x < kTriedMean * (float)a.y * (float)b.y;
}

// The FP64 value of one output's exact sums, scaled (but for an ab that is no power of
// two), before C is added.  FAST: every
// exponent of the tile lies where the result is a normal number (pend_fast).
template <bool F64, bool FAST>
__device__ __forceinline__ double finish_value(const TcGemmParams &p, long long lo, long long hi, int rowExp, int colExp) {
    if (!FAST && (rowExp == INT_MIN || colExp == INT_MIN)) return __longlong_as_double(0x7ff8000000000000ll);
    const int e = rowExp + colExp + p.shift_const;
    if constexpr (F64) return words_times_pow2_rn<FAST>(hi, lo, p.ab_neg, e);
    return int_times_pow2_rn<FAST>(p.ab_neg ? -lo : lo, e);
}

// Records `code` and stops this CTA's roles; in a CTA pair also the peer's
// (peer_flag: shared::cluster address of its abort flag, 0 without a peer).
__device__ __forceinline__ void raise_abort(const TcGemmParams &p, volatile int *abort_flag, int code,
                                            uint32_t peer_flag = 0) {
    report_lost(p.status_at, p.status, code);
    atomicCAS(p.lost, 0, code);
    *abort_flag = 1;
    if (peer_flag) ptx::st_cluster_u32(peer_flag, 1u);
}

// CL = 2 (launched as clusters of two CTAs): the pair computes 256 x 128 outputs
// with cta_group::2 MMAs (M = 256), each CTA holding its own 128 rows of A and of
// the accumulators.  Of the 256 columns of a two-group MMA the even CTA holds group
// hi's B tile and the odd CTA group hi - 1's; of a one-group MMA's 128 each holds
// half.  Both CTAs' loads complete on the even CTA's "full" barrier (which expects
// both CTAs' bytes); the even CTA's issuer alone issues and commits to both CTAs'
// "empty" and "accumulator full" barriers; both CTAs' epilogue warps release an
// accumulator on the even CTA's barrier (16 arrivals).
template <bool GROUPED, int CL, bool F64>
__global__ void __launch_bounds__(THREADS, 1)
    k_tc_split_gemm(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmBh, const __grid_constant__ TcGemmParams p,
                    const TcItem *items, const int4 *work) {
    static_assert(CL == 1 || (CL == 2 && !GROUPED), "CTA pairs serve single contractions");
    constexpr int PLANES = F64 ? 2 : 1; // int64 sums per output in the K slices' accumulator
    constexpr size_t kPlane = (size_t)kBM * kBN;
    const int qbeg = F64 ? -1 : 0, qend = step_count(p);
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *smA = smem, *smB = smem + kSlots * TILE_BYTES;
    uint64_t *full = (uint64_t *)(smem + 2 * kSlots * TILE_BYTES);
    uint64_t *empty = full + kSlots;
    uint64_t *accf = empty + kSlots;
    uint64_t *acce = accf + 2;
    uint64_t *done = acce + 2;
    uint32_t *tmem_slot = (uint32_t *)(done + 1);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
    volatile int *none_tried = abort_flag + 1; // single contractions: all_left_out
    // per-epilogue-warp copies of the tile's column offsets and exponents, so
    // the epilogue warps never wait on one another
    int64_t *colOffAll = (int64_t *)(smem + 2 * kSlots * TILE_BYTES + AUX_BYTES);
    int *colExpAll = (int *)(colOffAll + kEpiWarps * kCols);                // a warp: the running and the pending tile's
    double *finTAll = (double *)(colExpAll + 2 * kEpiWarps * kCols);            // a warp: kFin x FIN_T
    double **rowAtAll = (double **)(finTAll + kEpiWarps * kFin * FIN_T); // a warp: 32 rows (null: past the output)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = CL == 2 ? (int)ptx::cluster_ctarank() : 0;
    // shared::cluster addresses: the even CTA's barriers, and the peer's abort flag
    const uint32_t full_lead = CL == 2 ? ptx::mapa(ptx::smem_u32(full), 0) : 0;
    const uint32_t acce_lead = CL == 2 ? ptx::mapa(ptx::smem_u32(acce), 0) : 0;
    const uint32_t peer_flag = CL == 2 ? ptx::mapa(ptx::smem_u32((const void *)abort_flag), rank ^ 1) : 0;
    const long long t_start = p.prof ? clock64() : 0;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kSlots; i++) {
            ptx::mbar_init(&full[i], 1);
            ptx::mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            ptx::mbar_init(&accf[i], 1);
            ptx::mbar_init(&acce[i], kEpiWarps * CL);
        }
        ptx::mbar_init(done, 1);
        *abort_flag = 0;
        ptx::fence_mbar_init();
    }
    if (!GROUPED && F64 && warp == 3) {
        const bool out = all_left_out<F64>(p);
        if (lane == 0) *none_tried = out;
    }
    if (warp == 1) {
        ptx::tmem_alloc<CL>(tmem_slot, TMEM_COLS);
        ptx::tmem_relinquish<CL>();
    }
    ptx::tc_fence_before();
    __syncthreads();
    if (CL == 2) ptx::cluster_sync(); // the peer's barriers are initialised before any remote arrival
    ptx::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // first schedule entry and stride of this CTA (of its pair when CL = 2)
    const int cta0 = GROUPED ? p.ranges[blockIdx.x] : blockIdx.x / CL, ctas = GROUPED ? 1 : gridDim.x / CL;

    const int total_tiles =
        GROUPED ? p.ranges[blockIdx.x + 1] : p.t0 + (p.nbatch * ((p.mtiles + CL - 1) / CL) * p.ntiles - p.t0) * p.ksplit;

    if (warp < 4) {
        ptx::regs_dec<kRegsIssue>();
        if (warp == 0 || warp == 2) {
            // -------------------------------------------- TMA producers: A tiles, B tiles
            // Two warps, each with uniform control flow and one elected lane issuing:
            // one lane loading both tiles of a slot took longer over it than the MMAs.
            const bool isB = warp == 2;
            const bool leader = ptx::elect_one();
            if (leader) {
                ptx::tma_prefetch_desc(isB ? &tmB : &tmA);
                if (CL == 2 && isB) ptx::tma_prefetch_desc(&tmBh);
            }
            int stage = 0;
            uint32_t phase = 0;
            int issued = 0; // slots that have received tiles (they fill in order 0, 1, 2, ...)
            bool ok = true;
            const uint32_t ring0 = ptx::smem_u32(isB ? smB : smA);
            const uint32_t full0 = CL == 2 ? full_lead : ptx::smem_u32(full);
            const int end = !GROUPED && F64 && *none_tried ? 0 : total_tiles;
            for (int tile = cta0; tile < end && ok; tile += ctas) {
                const TileJob job = resolve<GROUPED, CL>(p, items, work, tile, rank);
                if (left_out<GROUPED, F64>(p, items, work, tile)) continue;
                const int row0 = (isB ? job.nt : job.mt) * kBM, z0 = isB ? job.zB : job.zA;
                const int kc0 = (p.kb0 + job.kbeg) * kBK, nkb = job.nkb;
                const void *map = isB ? &tmB : &tmA;
                if (GROUPED) {
                    map = isB ? job.mapB : job.mapA;
                    if (leader) {
                        if (tile + ctas < total_tiles) // the next tile's map, while this one runs
                            ptx::tma_prefetch_desc(p.item_maps + 2 * work[tile + ctas].x + (isB ? 1 : 0));
                        if (tile == cta0) ptx::tma_prefetch_desc(map);
                    }
                }
                for (int q = qbeg; q < qend && ok; q++) {
                    const Step st = step_of(p, q);
                    for (int kb = 0; kb < nkb && ok; kb++) {
                        const int kc = kc0 + kb * kBK;
                        for (int j = 0; j < st.slots; j++) {
                            const bool dual = st.two && j < st.hi;
                            const long long t0 = p.prof ? clock64() : 0;
                            const bool got = __all_sync(
                                0xffffffffu, ptx::mbar_wait(&empty[stage], phase ^ 1, p.timeout_ns, abort_flag));
                            if (p.prof && leader && !isB) prof_add(p, kProfProducerWaitEmpty, clock64() - t0);
                            if (!got) {
                                if (leader) raise_abort(p, abort_flag, 1, peer_flag);
                                ok = false;
                                break;
                            }
                            if (leader) {
                                const uint32_t dst = ring0 + (uint32_t)(stage * TILE_BYTES);
                                const uint32_t bar = full0 + (uint32_t)(stage * 8);
                                if (!isB) {
                                    // the slot's bytes (of both CTAs in a pair); the B tiles' may
                                    // arrive before they are expected
                                    if (rank == 0)
                                        ptx::mbar_arrive_expect_tx(&full[stage], CL == 1 ? 2u * TILE_BYTES
                                                                                 : dual  ? 4u * TILE_BYTES
                                                                                         : 3u * TILE_BYTES);
                                    ptx::tma_load_3d_at<CL>(dst, map, bar, kc, row0, z0 + slot_a(p, q, j));
                                } else {
                                    const int z = z0 + slot_b(p, q, st, j);
                                    if (CL == 1 || dual)
                                        ptx::tma_load_3d_at<CL>(dst, map, bar, kc, row0, CL == 1 ? z : z - rank);
                                    else
                                        ptx::tma_load_3d_at<CL>(dst, &tmBh, bar, kc, row0 + rank * (kBN / 2), z);
                                }
                            }
                            __syncwarp();
                            if (issued < kSlots) issued++;
                            if (++stage == kSlots) {
                                stage = 0;
                                phase ^= 1;
                            }
                        }
                    }
                }
            }
            // Slot i was last filled in the current round of the ring if i < stage,
            // else in the previous one.  In a pair the even CTA's barriers count both
            // CTAs' loads.
            if (rank == 0 && leader)
                for (int i = 0; i < issued; i++)
                    if (!ptx::mbar_wait(&full[i], i < stage ? phase : phase ^ 1, DRAIN_NS, nullptr))
                        raise_abort(p, abort_flag, 4, peer_flag);
            // An odd CTA that gives up may be slots ahead of the even one's count.
            if (CL == 2 && rank != 0 && !ok && leader)
                for (const uint64_t t0 = ptx::globaltimer_ns(); ptx::globaltimer_ns() - t0 < ODD_DRAIN_NS;) {}
            __syncwarp();
        } else if (warp == 1 && rank == 0) {
            // -------------------------------------------- MMA issuer (the even CTA of a pair)
            // The whole warp runs the loop and one elected lane issues: with uniform
            // control flow the operands stay in uniform registers, and a wait, the
            // issue of a slot's four MMAs and the commit fit inside the 512 clocks
            // that four MMAs of N = 256 take (a loop run by one lane took 520 clocks
            // for a slot whatever its MMAs, so N = 128 tiles ran at half rate).
            const bool leader = ptx::elect_one();
            const uint32_t idesc1 = ptx::idesc_bf16_f32(kBM * CL, kBN), idesc2 = ptx::idesc_bf16_f32(kBM * CL, 2 * kBN);
            const uint64_t desc0 = ptx::smem_desc_sw128(ptx::smem_u32(smA));
            constexpr uint64_t kTile = TILE_BYTES >> 4, kStep = 32 >> 4; // 16 BF16 along K
            uint32_t phase = 0, aphase = 0;
            int stage = 0, abuf = 0;
            bool ok = true;
            auto wait = [&](uint64_t *bar, uint32_t parity, int slot) {
                const long long t0 = p.prof ? clock64() : 0;
                const bool got = __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity, p.timeout_ns, abort_flag));
                if (p.prof && leader) prof_add(p, slot, clock64() - t0);
                if (!got) {
                    if (leader) raise_abort(p, abort_flag, 2, peer_flag);
                    ok = false;
                }
                return got;
            };
            auto commit = [&](uint64_t *bar) { // this CTA's barrier, and in a pair the peer's too
                if (CL == 1)
                    ptx::mma_commit(bar);
                else
                    ptx::mma_commit_both(bar);
            };
            const int end = !GROUPED && F64 && *none_tried ? 0 : total_tiles;
            for (int tile = cta0; tile < end && ok; tile += ctas) {
                const int nkb = entry_nkb<GROUPED>(p, items, work, tile);
                if (left_out<GROUPED, F64>(p, items, work, tile)) continue;
                for (int q = qbeg; q < qend && ok; q++) {
                    const Step st = step_of(p, q);
                    int c = 0; // K blocks in the open chunk
                    for (int kb = 0; kb < nkb && ok; kb++) {
                        if (c == 0 && !wait(&acce[abuf], aphase ^ 1, kProfMmaWaitAcc)) break;
                        const uint32_t D = tmem + (uint32_t)(abuf * 2 * kBN); // group hi, then group hi - 1
                        if (CL == 1 && !wait(&full[stage], phase, kProfMmaWaitFull)) break;
                        for (int j = 0; j < st.slots; j++) {
                            const bool dual = st.two && j < st.hi;
                            const int next = stage + 1 == kSlots ? 0 : stage + 1;
                            const uint32_t nphase = next == 0 ? phase ^ 1 : phase;
                            // one CTA: a two-group MMA also reads the next slot's B tile
                            if (CL == 2) {
                                if (!wait(&full[stage], phase, kProfMmaWaitFull)) break;
                            } else if (j + 1 < st.slots) {
                                if (!wait(&full[next], nphase, kProfMmaWaitFull)) break;
                            }
                            ptx::tc_fence_after();
                            if (leader) {
                                const uint64_t a = desc0 + (uint64_t)stage * kTile;
                                const uint64_t b = desc0 + (uint64_t)(kSlots + stage) * kTile;
                                const uint32_t keep = (c > 0 || (j > 0 && q >= 0)) ? 1u : 0u;
                                const uint32_t Dj = q < 0 && j == 0 ? D + kBN : D; // the check's sums lie apart
                                if (!dual || CL == 2 || next != 0) {
                                    const uint32_t idesc = dual ? idesc2 : idesc1;
#pragma unroll
                                    for (int k = 0; k < 4; k++)
                                        ptx::mma_bf16<CL>(Dj, a + k * kStep, b + k * kStep, idesc, k ? 1u : keep);
                                } else { // the ring wraps between the two B tiles
                                    const uint64_t b2 = desc0 + (uint64_t)kSlots * kTile;
#pragma unroll
                                    for (int k = 0; k < 4; k++) {
                                        ptx::mma_bf16<CL>(D, a + k * kStep, b + k * kStep, idesc1, k ? 1u : keep);
                                        ptx::mma_bf16<CL>(D + kBN, a + k * kStep, b2 + k * kStep, idesc1, k ? 1u : keep);
                                    }
                                }
                                commit(&empty[stage]);
                            }
                            __syncwarp();
                            stage = next;
                            phase = nphase;
                        }
                        if (!ok) break;
                        if (++c == st.kbc || kb + 1 == nkb) {
                            if (leader) commit(&accf[abuf]);
                            __syncwarp();
                            abuf ^= 1;
                            if (abuf == 0) aphase ^= 1;
                            c = 0;
                        }
                    }
                }
            }
            // All issued MMAs must complete before TMEM is released.
            if (leader) {
                if (CL == 1)
                    ptx::mma_commit(done);
                else
                    ptx::mma_commit_pair(ptx::smem_u32(done));
            }
            __syncwarp();
            if (!ptx::mbar_wait(done, 0, DRAIN_NS, nullptr)) raise_abort(p, abort_flag, 5, peer_flag);
        }
    } else {
        // ------------------------------------------------ epilogue (warps 4..11)
        // Two warps per TMEM lane quadrant; each owns 64 of the tile's 128 columns.
        ptx::regs_inc<kRegsEpilogue>();
        constexpr int FIN = F64 ? kFin / 2 : kFin; // the FP64 form holds two words per sum
        const int ew = warp - 4;              // 0..7
        const int quad = warp & 3;            // TMEM lane quadrant this warp may access
        const int half = ew >> 2; // of the columns, in turns of 16: columns 32 g + 16 half .. + 15
        const int row = quad * 32 + lane;     // tile row owned by this thread
        const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * 16);
        int64_t *colOff = colOffAll + ew * kCols;
        int *colExp = colExpAll + 2 * ew * kCols; // the pending tile's; the running tile's are at colExp + run_exp
        int run_exp = kCols;
        double *finT = finTAll + ew * (kFin * FIN_T);
        double **rowAt = rowAtAll + ew * 33;
        volatile int *const failed = (volatile int *)(rowAt + 32); // FP64 form: the check, in the running tile
        int abuf = 0;
        uint32_t aphase = 0;
        bool ok = true;
        const bool plain_store = p.zero && p.cp == 0.0; // once here: FP64 compares run on the slow FP64 pipe
        const bool timed = p.prof && ew == 0 && lane == 0;
        // The previous ("pending") tile: its sums wait in this CTA's scratch
        // (column-major, so a warp's stores and loads of them are contiguous, and a
        // thread reads back its own) and are scaled and added into C a batch of FIN
        // columns at a time between the chunks of this tile, so that neither the
        // latency of C nor the conversion holds the accumulators the issuer waits for.
        // A batch's loads are issued a chunk ahead: behind the tiles in flight for the
        // ring a load takes some 4000 clocks.  (The FP64 form loads the next batch's sums as
        // soon as this one's are converted: 4 x 421875 x 75 3749 -> 3635 us, 2304^3 569 ->
        // 558; the other form, with 8 columns a batch, was slower that way.)  The old values of C go to shared memory
        // (asynchronous copies): in registers, their loads share scoreboards with the
        // reads of the accumulators, which then waited for them too (25600 x 25600,
        // K = 1024: 16.1 ms against 13).  When C runs along
        // the rows a thread keeps its row; otherwise a batch is transposed through
        // shared memory so that the read-modify-write of C runs along a row (lanes
        // FIN*r .. FIN*r + FIN-1 take the batch's columns of row r).  colOff, colExp and rowAt
        // describe the pending tile.  One copy of this code, in a
        // loop: finishing a tile's columns straight from the registers is as many times
        // the code, which ran at the rate of instruction fetch (80k clocks a tile).
        long long *const rbc = p.rbuf + (size_t)blockIdx.x * (F64 ? 3 : 1) * kPlane + (size_t)(half * kCols) * kBM + row;
        // a K slice's sums: [128 columns][128 rows], two planes in the FP64 form
        auto part_of = [&](int tile) {
            return p.parts + (size_t)((tile - p.t0) * CL + rank) * PLANES * kPlane + (size_t)(half * kCols) * kBM + row;
        };
        int parity = 0; // FP64 form: which of two scratch planes takes this tile's high sums
        int pend_cols = 0, pend_done = 0; // columns of the pending tile, and how many are done
        bool pend_rows_fast = false, pend_fast = false;
        int pend_rowExp = 0;
        const long long *pend_lo = rbc; // its sums, and how far on its high sums are
        int pend_hi = 0;
        long long Rv[FIN], Hv[F64 ? FIN : 1];
        auto load_sums = [&](int c0) {
#pragma unroll
            for (int i = 0; i < FIN; i++) {
                Rv[i] = __ldcg(pend_lo + (c0 + i) * kBM);
                if constexpr (F64) Hv[i] = __ldcg(pend_lo + pend_hi + (c0 + i) * kBM);
            }
        };
        auto load_batch = [&]() {
            const int c0 = pend_done;
            if (!plain_store) {
#pragma unroll
                for (int i = 0; i < FIN; i++) {
                    const int e = i * 32 + lane;
                    const int r = pend_rows_fast ? lane : e / FIN, c = pend_rows_fast ? i : e % FIN;
                    if (rowAt[r] && c0 + c < pend_cols)
                        ptx::cp_async8(&finT[c * FIN_T + r], rowAt[r] + colOff[c0 + c]);
                }
            }
            if (!F64) load_sums(c0);
        };
        auto list_region = [&](const TileJob &job) { // this warp's, for the FMA kernel
            const int m0 = job.mt * kBM + quad * 32, n0 = job.nt * kBN + half * 16;
            p.redo[atomicAdd(p.redo_count, 1)] = GROUPED ? make_int4(job.item, job.b, m0, n0)
                                                         : make_int4(job.b, (int)p.m0 + m0, (int)p.n0 + n0, 0);
        };
        int first = cta0;
        if (!GROUPED && F64 && *none_tried) { // (k_tc_finish_slices lists what is cut along K)
            for (; first < p.t0 && first < total_tiles; first += ctas) {
                const TileJob job = resolve<GROUPED, CL>(p, items, work, first, rank);
                if (lane == 0 && (int64_t)job.mt * kBM + quad * 32 < job.M && (int64_t)job.nt * kBN + half * 16 < job.N)
                    list_region(job);
            }
            first = total_tiles;
        }
        for (int tile = first;; tile += ctas) {
            // after the last tile one more pass, without chunks, finishes what is pending
            const bool drain = tile >= total_tiles;
            if (drain && pend_done >= pend_cols) break;
            // only the K block count and the exponents (loaded early, like the batches) are
            // held through the chunks
            int nkb = 0, my_rowExp = 0;
            int live = 0; // this warp's columns inside the output (none when its rows are not): the others are skipped
            if (!drain) {
                const TileJob job = resolve<GROUPED, CL>(p, items, work, tile, rank);
                nkb = job.nkb;
                const int cols = (int)min((int64_t)kBN, job.N - (int64_t)job.nt * kBN);
                if ((int64_t)job.mt * kBM + quad * 32 < job.M)
                    live = cols / 32 * 16 + min(max(cols % 32 - half * 16, 0), 16);
                const int64_t m = (int64_t)job.mt * kBM + row;
                my_rowExp = m < job.M ? job.eA[m] : 0;
#pragma unroll
                for (int i = 0; i < kCols / 32; i++) {
                    const int64_t n = (int64_t)job.nt * kBN + tile_col(half, lane + 32 * i);
                    colExp[run_exp + lane + 32 * i] = n < job.N ? job.eB[n] : 0;
                }
            }
            // This thread's 64 exact sums, a Horner sum over the steps:
            // H = sum_d 2^(8 (last - d)) G_d.
            long long H[kCols];
#pragma unroll
            for (int i = 0; i < kCols; i++) H[i] = 0;
            const bool untried = !drain && left_out<GROUPED, F64>(p, items, work, tile);
            int q = drain || untried ? qend : qbeg, kb = 0;
            Step st = step_of(p, q);
            while (true) {
                const bool last = q == qend;
                if (pend_done < pend_cols) load_batch();
                if (!last) {
                    const long long tw = timed ? clock64() : 0;
                    const bool w = __all_sync(0xffffffffu, ptx::mbar_wait(&accf[abuf], aphase, p.timeout_ns, abort_flag));
                    const long long tw1 = timed ? clock64() : 0;
                    if (timed) prof_add(p, kProfEpiWaitAcc, tw1 - tw);
                    if (!w) {
                        if (lane == 0) raise_abort(p, abort_flag, 3, peer_flag);
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint32_t at = tl + (uint32_t)(abuf * 2 * kBN);
                    if (F64 && q < 0) { // the check; where it fails anywhere, the FMA kernel takes this warp's outputs
                        // quickly: a sum of few products anywhere, or a lack of magnitude?
                        float few = kCheckFew, least = 0.0f;
                        const bool slice = !GROUPED && tile >= p.t0; // (keeps each output's check)
#pragma unroll 1
                        for (int cc = 0; cc < live && !slice; cc += 16) {
                            uint32_t products[16], sums[16];
                            ptx::tmem_ld16(at + 2 * cc, products);
                            ptx::tmem_ld16(at + kBN + 2 * cc, sums);
                            ptx::tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; i++) { // (past the output there are no products)
                                const float n = __uint_as_float(products[i]);
                                few = fminf(few, n > 0.0f ? n : (float)kCheckFew);
                                least = fminf(least, fmaf(-(float)kCheckPer, n, __uint_as_float(sums[i])));
                            }
                        }
                        bool bad = few < kCheckFew || least < 0.0f;
                        if (slice || __any_sync(0xffffffffu, bad)) { // closely
                            bad = false;
#pragma unroll 1
                            for (int cc = 0; cc < live; cc += 16) {
                                uint32_t products[16], sums[16];
                                ptx::tmem_ld16(at + 2 * cc, products);
                                ptx::tmem_ld16(at + kBN + 2 * cc, sums);
                                ptx::tmem_wait_ld();
                                const uint32_t check = (uint32_t)(((tile - p.t0) * CL + rank) * kBN + half * kCols + cc) * kBM + row;
#pragma unroll
                                for (int i = 0; i < 16; i++) {
                                    const int n = __float2int_rn(__uint_as_float(products[i]));
                                    const int excess = __float2int_rn(__uint_as_float(sums[i])) - kCheckPer * n;
                                    bad = bad || check_fails(n, excess);
                                    if (slice) p.parts_check[check + i * kBM] = pack_check(n, excess);
                                }
                            }
                        }
                        *failed = __any_sync(0xffffffffu, bad) ? 1 : 0;
                    } else if (st.two) {
#pragma unroll
                        for (int cc = 0; cc < kCols; cc += 16) {
                            if (cc >= live) break;
                            uint32_t lo[16], hi[16];
                            ptx::tmem_ld16(at + 2 * cc, lo);
                            ptx::tmem_ld16(at + kBN + 2 * cc, hi);
                            ptx::tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; i++)
                                H[cc + i] += (long long)__float2int_rn(__uint_as_float(hi[i])) * (1 << kBits) +
                                             __float2int_rn(__uint_as_float(lo[i]));
                        }
                    } else {
#pragma unroll
                        for (int cc = 0; cc < kCols; cc += 16) {
                            if (cc >= live) break;
                            uint32_t lo[16];
                            ptx::tmem_ld16(at + 2 * cc, lo);
                            ptx::tmem_wait_ld();
#pragma unroll
                            for (int i = 0; i < 16; i++) H[cc + i] += __float2int_rn(__uint_as_float(lo[i]));
                        }
                    }
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (CL == 1)
                            ptx::mbar_arrive(&acce[abuf]);
                        else
                            ptx::mbar_arrive_cluster_relaxed(acce_lead + (uint32_t)(abuf * 8));
                    }
                    abuf ^= 1;
                    if (abuf == 0) aphase ^= 1;
                    kb += st.kbc;
                    if (kb >= nkb) { // the step is complete
                        kb = 0;
                        q++;
                        if (F64 && st.hi + 1 == p.hid) { // the high sums are complete
                            long long *const at_hi = !GROUPED && tile >= p.t0 ? part_of(tile) + kPlane : rbc + (1 + parity) * kPlane;
#pragma unroll
                            for (int i = 0; i < kCols; i++) {
                                at_hi[i * kBM] = H[i];
                                H[i] = 0;
                            }
                        } else if (q < qend) { // the step after has two groups
#pragma unroll
                            for (int i = 0; i < kCols; i++) H[i] *= 1 << (2 * kBits);
                        }
                        if (q < qend) st = step_of(p, q);
                    }
                    if (timed) prof_add(p, kProfEpiFlush, clock64() - tw1);
                }
                const long long tfin = timed ? clock64() : 0;
                // one batch after every chunk, the rest after the last
#pragma unroll 1
                while (pend_done < pend_cols) {
                    const int c0 = pend_done;
                    double val[FIN];
                    if (pend_fast) {
#pragma unroll
                        for (int i = 0; i < FIN; i++)
                            val[i] = finish_value<F64, true>(p, Rv[i], F64 ? Hv[F64 ? i : 0] : 0, pend_rowExp, colExp[c0 + i]);
                    } else {
#pragma unroll 1
                        for (int i = 0; i < FIN; i++) {
                            long long R = Rv[0], Hh = F64 ? Hv[0] : 0;
#pragma unroll
                            for (int k = 1; k < FIN; k++) {
                                if (k == i) R = Rv[k];
                                if (F64 && k == i) Hh = Hv[F64 ? k : 0];
                            }
                            const double v = finish_value<F64, false>(p, R, Hh, pend_rowExp, colExp[c0 + i]);
#pragma unroll
                            for (int k = 0; k < FIN; k++)
                                if (k == i) val[k] = v;
                        }
                    }
                    if (!p.ab_pow2) {
                        // opaque, so that it is not issued, unused, for every output; and apart
                        // from the conversions, whose chains interleave only without branches
#pragma unroll
                        for (int i = 0; i < FIN; i++) asm volatile("mul.rn.f64 %0, %0, %1;" : "+d"(val[i]) : "d"(p.ab));
                    }
                    if (F64 && c0 + FIN < pend_cols) load_sums(c0 + FIN); // a batch ahead
                    if (!plain_store) {
                        ptx::cp_async_wait_all();
                        __syncwarp();
                    }
                    if (pend_rows_fast) {
#pragma unroll
                        for (int i = 0; i < FIN; i++)
                            if (rowAt[lane] && c0 + i < pend_cols)
                                rowAt[lane][colOff[c0 + i]] = plain_store ? val[i] : fma(p.cp, finT[i * FIN_T + lane], val[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < FIN; i++) {
                            double &at = finT[i * FIN_T + lane];
                            at = plain_store ? val[i] : fma(p.cp, at, val[i]);
                        }
                        __syncwarp();
#pragma unroll
                        for (int i = 0; i < FIN; i++) {
                            const int e = i * 32 + lane, r = e / FIN, c = e % FIN;
                            if (rowAt[r] && c0 + c < pend_cols) rowAt[r][colOff[c0 + c]] = finT[c * FIN_T + r];
                        }
                        __syncwarp();
                    }
                    pend_done += FIN;
                    if (!last || pend_done >= pend_cols) break;
                    load_batch();
                }
                if (timed) prof_add(p, kProfEpiFinal, clock64() - tfin);
                if (last) break;
            }
            if (!ok || drain) break;
            // ---- end of tile: park its sums and make it the pending one
            pend_done = pend_cols = 0;
            const TileJob job = resolve<GROUPED, CL>(p, items, work, tile, rank);
            if (!GROUPED && job.part == -2) continue; // the odd half of a pair's last row of tiles
            if (untried) {
                if (live > 0 && lane == 0) list_region(job);
                continue;
            }
            const bool slice = !GROUPED && job.part >= 0; // k_tc_finish_slices adds it up
            long long *const sums = slice ? part_of(tile) : rbc;
#pragma unroll
            for (int i = 0; i < kCols; i++) sums[i * kBM] = H[i];
            if (slice) continue;
            long long *const own_hi = rbc + (F64 ? 1 + parity : 0) * kPlane;
            parity ^= 1;
            if (F64 && *failed) {
                if (lane == 0) list_region(job);
                continue;
            }
            if (live == 0) continue;
            __syncwarp(); // every lane has stored the tile before with the offsets replaced below
            pend_cols = live;
            pend_lo = sums;
            pend_hi = (int)(own_hi - sums);
            pend_rows_fast = job.mg->n > 0 && job.mg->s[2][job.mg->n - 1] == 1;
            const int64_t m = (int64_t)job.mt * kBM + row;
            const bool row_ok = m < job.M;
            int64_t rowOff = 0;
            pend_rowExp = row_ok ? my_rowExp : 0;
            if (row_ok) {
                int64_t oa, ob;
                group_offsets32(*job.mg, (uint32_t)(GROUPED ? m : p.m0 + m), oa, ob, rowOff);
            }
            // the largest and smallest exponents (a non-finite row or column counts as far below)
            int emax = INT_MIN, emin = INT_MAX;
#pragma unroll
            for (int k = 0; k < kCols / 32; k++) {
                const int i = lane + 32 * k, ex = colExp[run_exp + i];
                const int64_t n = (int64_t)job.nt * kBN + tile_col(half, i);
                int64_t oa, ob, oc = 0;
                if (i < live) group_offsets32(*job.ng, (uint32_t)(GROUPED ? n : p.n0 + n), oa, ob, oc);
                colOff[i] = oc;
                emax = max(emax, ex);
                emin = min(emin, max(ex, -(1 << 20)));
            }
            colExp += run_exp;
            run_exp = -run_exp;
            emax = __reduce_max_sync(0xffffffffu, emax) + __reduce_max_sync(0xffffffffu, pend_rowExp);
            emin = __reduce_min_sync(0xffffffffu, emin) + __reduce_min_sync(0xffffffffu, max(pend_rowExp, -(1 << 20)));
            pend_fast = emin + p.shift_const >= kFastMin && emax + p.shift_const <= kFastMax;
            rowAt[lane] = row_ok ? job.C + rowOff : nullptr;
            __syncwarp();
            if (F64) load_sums(0);
        }
    }

    __syncthreads();
    // A CTA of a pair leaves only when the peer is done too: the even CTA's MMAs
    // read the odd CTA's shared memory, and both CTAs arrive on each other's barriers.
    if (CL == 2) ptx::cluster_sync();
    if (p.prof && threadIdx.x == 0) prof_add(p, kProfTotal, clock64() - t_start);
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc<CL>(tmem, TMEM_COLS);
    }
}

// The tiles cut along K: a CTA adds up the slices of half the columns of a region of a
// tile (a region is one epilogue warp's), checks and scales the sums and applies them to C.  Bound: memory (8 or
// 16 bytes of sums per output and slice, mostly from L2).  Slices that add themselves to
// one accumulator with atomics, the last to arrive finishing it, took 36 us for the
// atomics (they retire some 70 a clock) and 29 us for the finishing of 144 x 2304, K =
// 2304 in FP64, while the other CTAs were done; stores and this kernel take about 15 us
// (the whole contraction 190 -> 132 us, 2304 x 2304 715 -> 672 us).
constexpr int kFinishRows = 8, kFinishCols = 32, kFinishParts = kCols / kFinishCols; // warps and columns of its CTAs
template <int CL, bool F64>
__global__ void __launch_bounds__(32 * kFinishRows, 3) k_tc_finish_slices(const __grid_constant__ TcGemmParams p) {
    __shared__ double tile[kFinishCols][33];
    constexpr int PLANES = F64 ? 2 : 1, PER = kFinishCols / kFinishRows;
    constexpr size_t kPlane = (size_t)kBM * kBN;
    const int c0 = blockIdx.x % kFinishParts * kFinishCols; // of the region's columns
    const int ew = blockIdx.x / kFinishParts % kTileRegions, u = blockIdx.x / (kFinishParts * kTileRegions);
    const int rank = u % CL, q = u / CL;
    int b, mu, nt;
    tile_coords<CL>(p, p.t0 + q, b, mu, nt);
    const int mt = mu * CL + rank;
    if (mt >= p.mtiles) return;
    const int quad = ew & 3, half = ew >> 2, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t m0 = (int64_t)mt * kBM + quad * 32, n0 = (int64_t)nt * kBN;
    const int rows = (int)min((int64_t)32, p.M - m0), cols = (int)min((int64_t)kBN, p.N - n0);
    const int live = min(cols / 32 * 16 + min(max(cols % 32 - half * 16, 0), 16) - c0, kFinishCols);
    if (rows <= 0 || live <= 0) return;
    auto list_region = [&] {
        p.redo[atomicAdd(p.redo_count, 1)] = make_int4((int)p.b0 + b, (int)(p.m0 + m0), (int)(p.n0 + n0) + half * 16, 0);
    };
    const int e0 = q * p.ksplit * CL + rank; // the tile's first slice; the next ones are CL further on
    const int lost = __ldcg(p.lost); // with a slice missing there is nothing to add up
    bool bad = all_left_out<F64>(p);
    if (F64 && !bad) {
        // the region's check, over the slices, as in a whole tile (both of its CTAs see all of it)
        const int all = cols / 32 * 16 + min(max(cols % 32 - half * 16, 0), 16);
        const int *at = p.parts_check + (size_t)e0 * kPlane + (size_t)(half * kCols) * kBM + quad * 32 + lane;
        constexpr int COLS = kCols / kFinishRows; // of a warp: all of them and four slices at a time
        int products[COLS] = {}, excess[COLS] = {};
#pragma unroll 4
        for (int k = 0; k < p.ksplit; k++, at += CL * kPlane) {
#pragma unroll
            for (int i = 0; i < COLS; i++) {
                const int c = warp + i * kFinishRows, x = c < all ? __ldcg(at + c * kBM) : 0;
                products[i] += x & 15;
                excess[i] += x >> 4;
            }
        }
#pragma unroll
        for (int i = 0; i < COLS; i++) bad = bad || check_fails(products[i], excess[i]);
        bad = bad && lane < rows;
    }
    // where this thread will write, along C's rows or columns, and C's old values there
    const bool plain_store = p.zero && p.cp == 0.0;
    const bool rows_fast = p.mg.n > 0 && p.mg.s[2][p.mg.n - 1] == 1;
    int64_t oa, ob, oc;
    group_offsets(p.bg, p.b0 + b, oa, ob, oc);
    double *out[PER], old[PER];
    const double *from[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int x = (threadIdx.x >> 5) + i * kFinishRows;
        const int r = rows_fast ? lane : x, c = rows_fast ? x : lane;
        from[i] = &tile[c][r];
        out[i] = nullptr;
        old[i] = 0.0;
        if (r < rows && c < live) {
            int64_t om, on;
            group_offsets32(p.mg, (uint32_t)(p.m0 + m0 + r), oa, ob, om);
            group_offsets32(p.ng, (uint32_t)(p.n0 + n0 + tile_col(half, c0 + c)), oa, ob, on);
            out[i] = p.C + oc + om + on;
            if (!plain_store) old[i] = *out[i];
        }
    }
    // a warp takes every kFinishRows-th column, lanes along the rows
    long long lo[PER] = {}, hi[PER] = {};
    const long long *at =
        p.parts + (size_t)e0 * PLANES * kPlane + (size_t)(half * kCols + c0 + warp) * kBM + quad * 32 + lane;
    // (eight slices at a time: complex 300 x 170 x 257 in nine slices 16.3 -> 14.5 us)
#pragma unroll 8
    for (int k = 0; k < p.ksplit; k++, at += CL * PLANES * kPlane) {
#pragma unroll
        for (int i = 0; i < PER; i++) {
            lo[i] += __ldcg(at + i * kFinishRows * kBM);
            if (F64) hi[i] += __ldcg(at + kPlane + i * kFinishRows * kBM);
        }
    }
    const int rowExp = lane < rows ? p.eA[(int64_t)b * p.Mp + m0 + lane] : 0;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int c = warp + i * kFinishRows;
        if (c >= live) break;
        const int colExp = p.eB[(int64_t)b * p.Np + n0 + tile_col(half, c0 + c)];
        const double v = finish_value<F64, false>(p, lo[i], hi[i], rowExp, colExp);
        tile[c][lane] = p.ab_pow2 ? v : p.ab * v;
    }
    if (__syncthreads_or(bad) || lost) { // the FMA kernel computes the region
        if (lost && blockIdx.x == 0 && threadIdx.x == 0) report_lost(p.status_at, p.status, lost);
        if (!lost && threadIdx.x == 0 && c0 == 0) list_region();
        return;
    }
#pragma unroll
    for (int i = 0; i < PER; i++)
        if (out[i]) *out[i] = plain_store ? *from[i] : fma(p.cp, old[i], *from[i]);
}

} // namespace

eg_status ensure_tc_attributes() {
    static PerDevice<cudaError_t> attributes;
    const cudaError_t err = attributes.get(current_device(), [] {
        cudaError_t err = cudaSuccess;
        for (const void *f : {(const void *)k_tc_split_gemm<false, 1, false>, (const void *)k_tc_split_gemm<true, 1, false>,
                              (const void *)k_tc_split_gemm<false, 2, false>, (const void *)k_tc_split_gemm<false, 1, true>,
                              (const void *)k_tc_split_gemm<false, 2, true>, (const void *)k_tc_split_gemm<true, 1, true>})
            if (err == cudaSuccess) err = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        return err;
    });
    if (err != cudaSuccess) return cuda_fail(err, "cudaFuncSetAttribute(k_tc_split_gemm)");
    return EG_SUCCESS;
}

namespace {
cudaLaunchConfig_t pair_config(int grid, cudaStream_t s, cudaLaunchAttribute *attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.stream = s;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = 2;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// EINSUMS_GB300_TC_PAIRS: 1 asks for CTA pairs wherever the output has two row
// tiles, 0 for single CTAs, anything else leaves the choice to the estimate.
int pairs_wish() {
    static const int wish = [] {
        const char *env = std::getenv("EINSUMS_GB300_TC_PAIRS");
        return env && (env[0] == '0' || env[0] == '1') ? env[0] - '0' : -1;
    }();
    return wish;
}
} // namespace

int tc_pair_clusters() {
    static PerDevice<int> clusters;
    return clusters.get(current_device(), [] {
        if (pairs_wish() == 0 || ensure_tc_attributes() != EG_SUCCESS) return 0;
        cudaLaunchAttribute attr;
        cudaLaunchConfig_t cfg = pair_config(num_sms(), nullptr, &attr);
        int c = 0;
        if (cudaOccupancyMaxActiveClusters(&c, (void *)k_tc_split_gemm<false, 2, false>, &cfg) != cudaSuccess) c = 0;
        cudaGetLastError();
        return c;
    });
}

bool tc_pairs_forced() { return pairs_wish() == 1 && tc_pair_clusters() > 0; }

eg_status launch_tc_gemm(const CUtensorMap &tmA, const CUtensorMap &tmB, const CUtensorMap &tmBh, const TcGemmParams &p,
                         cudaStream_t s) {
    eg_status st = ensure_tc_attributes();
    if (st != EG_SUCCESS) return st;
    const int CL = p.pair ? 2 : 1;
    const int workers = p.pair ? tc_pair_clusters() : num_sms();
    if (workers < 1) return fail(EG_ERROR_CUDA, "k_tc_split_gemm: CTA pairs are not available");
    const int total = p.t0 + (p.nbatch * ((p.mtiles + CL - 1) / CL) * p.ntiles - p.t0) * p.ksplit;
    if (total <= 0) return EG_SUCCESS;
    const int grid = CL * (total < workers ? total : workers);
    const bool f64 = p.redo != nullptr;
    {
        LaunchScope ls_(f64 ? "k_tc_split_gemm_f64" : "k_tc_split_gemm", s);
        const TcItem *no_items = nullptr;
        const int4 *no_work = nullptr;
        if (p.pair) {
            cudaLaunchAttribute attr;
            cudaLaunchConfig_t cfg = pair_config(grid, s, &attr);
            if (f64)
                EG_CUDA(cudaLaunchKernelEx(&cfg, k_tc_split_gemm<false, 2, true>, tmA, tmB, tmBh, p, no_items, no_work));
            else
                EG_CUDA(cudaLaunchKernelEx(&cfg, k_tc_split_gemm<false, 2, false>, tmA, tmB, tmBh, p, no_items, no_work));
        } else if (f64) {
            k_tc_split_gemm<false, 1, true><<<grid, THREADS, SMEM_BYTES, s>>>(tmA, tmB, tmBh, p, no_items, no_work);
        } else {
            k_tc_split_gemm<false, 1, false><<<grid, THREADS, SMEM_BYTES, s>>>(tmA, tmB, tmBh, p, no_items, no_work);
        }
    }
    EG_CHECK_LAUNCH("k_tc_split_gemm");
    const int slices = total - p.t0;
    if (p.ksplit > 1 && slices > 0) {
        {
            LaunchScope ls_("k_tc_finish_slices", s);
            auto finish = p.pair ? (f64 ? k_tc_finish_slices<2, true> : k_tc_finish_slices<2, false>)
                                 : (f64 ? k_tc_finish_slices<1, true> : k_tc_finish_slices<1, false>);
            finish<<<(unsigned)(slices / p.ksplit * CL * kTileRegions * kFinishParts), 32 * kFinishRows, 0, s>>>(p);
        }
        EG_CHECK_LAUNCH("k_tc_finish_slices");
    }
    return EG_SUCCESS;
}

eg_status launch_tc_gemm_grouped(const CUtensorMap &tmA, const CUtensorMap &tmB, const TcGemmParams &p,
                                 const TcItem *items, const int4 *work, int grid, cudaStream_t s) {
    eg_status st = ensure_tc_attributes();
    if (st != EG_SUCCESS) return st;
    if (grid <= 0) return EG_SUCCESS;
    {
        LaunchScope ls_(p.redo ? "k_tc_split_gemm_grouped_f64" : "k_tc_split_gemm_grouped", s);
        if (p.redo)
            k_tc_split_gemm<true, 1, true><<<grid, THREADS, SMEM_BYTES, s>>>(tmA, tmB, tmB, p, items, work);
        else
            k_tc_split_gemm<true, 1, false><<<grid, THREADS, SMEM_BYTES, s>>>(tmA, tmB, tmB, p, items, work);
    }
    EG_CHECK_LAUNCH("k_tc_split_gemm_grouped");
    return EG_SUCCESS;
}

} // namespace eg::split

extern "C" eg_status eg_tc_pair_clusters(int32_t *clusters) {
    if (!clusters) return eg::fail(EG_ERROR_INVALID_ARGUMENT, "eg_tc_pair_clusters: NULL output");
    *clusters = eg::split::tc_pairs_forced() ? eg::split::tc_pair_clusters() : 0;
    return EG_SUCCESS;
}
