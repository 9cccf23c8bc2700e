// Complex128 einsum with conjugation: eg_einsum_complex.
//
// The reference instantiates its einsum for std::complex<double> tensors and
// conjugates A or B through the ConjA / ConjB template flags
// (Backends/Dispatch.hpp:48,136; the generic loops of BaseAlgebra.hpp:33-38
// apply them per element), lowering to zgemm / zgemv / zdot.  Here a complex
// tensor is the pair of FP64 views of its interleaved storage -- the real parts
// at stride 2 s and the imaginary parts one double further on -- and the
// complex contraction is the real contractions of those views that make it up
// (with a = -1 for a conjugated A, b likewise):
//
//   Re(AB) = sum Ar Br - a b Ai Bi        Im(AB) = b sum Ar Bi + a sum Ai Br
//
// each one an eg_einsum through the same dispatch, so every algorithm choice
// and both precisions (FP64 and split-BF16) serve complex operands.  A real
// C_prefactor rides on the first contraction into each part, keeping the real
// path's zeroing rules; a complex one is applied first by k_complex_scale.
//
// An FP64 contraction with a real AB_prefactor runs once instead of four times: the real
// and imaginary parts become a mode p of C and a mode q of the sums, the larger operand
// serves both as it is stored, and the smaller is written out as the 2 x 2 real block of
// each of its elements.  One launch of four times the work fills the chip where four did
// not, the summed modes of an interleaved operand are contiguous, and the tensor cores pay
// for sizes where they would not for each of the four.
#include <algorithm>
#include <climits>

#include "common.cuh"

namespace eg {
eg_status einsum_impl(double cp, const int32_t *Cl, const eg_tensor *C, double ab, const int32_t *Al,
                      const eg_tensor *A, const int32_t *Bl, const eg_tensor *B, const eg_options *opt_in,
                      cudaStream_t stream, int32_t *alg_out);
void set_split_report(const eg_split_report &r);
eg_status classify_call(const int32_t *Cl, const eg_tensor *C, const int32_t *Al, const eg_tensor *A,
                        const int32_t *Bl, const eg_tensor *B, const eg_options *opt_in, int32_t *alg_out);

namespace {

__global__ void k_complex_scale(ModeGroup g, double *C, double cr, double ci) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.total; i += stride) {
        int64_t oa, ob, oc;
        group_offsets(g, i, oa, ob, oc);
        double *c = C + 2 * oc;
        const double re = c[0], im = c[1];
        c[0] = cr * re - ci * im;
        c[1] = cr * im + ci * re;
    }
}

// The real (part 0) or imaginary (part 1) FP64 view of a complex tensor.
eg_tensor part_view(const eg_tensor &t, int part) {
    eg_tensor v = t;
    v.data = t.data ? t.data + part : nullptr;
    for (int d = 0; d < t.rank && d < EG_MAX_RANK; d++) v.stride[d] = 2 * t.stride[d];
    return v;
}

// Element i of the smaller operand (g: its modes, strides 0 in the source and 1 in E) as
// the block E[q, p]: {re, -own other im} for the real part, {own im, other re} for the
// imaginary one, own and other -1 for a conjugated operand.
__global__ void __launch_bounds__(256) k_complex_blocks(ModeGroup g, const double *__restrict__ src, double *E,
                                                        int64_t sq, int64_t sp, double own, double other) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < (uint32_t)g.total; i += stride) {
        int64_t os, oe, unused;
        group_offsets32(g, i, os, oe, unused);
        const double re = __ldg(src + os), im = __ldg(src + os + 1);
        double *e = E + oe;
        e[0] = re;
        e[sq] = -(own * other) * im;
        e[sp] = own * im;
        e[sq + sp] = other * re;
    }
}

// g with a mode of extent 2 and the given strides as its fastest, its modes merged where
// all three operands allow; false when there is no room.
bool append_part(ModeGroup &g, int64_t s0, int64_t s1, int64_t s2) {
    if (g.n == kMaxModes) return false;
    const int64_t s[3] = {s0, s1, s2};
    ModeGroup out;
    for (int d = 0; d <= g.n; d++) {
        const bool part = d == g.n;
        const int64_t ext = part ? 2 : g.ext[d];
        bool merge = out.n > 0;
        for (int t = 0; t < 3 && merge; t++) merge = out.s[t][out.n - 1] == (part ? s[t] : g.s[t][d]) * ext;
        if (!merge) out.ext[out.n++] = 1;
        out.ext[out.n - 1] *= ext;
        for (int t = 0; t < 3; t++) out.s[t][out.n - 1] = part ? s[t] : g.s[t][d];
    }
    out.total = 2 * g.total;
    g = out;
    return true;
}

// The contraction c of the real parts as one real contraction of the whole complex
// operands (file comment).  NOT_SUPPORTED: the caller's four contractions, when the shape,
// a capture or the scratch say so.  300 x 170 x 257: 55 us on the tensor cores; FMAs take
// 125 us in one launch (83 us of the FP64 pipe) and in four 156 us, each with a last wave
// of its own and operands at stride 2.
constexpr int64_t kBlocksMax = int64_t(1) << 23; // elements of the smaller operand: 256 MB of blocks
eg_status launch_complex_blocks(Contraction c, double sa, double sb, cudaStream_t s) {
    if (c.k.n == 0 || c.m.n == 0 || c.n.n == 0) return EG_ERROR_NOT_SUPPORTED;
    const bool four_tensor = f64_tensor_pays(c); // each of the four contractions
    if (c.batch.n + c.m.n + c.n.n >= kMaxModes) return EG_ERROR_NOT_SUPPORTED;
    const int t = c.m.total < c.n.total ? 0 : 1; // the operand written out as blocks
    ModeGroup &f = t == 0 ? c.m : c.n, &k = c.k, &b = c.batch;
    if (b.n + f.n + k.n > kMaxModes || k.n == kMaxModes || f.n == kMaxModes) return EG_ERROR_NOT_SUPPORTED;
    const double rows = (double)f.total * (double)b.total;
    if (rows * (double)k.total > (double)kBlocksMax) return EG_ERROR_NOT_SUPPORTED;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    EG_CUDA(cudaStreamIsCapturing(s, &capturing));
    if (capturing != cudaStreamCaptureStatusNone) return EG_ERROR_NOT_SUPPORTED;

    // E's strides: batch, then the free modes and p, then the summed modes and q, or the
    // last two the other way round, as the operand itself is faster along the one or other
    auto fastest = [&](const ModeGroup &g) { return *std::min_element(g.s[t], g.s[t] + g.n); };
    const bool k_inner = fastest(k) <= fastest(f);
    ModeGroup src; // source strides 0, E's strides 1, slowest mode first
    int64_t step = 1, part[2] = {0, 0}; // strides of q and p
    ModeGroup *order[3] = {k_inner ? &k : &f, k_inner ? &f : &k, &b};
    int at = b.n + f.n + k.n;
    src.n = at;
    for (ModeGroup *g : order) {
        if (g != &b) {
            part[g == &k ? 0 : 1] = step;
            step *= 2;
        }
        for (int d = g->n - 1; d >= 0; d--) {
            at--;
            src.ext[at] = g->ext[d];
            src.s[0][at] = g->s[t][d];
            src.s[1][at] = step;
            src.total *= g->ext[d];
            g->s[t][d] = step;
            step *= g->ext[d];
        }
    }
    const double *from = t == 0 ? c.A : c.B;
    const bool room = t == 0 ? append_part(k, part[0], 1, 0) && append_part(f, part[1], 0, 1)
                             : append_part(k, 1, part[0], 0) && append_part(f, 0, part[1], 1);
    if (!room) return EG_ERROR_NOT_SUPPORTED;
    const size_t bytes = (size_t)step * sizeof(double);
    auto fill = [&](Contraction &x, void *E) -> eg_status {
        (t == 0 ? x.A : x.B) = (double *)E;
        {
            LaunchScope ls_("k_complex_blocks", s);
            const int64_t blocks = std::min<int64_t>((src.total + 255) / 256, (int64_t)num_sms() * 8);
            k_complex_blocks<<<(unsigned)blocks, 256, 0, s>>>(src, from, (double *)E, part[0], part[1], t == 0 ? sa : sb,
                                                              t == 0 ? sb : sa);
        }
        EG_CHECK_LAUNCH("k_complex_blocks");
        set_split_report(eg_split_report{0, 0, 0, 0.0});
        return EG_SUCCESS;
    };
    if (f64_tensor_pays(c)) {
        const eg_status st = launch_f64_tensor(c, s, bytes, fill);
        if (st != EG_ERROR_NOT_SUPPORTED) return st;
    }
    if (four_tensor) return EG_ERROR_NOT_SUPPORTED; // better than FMAs in one launch
    ScratchLease lease(s, bytes);
    if (!lease.ptr()) return EG_ERROR_NOT_SUPPORTED;
    const eg_status st = fill(c, lease.ptr());
    return st == EG_SUCCESS ? launch_contract_f64(c, s) : st;
}

} // namespace

} // namespace eg

namespace {

eg_status einsum_complex(const double *C_prefactor, const int32_t *C_labels, const eg_tensor *C,
                         const double *AB_prefactor, const int32_t *A_labels, const eg_tensor *A,
                         const int32_t *B_labels, const eg_tensor *B, int32_t conj_A, int32_t conj_B,
                         const eg_options *opt, void *stream, int32_t *algorithm_choice) {
    using namespace eg;
    if (!C_prefactor || !AB_prefactor) return fail(EG_ERROR_INVALID_ARGUMENT, "eg_einsum_complex: NULL prefactor");
    if (!C || !A || !B) return fail(EG_ERROR_INVALID_ARGUMENT, "eg_einsum_complex: NULL tensor");
    if (C->rank < 0 || C->rank > EG_MAX_RANK) return fail(EG_ERROR_RANK, "eg_einsum_complex: C rank out of range");
    cudaStream_t s = (cudaStream_t)stream;
    // the choice the reference reports for these complex tensors (their own strides)
    int32_t alg_c = 0;
    eg_status st0 = classify_call(C_labels, C, A_labels, A, B_labels, B, opt, &alg_c);
    if (st0 != EG_SUCCESS) return st0;
    if (algorithm_choice) *algorithm_choice = alg_c;
    const double cpr = C_prefactor[0], cpi = C_prefactor[1], abr = AB_prefactor[0], abi = AB_prefactor[1];
    const double sa = conj_A ? -1.0 : 1.0, sb = conj_B ? -1.0 : 1.0;
    double cp0 = cpr; // the prefactor of each part's first contraction
    if (cpi != 0.0) {
        ModeGroup g;
        g.n = C->rank;
        g.total = 1;
        for (int d = 0; d < C->rank; d++) {
            if (C->extent[d] < 0 || C->stride[d] < 0)
                return fail(EG_ERROR_DIMENSION, "eg_einsum_complex: negative extent or stride in C");
            g.ext[d] = C->extent[d];
            g.s[2][d] = C->stride[d];
            g.total *= C->extent[d];
        }
        if (g.total > 0) {
            if (!C->data) return fail(EG_ERROR_INVALID_ARGUMENT, "eg_einsum_complex: C data is NULL");
            const int64_t blocks = (g.total + 255) / 256;
            {
                LaunchScope ls_("k_complex_scale", s);
                k_complex_scale<<<(unsigned)(blocks < num_sms() * 8 ? blocks : num_sms() * 8), 256, 0, s>>>(
                    g, C->data, cpr, cpi);
            }
            EG_CHECK_LAUNCH("k_complex_scale");
        }
        cp0 = 1.0;
    }
    const eg_tensor Cr = part_view(*C, 0), Ci = part_view(*C, 1);
    const eg_tensor Ar = part_view(*A, 0), Ai = part_view(*A, 1);
    const eg_tensor Br = part_view(*B, 0), Bi = part_view(*B, 1);
    eg_options o;
    eg_options_default(&o);
    if (opt) o = *opt;
    if (abi == 0.0 && abr != 0.0 && o.precision == EG_PRECISION_FP64 &&
        (o.semantics == EG_SEMANTICS_CPP || o.semantics == EG_SEMANTICS_PYTHON)) {
        Contraction c;
        int32_t alg = 0;
        bool gemm_shaped = false;
        ListPattern pattern;
        eg_status st = lower_for_group(cp0, C_labels, &Cr, abr, A_labels, &Ar, B_labels, &Br, o, c, &alg, gemm_shaped,
                                       pattern);
        if (st != EG_SUCCESS) return st;
        if (gemm_shaped && (st = launch_complex_blocks(c, sa, sb, s)) != EG_ERROR_NOT_SUPPORTED) return st;
    }
    // (destination, A part, B part, coefficient): Re gets abr Pr - abi Pi, Im gets abr Pi + abi Pr
    struct Term {
        const eg_tensor *c, *a, *b;
        double coef;
    };
    const Term terms[8] = {
        {&Cr, &Ar, &Br, abr},           {&Cr, &Ai, &Bi, -abr * sa * sb}, {&Cr, &Ar, &Bi, -abi * sb},
        {&Cr, &Ai, &Br, -abi * sa},     {&Ci, &Ar, &Bi, abr * sb},       {&Ci, &Ai, &Br, abr * sa},
        {&Ci, &Ar, &Br, abi},           {&Ci, &Ai, &Bi, -abi * sa * sb},
    };
    bool first[2] = {true, true};
    for (const Term &t : terms) {
        const int part = t.c == &Cr ? 0 : 1;
        if (t.coef == 0.0 && !first[part]) continue;
        int32_t alg = 0;
        const eg_status st = einsum_impl(first[part] ? cp0 : 1.0, C_labels, t.c, t.coef, A_labels, t.a, B_labels, t.b,
                                         opt, s, &alg);
        if (st != EG_SUCCESS) return st;
        first[part] = false;
    }
    return EG_SUCCESS;
}

} // namespace

extern "C" eg_status eg_einsum_complex(const double *C_prefactor, const int32_t *C_labels, const eg_tensor *C,
                                       const double *AB_prefactor, const int32_t *A_labels, const eg_tensor *A,
                                       const int32_t *B_labels, const eg_tensor *B, int32_t conj_A, int32_t conj_B,
                                       const eg_options *opt, void *stream, int32_t *algorithm_choice) {
    eg::set_error("");
    try {
        return einsum_complex(C_prefactor, C_labels, C, AB_prefactor, A_labels, A, B_labels, B, conj_A, conj_B, opt,
                              stream, algorithm_choice);
    } catch (const std::exception &e) {
        return eg::fail(EG_ERROR_OUT_OF_MEMORY, e.what());
    }
}
