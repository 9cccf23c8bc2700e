// The sums of one T x T tile of outputs on the FP64 pipe, by the 256 threads of a CTA: the
// inner part of k_contract_f64 (kernels_fp64.cu, which says why tiles are small) and of the
// kernel that computes what the tensor cores leave out of a list (grouped.cu).
#pragma once

#include "common.cuh"
#include "ptx.cuh"

namespace eg::f64 {

constexpr int kThreads = 256, kStages = 3;

template <int T>
struct Tile {
    static constexpr int R = T == 32 ? 2 : 1; // outputs of a thread along each side
    static constexpr int KG = kThreads / ((T / R) * (T / R)); // groups of threads along k
    static constexpr int BK = T == 32 ? 16 : 32;
    static constexpr int LD = T + 1;
    static constexpr int PER = T * BK / kThreads; // elements a thread loads per operand and chunk
};

template <int T>
struct Buffers {
    double A[kStages][Tile<T>::BK][Tile<T>::LD];
    double B[kStages][Tile<T>::BK][Tile<T>::LD];
};

// One contraction at one batch index.
struct Operands {
    const ModeGroup &m, &n, &k;
    const double *A, *B;
    int a_kfast, b_kfast; // the operand is read along k (its smaller stride), else along its rows
    int64_t ka, kb;       // single k strides of A and B (0: none)
};

// How a k index becomes an element offset of one operand: a single stride when
// the group's modes nest in it, else the decomposition over the modes.
__device__ __forceinline__ int64_t k_offset(const ModeGroup &kg, int64_t stride, int comp, uint32_t k) {
    if (stride) return (int64_t)k * stride;
    int64_t oa, ob, oc;
    group_offsets32(kg, k, oa, ob, oc);
    return comp ? ob : oa;
}

// Adds to acc[i][j] the sums of output (ty + W i, tx + W j) of the tile at (m0, n0), W = T / R,
// over the chunks cbeg .. cend - 1 of BK k, of which this thread's k group takes its part.
// Column j of the tile is column j + (j & gap) from its first.
template <int T>
__device__ __forceinline__ void accumulate(Buffers<T> &sh, const Operands &o, int64_t m0, int64_t n0, int gap, int cbeg,
                                           int cend, double (&acc)[Tile<T>::R][Tile<T>::R]) {
    using Q = Tile<T>;
    constexpr int R = Q::R, KG = Q::KG, BK = Q::BK, PER = Q::PER, W = T / R;
    const int tid = threadIdx.x;
    const int kgrp = tid / (W * W), tx = tid % W, ty = (tid / W) % W;
    const int64_t M = o.m.total, N = o.n.total, K = o.k.total;
    int am[PER], ak[PER], bn[PER], bk[PER];
    const double *pa[PER], *pb[PER];
    bool oka[PER], okb[PER];
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int e = tid + kThreads * i;
        am[i] = o.a_kfast ? e / BK : e % T;
        ak[i] = o.a_kfast ? e % BK : e / T;
        bn[i] = o.b_kfast ? e / BK : e % T;
        bk[i] = o.b_kfast ? e % BK : e / T;
        int64_t oa, ob, oc;
        oka[i] = m0 + am[i] < M;
        group_offsets32(o.m, (uint32_t)(oka[i] ? m0 + am[i] : 0), oa, ob, oc);
        pa[i] = o.A + oa;
        const int64_t n = n0 + bn[i] + (bn[i] & gap);
        okb[i] = n < N;
        group_offsets32(o.n, (uint32_t)(okb[i] ? n : 0), oa, ob, oc);
        pb[i] = o.B + ob;
    }
    auto load = [&](int c) {
        if (c < cend) {
            const int slot = (c - cbeg) % kStages;
#pragma unroll
            for (int i = 0; i < PER; i++) {
                const int64_t ka = (int64_t)c * BK + ak[i], kb = (int64_t)c * BK + bk[i];
                const bool va = oka[i] && ka < K, vb = okb[i] && kb < K;
                ptx::cp_async8(&sh.A[slot][ak[i]][am[i]], va ? pa[i] + k_offset(o.k, o.ka, 0, (uint32_t)ka) : pa[i], va);
                ptx::cp_async8(&sh.B[slot][bk[i]][bn[i]], vb ? pb[i] + k_offset(o.k, o.kb, 1, (uint32_t)kb) : pb[i], vb);
            }
        }
        ptx::cp_async_commit();
    };
    load(cbeg);
    load(cbeg + 1);
    for (int c = cbeg; c < cend; c++) {
        ptx::cp_async_wait<1>();
        __syncthreads(); // chunk c has landed for every thread, and chunk c - 1 is read
        load(c + 2);
        const int slot = (c - cbeg) % kStages;
#pragma unroll 8
        for (int kk = kgrp; kk < BK; kk += KG) {
            double a[R], v[R];
#pragma unroll
            for (int i = 0; i < R; i++) a[i] = sh.A[slot][kk][ty + W * i];
#pragma unroll
            for (int j = 0; j < R; j++) v[j] = sh.B[slot][kk][tx + W * j];
#pragma unroll
            for (int i = 0; i < R; i++)
#pragma unroll
                for (int j = 0; j < R; j++) acc[i][j] = fma(a[i], v[j], acc[i][j]);
        }
    }
    ptx::cp_async_wait<0>();
}

} // namespace eg::f64
