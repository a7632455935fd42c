// rms_walk_split.cu -- the split-precision walk (RMS_PREC_SPLIT).
//
// The same walk as the reference kernel `propagate` (hpc_code/lib/main.cu:
// 63-384, main_PGSE.cu:65-410) -- fixed-length isotropic steps, at most nite
// sub-segments, voxel-face reflection or Bernoulli(Pij) permeation, mirror
// walls, T2 weighting, moments and signal at the same records -- in the
// arithmetic a B200 issues fastest:
//
//  - position = voxel + FP32 offset inside it per axis (0..1, split_step.cuh).
//    A straight move is one FMA and a floor per axis.  The face loop works on
//    d_a, the distance to the next face in the direction of travel: the time
//    to a face is one multiply, and after any face event -- a cross into the
//    neighbour or a reflection -- the walker sits on that face with a whole
//    voxel ahead, d = 1 exactly, so no drift accumulates;
//  - the voxel is one linear index into a lattice padded with a one-voxel
//    border that holds a wall code: a face step is `lin += stride`, and
//    reaching a wall is a label like any other (rare branch); the integer
//    part of the displacement, D = voxel - origin image, is carried per axis;
//  - free flight: a voxel whose 26 neighbours all carry its label (and none
//    is a wall) has a flag bit in the lattice; a step that starts there is
//    shorter than a voxel, so it cannot meet a membrane or a wall and moves in
//    one straight line -- a floor per axis instead of the face loop.  It is
//    the face loop's own outcome (every face on the way is a same-label face,
//    always crossed) with at most three crossings, within the nite = 4 cap;
//  - labels one byte per voxel (7-bit label, wall = 127, plus the flag), or
//    packed 4 bits (3-bit label, wall = 7, plus the flag) where that keeps a
//    large lattice in the 126 MB L2 (a padded 256x256x2048 one is 68 MB);
//  - FP32 uniforms (21-bit), one Philox4x32-10 block per three steps;
//    hardware sine/cosine and reciprocal for the direction and face times;
//  - per-walker sums that grow over the walk (T2 exponent, PGSE displacement
//    sums) are carried in FP32 for at most 32 steps and folded into FP64;
//  - cross-walker sums: records staged in shared memory, and every few records
//    the FP32 products of a warp's walkers summed in FP64 and added with FP64
//    atomics into a few row sets per axon, which a last pass adds up (the
//    no-allocation walk: per-warp rows and an ordered reduction, rms_reduce.cu).
//
// Mirror walls: the reference mirrors the origin image at the end of a step
// for each wall the step touched (main.cu:302-310).  A step shorter than a
// voxel touches a wall at most once per axis and nothing else moves the
// origin during the step, so the mirror is applied at the wall event itself.
//
// Random streams (philox.cuh): per walker, direction uniforms of steps 3k,
// 3k+1 and 3k+2 come from one Philox4x32-10 block indexed by k, so all lanes of
// a warp generate in lock step; start positions and partial-permeation draws
// read their own sequential counter domains.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>

#include "philox.cuh"
#include "rms_internal.h"
#include "split_lattice.cuh"
#include "split_step.cuh"
#include "warp_reduce.cuh"

namespace rms {
namespace {

// Launch variants (block size, minimum resident blocks per SM): the second
// number caps registers per thread at 65536 / (block * minb), trading spills
// in the rare record path for more resident warps to hide gather latency.
struct SplitVariant { int block, minb; };
constexpr int kLeapCap = 64;   // equal-step-length leap: tries per step before staying put
constexpr SplitVariant kVariants[] = {{256, 4}, {256, 3}, {256, 2}, {128, 8}, {512, 2}};
constexpr int kNumVariants = sizeof(kVariants) / sizeof(kVariants[0]);

// General waveforms, at the end of bin `bin`: X (voxels) is the bin's
// displacement sum; every waveform's phase gets wave_b . X res, and the bin's
// mean displacement (um) goes to the trajectory output when one is given.
//
// Waveforms go four at a time: a phase is read from and written to the thread's
// scratch in L2, and one at a time each waited out that latency alone.  A
// trajectory row is 12 bytes a bin, one row per lane: written bin by bin, every
// store touched 32 sectors for a few bytes each, so kTrajBins bins wait in
// `wait` (local memory) and leave as 16-byte stores where rows are 16-byte
// aligned (traj_vec).
constexpr int kTrajBins = 8;
__device__ __noinline__ void wave_bin(const double* __restrict__ wave, int nwave, int bin, double X0, double X1,
                                      double X2, double res, double* ph, int nthr, float* traj, int64_t tw,
                                      int nbins, int bin_steps, int split, int vec, int64_t traj_n, uint32_t* wait) {
    const double x0 = X0 * res, x1 = X1 * res, x2 = X2 * res;
    const double* wv = wave + (size_t)bin * nwave * 3;
    int j = 0;
    for (; j + 4 <= nwave; j += 4) {
        double p[4], g[12];
#pragma unroll
        for (int q = 0; q < 4; ++q) p[q] = ph[(size_t)(j + q) * nthr];
#pragma unroll
        for (int q = 0; q < 12; ++q) g[q] = __ldg(wv + 3 * j + q);
#pragma unroll
        for (int q = 0; q < 4; ++q) p[q] += g[3 * q] * x0 + g[3 * q + 1] * x1 + g[3 * q + 2] * x2;
#pragma unroll
        for (int q = 0; q < 4; ++q) ph[(size_t)(j + q) * nthr] = p[q];
    }
    for (; j < nwave; ++j) ph[(size_t)j * nthr] += wv[3 * j] * x0 + wv[3 * j + 1] * x1 + wv[3 * j + 2] * x2;
    if (!traj || tw < 0) return;
    const double inv = 1.0 / (double)bin_steps;
    const float m[3] = {(float)(x0 * inv), (float)(x1 * inv), (float)(x2 * inv)};
    const size_t at = ((size_t)tw * nbins + bin) * 3;
    // split: BF16 pairs, hi = bf16(x), lo = bf16(x - hi): the operands of the
    // tensor-core contraction, split once here
    uint32_t word[3];   // hi | lo << 16
    if (split) {
        for (int k = 0; k < 3; ++k) {
            const __nv_bfloat16 h = __float2bfloat16_rn(m[k]);
            const __nv_bfloat16 l = __float2bfloat16_rn(m[k] - __bfloat162float(h));
            word[k] = (uint32_t)__bfloat16_as_ushort(h) | ((uint32_t)__bfloat16_as_ushort(l) << 16);
        }
    } else {
        for (int k = 0; k < 3; ++k) word[k] = __float_as_uint(m[k]);
    }
    if (!vec) {
        if (split) {
            unsigned short* hi = reinterpret_cast<unsigned short*>(traj);
            unsigned short* lo = hi + (size_t)traj_n * nbins * 3;
            for (int k = 0; k < 3; ++k) {
                hi[at + k] = (unsigned short)(word[k] & 0xffffu);
                lo[at + k] = (unsigned short)(word[k] >> 16);
            }
        } else {
            for (int k = 0; k < 3; ++k) traj[at + k] = __uint_as_float(word[k]);
        }
        return;
    }
    const int slot = bin % kTrajBins;
    for (int k = 0; k < 3; ++k) wait[3 * slot + k] = word[k];
    if (slot != kTrajBins - 1) return;
    const size_t first = at - 3 * (kTrajBins - 1);   // the batch's first bin
    uint32_t w[3 * kTrajBins];
#pragma unroll
    for (int q = 0; q < 3 * kTrajBins; ++q) w[q] = wait[q];
    if (split) {
        uint4* hi = reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(traj) + first);
        uint4* lo = reinterpret_cast<uint4*>(reinterpret_cast<unsigned short*>(traj) + (size_t)traj_n * nbins * 3 + first);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const uint32_t* e = w + 8 * q;
            hi[q] = make_uint4(__byte_perm(e[0], e[1], 0x5410), __byte_perm(e[2], e[3], 0x5410),
                               __byte_perm(e[4], e[5], 0x5410), __byte_perm(e[6], e[7], 0x5410));
            lo[q] = make_uint4(__byte_perm(e[0], e[1], 0x7632), __byte_perm(e[2], e[3], 0x7632),
                               __byte_perm(e[4], e[5], 0x7632), __byte_perm(e[6], e[7], 0x7632));
        }
    } else {
        uint4* out = reinterpret_cast<uint4*>(traj + first);
#pragma unroll
        for (int q = 0; q < 6; ++q) out[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    }
}

// A value into the totals: the no-allocation walk's rows are the warp's own
// (a plain add, summed in order afterwards), every other launch's are shared.
template <bool ONE>
__device__ __forceinline__ void add_out(double* p, double x) {
    if (ONE) *p += x;
    else atomicAdd(p, x);
}

// General waveforms, after the last step: the warp's sums of s0 cos(phase) and
// s0 sin(phase) per waveform, (cos, sin) pairs into the signal row.
template <bool ONE>
__device__ __noinline__ void wave_final(const double* ph, int nthr, int nwave, double s0, double* sig_slot,
                                        int lane) {
    for (int base = 0; base < 2 * nwave; base += 32) {
        double mine = 0.0;
        const int cnt = min(32, 2 * nwave - base);
        for (int k = 0; k < cnt; k += 2) {
            const int j = (base + k) >> 1;
            double sn, cs;
            sincos(ph[(size_t)j * nthr], &sn, &cs);
            const double rc = warp_sum(s0 * cs);
            const double rs = warp_sum(s0 * sn);
            if (lane == k) mine = rc;
            if (lane == k + 1) mine = rs;
        }
        if (lane < cnt) add_out<ONE>(sig_slot + base + lane, mine);
    }
}

// Records are taken in batches of KR: at a record every lane stages its
// walker's displacement and T2 weight in shared memory, and every KR
// records the warp adds the batch up.  With KR = 8, lane (r, g) = (lane % 8,
// lane / 8) sums six of record r's 22 moments [sig0, dx2 x6, dx4 x15] over the
// 32 walkers (FP32 products, FP64 sums): group g holds the six second-order
// products of A = s0, s0 x^2, s0 y^2 or s0 z^2, which are dx2 and, each once,
// dx4 (of the products that two groups could form one keeps its own column);
// the spare one of group 2 is sig0.  KR = 4 halves the walkers between two
// lanes.  A staged row is 4 x 32 floats and 4 of padding, so the 16-byte loads
// of KR lanes (four walkers of KR records) cover all banks.
//
// Why batches: one record at a time cost 32 shared loads, 32 FP32 -> FP64
// conversions (a 16-per-clock pipe), 32 FP64 adds and 22 stores per warp with
// one lane per column, and 10 warp reductions for the counts; here a
// warp-record costs five loads, 24 conversions and adds and ~30 paired products
// (__fmul2_rn: two walkers an instruction), no shuffle.  1e6 walkers x 2000
// steps on a 128x128x900 axon, walk kernel: 12.5 / 35.6 ms with 100 / 2000
// records one at a time, 12.3 / 27.1 in batches; 10.4 / 25.3 ms since the step
// itself is shorter (split_step.cuh).  KR = 8 up to 256 threads a block (4.2 KB of
// staging per warp), 4 above, so the static shared memory stays under 48 KB.
__host__ __device__ constexpr int rec_batch(int block) { return block <= 256 ? 8 : 4; }
constexpr int kStageRow = 4 * 32 + 4;   // floats of a staged record: x, y, z, s0 of 32 walkers, and 4 of padding
constexpr int kStageOnes = -4;          // before the first record, four ones

// Where the sums go.  ONE: the warp's own rows [timepoint][nvals] (plain adds).
// Otherwise one of the axon's ncopy row sets, moments as [column][tpad] so that
// the KR records of a batch are neighbours, by fire-and-forget FP64 atomics in
// L2: a few row sets shared by all warps stay in L2 and need neither a row set
// per warp (1.2 GB for 1000 records, cleared and streamed through HBM) nor a
// flush when a warp moves on to another axon.
template <int KR, bool ONE>
__device__ __noinline__ void add_moments(const float* st, const unsigned* msk, double* dst, int stride, int nrec,
                                         unsigned act, int nc, int nw, int lane) {
    constexpr int NW = 4 * KR;   // walkers per lane, of the tile's nw (the rest weigh nothing)
    const int r = lane & (KR - 1), g = (lane / KR) & 3, half = lane / (4 * KR);
    __syncwarp();
    double q0 = 0.0, q1 = 0.0, q2 = 0.0, q3 = 0.0, q4 = 0.0, q5 = 0.0;
    const float* row_st = st + r * kStageRow + half * NW;
    // the group's m with A = s0 m^2: ones, x, y or z
    const float* mp = g == 0 ? st + kStageOnes : row_st + (g - 1) * 32;
    const int minc = g == 0 ? 0 : 4;
#pragma unroll 1
    for (int k = 0; k < min(NW, nw - half * NW); k += 4, mp += minc) {
        const float4 X = *reinterpret_cast<const float4*>(row_st + k), Y = *reinterpret_cast<const float4*>(row_st + 32 + k),
                     Z = *reinterpret_cast<const float4*>(row_st + 64 + k),
                     S = *reinterpret_cast<const float4*>(row_st + 96 + k), M = *reinterpret_cast<const float4*>(mp);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            // two walkers at a time (paired FP32 products)
            const float2 x = h ? make_float2(X.z, X.w) : make_float2(X.x, X.y);
            const float2 y = h ? make_float2(Y.z, Y.w) : make_float2(Y.x, Y.y);
            const float2 z = h ? make_float2(Z.z, Z.w) : make_float2(Z.x, Z.y);
            const float2 s0 = h ? make_float2(S.z, S.w) : make_float2(S.x, S.y);
            const float2 m = h ? make_float2(M.z, M.w) : make_float2(M.x, M.y);
            const float2 A = __fmul2_rn(s0, __fmul2_rn(m, m)), Ax = __fmul2_rn(A, x);
            const float2 p0 = __fmul2_rn(A, __fmul2_rn(x, x)), p1 = __fmul2_rn(Ax, y), p2 = __fmul2_rn(Ax, z),
                         p3 = __fmul2_rn(A, __fmul2_rn(y, y)), p4 = __fmul2_rn(__fmul2_rn(A, y), z),
                         p5 = __fmul2_rn(A, __fmul2_rn(z, z));
            q0 += (double)(g == 2 ? s0.x : p0.x); q0 += (double)(g == 2 ? s0.y : p0.y);
            q1 += (double)p1.x; q1 += (double)p1.y;
            q2 += (double)p2.x; q2 += (double)p2.y;
            q3 += (double)p3.x; q3 += (double)p3.y;
            q4 += (double)p4.x; q4 += (double)p4.y;
            q5 += (double)p5.x; q5 += (double)p5.y;
        }
    }
    if (NW < 32) {
        q0 += __shfl_xor_sync(0xffffffffu, q0, 16); q1 += __shfl_xor_sync(0xffffffffu, q1, 16);
        q2 += __shfl_xor_sync(0xffffffffu, q2, 16); q3 += __shfl_xor_sync(0xffffffffu, q3, 16);
        q4 += __shfl_xor_sync(0xffffffffu, q4, 16); q5 += __shfl_xor_sync(0xffffffffu, q5, 16);
    }
    if (r >= nrec || half) return;
    double* row = ONE ? dst + (size_t)r * stride : dst + r;
    const size_t cs = ONE ? 1 : (size_t)stride;
    // columns of the group's six products (-1: another group's)
    const int c0 = g == 0 ? 1 : (g == 1 ? 7 : (g == 2 ? 0 : -1));
    const int c1 = g == 0 ? 2 : (g == 1 ? 8 : (g == 2 ? 13 : 15));
    const int c3 = g == 0 ? 4 : (g == 1 ? 10 : (g == 2 ? 17 : -1));
    const int c4 = g == 0 ? 5 : (g == 1 ? 11 : (g == 2 ? 18 : 20));
    if (c0 >= 0) add_out<ONE>(row + c0 * cs, q0);
    add_out<ONE>(row + c1 * cs, q1);
    add_out<ONE>(row + (c1 + 1) * cs, q2);
    if (c3 >= 0) add_out<ONE>(row + c3 * cs, q3);
    add_out<ONE>(row + c4 * cs, q4);
    add_out<ONE>(row + (c4 + 1) * cs, q5);
    // compartment counts from the staged label bits
    const unsigned m0 = msk[3 * r], m1 = msk[3 * r + 1], m2 = msk[3 * r + 2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int c = 2 * g + k;
        const int cnt = __popc(act & ((c & 1) ? m0 : ~m0) & ((c & 2) ? m1 : ~m1) & ((c & 4) ? m2 : ~m2));
        if (c < nc && cnt) add_out<ONE>(row + (kColCount + c) * cs, (double)cnt);
    }
}

// The batch's narrow-pulse signals: a lane (or several, signal_lanes) holds one
// b-value and adds s0 cos(q n.dx) over the tile's walkers, read as broadcasts
// from the staged rows -- one cosine, one conversion and one FP64 add per walker and b-value.
// One b-value at a time over the 32 lanes took 10 shuffles and 5 FP64 adds more.
template <bool ONE>
__device__ __noinline__ void add_signals(const float* st, const double* __restrict__ qtab,
                                         const double* __restrict__ bvec, int nb, double* dst, int stride, int nrec,
                                         int nw, int lane) {
    __syncwarp();
    auto group = [&](int jb, bool in, int first_w, int step, auto&& total) {
        const float bx = in ? (float)__ldg(bvec + jb * 3) : 0.0f, by = in ? (float)__ldg(bvec + jb * 3 + 1) : 0.0f,
                    bz = in ? (float)__ldg(bvec + jb * 3 + 2) : 0.0f;
        for (int r = 0; r < nrec; ++r) {
            const float q = in ? (float)__ldg(qtab + (size_t)r * nb + jb) : 0.0f;
            const float* v = st + r * kStageRow;
            auto cosine = [&](float dx, float dy, float dz, float s0) {
                const float qx = q * (dx * bx + dy * by + dz * bz);
                return (double)(s0 * cosf(qx));
            };
            double s = 0.0;
#pragma unroll 1
            for (int w = first_w; w < nw; w += step) {
                // past the tile's walkers the weights are zero
                const float4 X = *reinterpret_cast<const float4*>(v + w), Y = *reinterpret_cast<const float4*>(v + 32 + w),
                             Z = *reinterpret_cast<const float4*>(v + 64 + w), S = *reinterpret_cast<const float4*>(v + 96 + w);
                s += (cosine(X.x, Y.x, Z.x, S.x) + cosine(X.y, Y.y, Z.y, S.y)) +
                     (cosine(X.z, Y.z, Z.z, S.z) + cosine(X.w, Y.w, Z.w, S.w));
            }
            total(dst + (size_t)r * stride + jb, s);
        }
    };
    int base = 0;
    // a lane to a b-value, while more than half the lanes have one
    for (; nb - base > 16 || (base < nb && nw <= 4); base += 32) {
        const int jb = base + lane;
        if (jb < nb) group(jb, true, 0, 4, [&](double* p, double s) { add_out<ONE>(p, s); });
    }
    if (base < nb) {
        const SignalLanes l = signal_lanes(lane, nb - base, (nw + 3) / 4);   // (walkers go by fours)
        const int jb = base + l.item;
        const bool in = jb < nb;
        group(jb, in, 4 * l.share, 4 * l.shares, [&](double* p, double s) {
            s = share_sum(s, l);
            if (in && l.share == 0) add_out<ONE>(p, s);
        });
    }
}

constexpr int kPark = 22;
__device__ __forceinline__ void park_walker(volatile uint32_t* p, const SplitWalker& w, const DomainStream& perm,
                                            float q0, float q1, float q2, float q3) {
    p[0] = w.lin; p[1] = w.cell;
    p[2] = __float_as_uint(w.o0); p[3] = __float_as_uint(w.o1); p[4] = __float_as_uint(w.o2);
    p[5] = __float_as_uint(w.D0); p[6] = __float_as_uint(w.D1); p[7] = __float_as_uint(w.D2);
    p[8] = __float_as_uint(w.Fm0); p[9] = __float_as_uint(w.Fm1); p[10] = __float_as_uint(w.Fm2);
    p[11] = (uint32_t)w.ai; p[12] = __float_as_uint(w.cur_step); p[13] = __float_as_uint(w.cur_k);
    p[14] = __float_as_uint(w.w32);
    p[15] = perm.q1; p[16] = perm.q2; p[17] = perm.q3;
    p[18] = __float_as_uint(q0); p[19] = __float_as_uint(q1); p[20] = __float_as_uint(q2); p[21] = __float_as_uint(q3);
}
__device__ __forceinline__ void unpark_walker(const volatile uint32_t* p, SplitWalker& w, DomainStream& perm,
                                              float& q0, float& q1, float& q2, float& q3) {
    w.lin = p[0]; w.cell = p[1];
    w.o0 = __uint_as_float(p[2]); w.o1 = __uint_as_float(p[3]); w.o2 = __uint_as_float(p[4]);
    w.D0 = __uint_as_float(p[5]); w.D1 = __uint_as_float(p[6]); w.D2 = __uint_as_float(p[7]);
    w.Fm0 = __uint_as_float(p[8]); w.Fm1 = __uint_as_float(p[9]); w.Fm2 = __uint_as_float(p[10]);
    w.ai = (int)p[11]; w.cur_step = __uint_as_float(p[12]); w.cur_k = __uint_as_float(p[13]);
    w.w32 = __uint_as_float(p[14]);
    perm.q1 = p[15]; perm.q2 = p[16]; perm.q3 = p[17];
    q0 = __uint_as_float(p[18]); q1 = __uint_as_float(p[19]); q2 = __uint_as_float(p[20]); q3 = __uint_as_float(p[21]);
}

// Final T2-weighted PGSE signal of a tile, a lane (or several) to a gradient:
// phase_j = |g| (g_hat . V) res dt with the walkers' window sums V in vscr
// ([pair * 3 + axis][thread], thread t0 + w).  One gradient at a time over the
// 32 walkers took 10 shuffles and 5 FP64 adds more, and a warp's 32 lanes for
// however few walkers its tile has.
template <bool ONE>
__device__ __forceinline__ void add_pgse(const WalkArgs& a, int nthr, int t0, double s0, int nw, double* sig, int lane) {
    __syncwarp();
    const double scale = a.res * a.dt;
    for (int base = 0; base < a.ngrad; base += 32) {
        const SignalLanes l = signal_lanes(lane, min(32, a.ngrad - base), nw);
        const int j = min(base + l.item, a.ngrad - 1);
        const double* g = a.grad + 6 * j;
        const double* vv = a.vscr + (size_t)(a.gpair[j] * 3) * nthr + t0;
        const double g2 = g[2], g3 = g[3], g4 = g[4], g5 = g[5];
        double s = 0.0;
        for (int k = 0; k < nw; k += l.shares) {
            const int w = min(k + l.share, nw - 1);
            const double phase = g2 * (vv[w] * g3 + vv[nthr + w] * g4 + vv[2 * (size_t)nthr + w] * g5) * scale;
            const double sw = __shfl_sync(0xffffffffu, s0, w);
            s += (k + l.share < nw ? sw : 0.0) * cos(phase);
        }
        s = share_sum(s, l);
        if (base + l.item < a.ngrad && l.share == 0) add_out<ONE>(sig + j, s);
    }
    // the next tile's walkers clear these sums: every lane has read them by then
    // (a shuffle orders no memory)
    __syncwarp();
}

// ONE: the no-allocation walk's form -- one axon, whose scalars are read from
// the kernel parameters (a.axon0); every other launch reads the axon table.
template <int NCMAX, int BITS, int BLOCK, int MINB, bool ONE, int RULE = 0, int MODE = 0>
__global__ void __launch_bounds__(BLOCK, MINB) walk_split_kernel(const WalkArgs a) {
    // per warp, the current axon's tables: step (voxels), T2 exponent per voxel
    // of path, Pij and the step-length ratio that rescales the rest of a step
    constexpr int kTab = 2 * NCMAX + 2 * NCMAX * NCMAX;
    __shared__ float s_tab[BLOCK / 32][kTab];
    // per warp, a batch of records of its 32 walkers (add_moments) and the
    // bits of their labels
    constexpr int KR = rec_batch(BLOCK);
    __shared__ __align__(16) float s_stage[BLOCK / 32][4 + KR * kStageRow];
    __shared__ unsigned s_mask[BLOCK / 32][KR * 3];

    const int lane = threadIdx.x & 31;
    if (lane < 4) s_stage[threadIdx.x >> 5][lane] = 1.0f;   // kStageOnes
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nthr = gridDim.x * blockDim.x;
    const int warp_global = gtid >> 5;
    const int nwarps = nthr >> 5;
    float* tab = s_tab[threadIdx.x >> 5];
    // the signal mode is compiled in: a walk carries no code of the others
    constexpr bool pgse = (MODE == 1);
    constexpr bool wave = (MODE == 2);
    constexpr bool sums = pgse || wave;   // displacement sums over the walk
    const bool mirror = (a.boundary == 0);

    int ax = 0;          // current axon
    int held = -1;       // axon whose tables the warp holds
    int64_t next_tb = ONE ? INT64_MAX : ((a.naxons > 1) ? a.axons[1].tile_begin : INT64_MAX);
    // a field of the current axon: kernel parameters for ONE, else the axon
    // table (read where used, so it holds no registers)
#define AXF(f) (ONE ? a.axon0.f : a.axons[ax].f)

    // The table form (every SPLIT launch but the no-allocation walk, one axon
    // or many): a queue (one counter per launch) hands out tiles in order, so
    // the tiles in flight stay one narrow window of the list -- one or two
    // axons, whose lattices then share the L2 -- however far warps drift
    // apart.  ONE: tiles in strided order (warp w: w, w + nwarps, ...), so each
    // warp's rows, reduced in a fixed order, are the same every run.
    auto claim = [&]() -> int64_t {
        unsigned long long t = 0;
        if (lane == 0) t = atomicAdd(a.tile_ctr, 1ull);
        return (int64_t)__shfl_sync(0xffffffffu, t, 0);
    };
    for (int64_t tile = ONE ? warp_global : claim(); tile < a.ntiles; tile = ONE ? tile + nwarps : claim()) {
        if (!ONE) {
            while (tile >= next_tb) {
                ++ax;
                next_tb = (ax + 1 < a.naxons) ? a.axons[ax + 1].tile_begin : INT64_MAX;
            }
        }
        if (held != ax) {
            held = ax;
            // this axon's tables into the warp's shared memory
            __syncwarp();
            for (int i = lane; i < kTab; i += 32) {
                float v;
                if (i < NCMAX) v = AXF(step[i]);
                else if (i < 2 * NCMAX) v = AXF(k[i - NCMAX]);
                else if (i < 2 * NCMAX + NCMAX * NCMAX) {
                    const int r = (i - 2 * NCMAX) / NCMAX, c = (i - 2 * NCMAX) % NCMAX;
                    v = AXF(pij[r * kNcMax + c]);
                } else {
                    const int r = (i - 2 * NCMAX - NCMAX * NCMAX) / NCMAX, c = (i - 2 * NCMAX - NCMAX * NCMAX) % NCMAX;
                    v = AXF(ratio[r * kNcMax + c]);
                }
                tab[i] = v;
            }
            __syncwarp();
        }
        const uint8_t* lat = AXF(lat);
        const int s0 = AXF(s0), s1 = AXF(s1);
        const uint64_t seed = AXF(seed);   // a graph captures the table form, whose seed a replay rewrites
        const bool flight = AXF(flight);
        const bool same_certain = AXF(same_cross);
        const float* t_step = tab;
        const float* t_k = tab + NCMAX;
        const float* t_pij = tab + 2 * NCMAX;
        const float* t_ratio = tab + 2 * NCMAX + NCMAX * NCMAX;
        const uint32_t key0 = (uint32_t)seed, key1 = (uint32_t)(seed >> 32);

        // (the walkers past a narrow tile are the next tile's)
        const int tile_w = ONE ? 32 : a.tile_w;
        const int64_t w = AXF(walker_begin) + (tile - (ONE ? 0 : AXF(tile_begin))) * tile_w + lane;
        bool active = w < AXF(walker_end) && lane < tile_w;
        const uint32_t wlo = (uint32_t)w, whi = (uint32_t)((uint64_t)w >> 32);

        // initial position: uniform in the labelled voxels (rejection sampling)
        float f0 = 0.5f, f1 = 0.5f, f2 = 0.5f;
        unsigned lin = 0;
        if (active) {
            DomainStream init;
            init.init(seed, (uint64_t)w, kDomInit);
            long long tries = 0;
            for (;;) {
                const int n1 = AXF(n1), n2 = AXF(n2), n3 = AXF(n3);
                const float x0 = init.next() * (float)n1;
                const float x1 = init.next() * (float)n2;
                const float x2 = init.next() * (float)n3;
                const int g0 = min((int)x0, n1 - 1), g1 = min((int)x1, n2 - 1), g2 = min((int)x2, n3 - 1);
                f0 = x0 - (float)g0; f1 = x1 - (float)g1; f2 = x2 - (float)g2;
                lin = (unsigned)(g0 + 1) * (unsigned)s0 + (unsigned)(g1 + 1) * (unsigned)s1 + (unsigned)(g2 + 1);
                if (label_at<BITS>(lat, lin) != 0) break;
                if (++tries >= kInitTryCap) { atomicOr(a.err, kErrInitCap); active = false; break; }
            }
        }
        const int ai0 = active ? label_at<BITS>(lat, lin) : 0;
        // displacement = D + (offset - Fm) per axis
        SplitWalker wk{lin, active ? cell_at<BITS>(lat, lin) : 0u, f0, f1, f2, 0.0f, 0.0f, 0.0f, f0, f1, f2, ai0,
                        t_step[ai0], t_k[ai0], 0.0f};
        const SplitGeom geo{lat, s0, s1, floor_bias(s0, s1), a.nite, flight, same_certain, mirror};
        auto nsize = [&](int axis) { return axis == 0 ? AXF(n1) : (axis == 1 ? AXF(n2) : AXF(n3)); };
        NoHooks hooks;
        DomainStream perm;
        perm.init(seed, (uint64_t)w, kDomPerm);

        double w64 = 0.0;          // T2 exponent, folded
        double P0 = 0.0, P1 = 0.0, P2 = 0.0;   // displacement sums (voxels), folded
        float p0 = 0.0f, p1 = 0.0f, p2 = 0.0f;
        // records taken, and steps to go to the next one (step 0 is the first) or,
        // past the last, to the walk's end
        int rec = 0, left = 1;
        int evi = 0;   // next PGSE event, or current waveform bin
        int next_ev = pgse ? (a.nevents > 0 ? a.ev_step[0] : -1) : (wave ? a.bin_steps : -1);
        // the step that ends the FP32 sums: every 32nd, and every event
        int next_fold = next_ev > 0 ? min(32, next_ev) : 32;
        if (sums)
            for (int k = 0; k < (pgse ? a.npairs * 3 : a.nwave); ++k) a.vscr[(size_t)k * nthr + gtid] = 0.0;
        // direction uniforms: one Philox block per three steps, in lock step;
        // the next two steps' pairs wait in q0..q3 and move up (phase: how many)
        float q0 = 0.0f, q1 = 0.0f, q2 = 0.0f, q3 = 0.0f;
        int phase = 0;
        uint32_t dblk = 0u;

        uint32_t traj_wait[wave ? 3 * kTrajBins : 1];   // bins of this walker's trajectory not yet written
        for (int i = 0;; ++i) {
            float u1, u2;
            if (phase == 0) {
                float u[6];
                dir_fields(dir_block(dblk++, key0, key1, wlo, whi), u);
                u1 = u[0]; u2 = u[1]; q0 = u[2]; q1 = u[3]; q2 = u[4]; q3 = u[5];
                phase = 2;
            } else {
                u1 = q0; u2 = q1; q0 = q2; q1 = q3;
                --phase;
            }
            if (active) {
                // RULE != 0: the step's start, restored when a membrane turns the step back
                const SplitWalker start = wk;
                for (int attempt = 0;; ++attempt) {
                    float v0, v1, v2;
                    split_direction(u1, u2, v0, v1, v2);
                    const bool back = split_step<NCMAX, BITS, RULE>(wk, v0, v1, v2, geo, t_step, t_k, t_pij, t_ratio,
                                                                    perm, nsize, hooks);
                    if (RULE == 0 || !back) break;
                    // the step is taken back (interaction.m:256-345): rejection
                    // sampling stays put for the step; the equal-step-length leap
                    // redraws the direction (partial-permeation stream) and walks
                    // the step again, up to kLeapCap tries, then stays
                    wk = start;
                    if (RULE == 1 || attempt + 1 >= kLeapCap) {
                        wk.w32 = fmaf(wk.cur_step, wk.cur_k, wk.w32);   // the step's time passes in place
                        break;
                    }
                    u1 = perm.next();
                    u2 = perm.next();
                }
            }
            // in-voxel offsets of the current position
            const float o0 = wk.o0, o1 = wk.o1, o2 = wk.o2;
            const float D0 = wk.D0, D1 = wk.D1, D2 = wk.D2;
            const float Fm0 = wk.Fm0, Fm1 = wk.Fm1, Fm2 = wk.Fm2;

            if (sums) {
                // displacement sums (voxels): PGSE, prefix sums read at the
                // lobe edges; waveforms, one sum per time bin
                p0 += D0 + (o0 - Fm0);
                p1 += D1 + (o1 - Fm1);
                p2 += D2 + (o2 - Fm2);
                bool event = false;
                if (i + 1 == next_fold) {
                    P0 += (double)p0; P1 += (double)p1; P2 += (double)p2;
                    p0 = p1 = p2 = 0.0f;
                    event = (i + 1 == next_ev);
                    next_fold = ((i + 1) & ~31) + 32;
                    if (!event && next_ev > 0) next_fold = min(next_fold, next_ev);
                }
                if (event && wave) {
                    wave_bin(a.wave, a.nwave, evi, P0, P1, P2, (double)AXF(res), a.vscr + gtid, nthr, a.traj,
                             active ? w - AXF(walker_begin) : -1, a.nbins, a.bin_steps, a.traj_split, a.traj_vec, a.traj_n,
                             traj_wait);
                    P0 = P1 = P2 = 0.0;
                    ++evi;
                    next_ev += a.bin_steps;
                    next_fold = min(next_fold, next_ev);
                } else if (event) {
                    do {
                        const double cf = a.ev_coef[evi];
                        double* vv = a.vscr + (size_t)(a.ev_pair[evi] * 3) * nthr + gtid;
                        vv[0] += cf * P0;
                        vv[nthr] += cf * P1;
                        vv[2 * (size_t)nthr] += cf * P2;
                        ++evi;
                    } while (evi < a.nevents && a.ev_step[evi] == i + 1);
                    next_ev = (evi < a.nevents) ? a.ev_step[evi] : -1;
                    if (next_ev > 0) next_fold = min(next_fold, next_ev);
                }
            }

            if (--left == 0) {
                if (rec == a.timepoints) break;
                const int r = rec & (KR - 1), rec0 = rec - r;   // slot in the batch, the batch's first record
                ++rec;
                w64 += (double)wk.w32;
                wk.w32 = 0.0f;
                const float s0 = active ? expf(-(float)w64) : 0.0f;
                const float res = AXF(res);
                const float dx = (D0 + (o0 - Fm0)) * res;
                const float dy = (D1 + (o1 - Fm1)) * res;
                const float dz = (D2 + (o2 - Fm2)) * res;
                float* st = s_stage[threadIdx.x >> 5] + 4;
                unsigned* msk = s_mask[threadIdx.x >> 5];
                float* mine = st + r * kStageRow + lane;
                mine[0] = dx; mine[32] = dy; mine[64] = dz; mine[96] = s0;
                const unsigned b0 = __ballot_sync(0xffffffffu, wk.ai & 1), b1 = __ballot_sync(0xffffffffu, wk.ai & 2),
                               b2 = __ballot_sync(0xffffffffu, wk.ai & 4);
                if (lane < 3) msk[3 * r + lane] = lane == 0 ? b0 : (lane == 1 ? b1 : b2);
                if (r == KR - 1 || rec == a.timepoints) {
                    // the batch's sums into the totals (a warp's own rows, or one
                    // of the axon's row sets); the walker waits in local memory
                    // meanwhile, its registers are the sums' (left to itself the
                    // compiler keeps part of it there through the step loop)
                    volatile uint32_t park[kPark];
                    park_walker(park, wk, perm, q0, q1, q2, q3);
                    const unsigned act = __ballot_sync(0xffffffffu, active);
                    double* set = ONE ? a.slots + (size_t)warp_global * a.timepoints * a.nvals
                                      : a.rows + AXF(row_off) + (size_t)(warp_global % AXF(ncopy)) * a.row_sz;
                    add_moments<KR, ONE>(st, msk, ONE ? set + (size_t)rec0 * a.nvals : set + rec0,
                                         ONE ? a.nvals : a.tpad, rec - rec0, act, AXF(nc), tile_w, lane);
                    if (!sums && a.nbvec > 0)
                        add_signals<ONE>(st, a.qtab + (size_t)rec0 * a.nbvec, a.bvec, a.nbvec,
                                         ONE ? set + (size_t)rec0 * a.nvals + kRowHead
                                             : set + (size_t)kRowHead * a.tpad + (size_t)rec0 * a.nb_pad,
                                         ONE ? a.nvals : a.nb_pad, rec - rec0, tile_w, lane);
                    __syncwarp();
                    unpark_walker(park, wk, perm, q0, q1, q2, q3);
                }
                left = rec < a.timepoints ? a.tstep : a.tn - 1 - (rec - 1) * a.tstep;
                if (left == 0) break;
            }
        }
        if (sums) {
            double* sig_slot = ONE ? a.sig_slots + (size_t)warp_global * a.ngrad_pad
                                   : a.out_sig + (size_t)ax * a.ngrad_pad;
            if (wave) {
                wave_final<ONE>(a.vscr + gtid, nthr, a.nwave, active ? exp(-(w64 + (double)wk.w32)) : 0.0, sig_slot, lane);
            } else {
                add_pgse<ONE>(a, nthr, gtid - lane, active ? exp(-(w64 + (double)wk.w32)) : 0.0, tile_w, sig_slot, lane);
            }
        }
    }
}

#undef AXF

// Totals of every axon from its row sets, in the result fields' layout: axon
// k's block of `fields` doubles holds sig0 [T], dx2 [T][6], dx4 [T][15], counts
// [T][nc] and signals [T][nbvec], so the host copies each field as it lies.
__global__ void gather_rows_kernel(const WalkArgs a, double* __restrict__ out, size_t fields) {
    const AxonDesc* x = a.axons + blockIdx.y;
    const int T = a.timepoints, nc = x->nc, ncopy = x->ncopy;
    const double* src = a.rows + x->row_off;
    double* dst = out + (size_t)blockIdx.y * fields;
    const size_t n = (size_t)T * (kColCount + nc + a.nbvec);
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        // element e of the block -> (record, column) of the row sets
        size_t at;
        const size_t uT = (size_t)T;
        if (e < uT) at = e;
        else if (e < 7 * uT) { const size_t i = e - uT; at = (1 + i % 6) * a.tpad + i / 6; }
        else if (e < 22 * uT) { const size_t i = e - 7 * uT; at = (7 + i % 15) * a.tpad + i / 15; }
        else if (e < (22 + (size_t)nc) * uT) { const size_t i = e - 22 * uT; at = (kColCount + i % nc) * a.tpad + i / nc; }
        else {
            const size_t i = e - (22 + (size_t)nc) * uT;
            at = (size_t)kRowHead * a.tpad + i / a.nbvec * a.nb_pad + i % a.nbvec;
        }
        double s = 0.0;
        for (int c = 0; c < ncopy; ++c) s += __ldcs(src + (size_t)c * a.row_sz + at);
        dst[e] = s;
    }
}

// Padded lattice: (n1+2) x (n2+2) x (n3+2), interior = the labels, border =
// the wall code.  An interior voxel also gets the free-flight flag when its 26
// neighbours carry its label -- with mirror walls counting only the neighbours
// inside the lattice (a straight line out through a wall is reflected in the
// walk), with periodic walls only for voxels off the lattice's faces.
//
// Bound by the labels' bytes (read once from HBM, nine times from L1/L2).  One
// thread makes eight cells of a row from word loads of the nine rows around
// them: a byte that differs from the voxel's own label anywhere in the 3 x 3 x
// 3 block leaves a bit in `differ`, one three-input operation per word.  With
// 27 byte loads per voxel and 64-bit divisions per cell the 256x256x2048
// lattice took 3.51 ms, now 0.43.
struct RowWindow { unsigned w0, w1, w2; };   // 12 bytes of a label row

// Bytes s .. s + 11 of the labels (offsets from the word-aligned base; lo, hi:
// the labels' own).  CHECK: words without a byte of the labels are not read.
template <bool CHECK>
__device__ __forceinline__ RowWindow row_window(const uint8_t* __restrict__ base, int64_t s, int64_t lo, int64_t hi) {
    const int64_t a = s & ~(int64_t)3;
    const unsigned sh = (unsigned)(s & 3) * 8u;
    const unsigned* p = reinterpret_cast<const unsigned*>(base + a);
    unsigned l[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        l[q] = (!CHECK || (a + 4 * q + 4 > lo && a + 4 * q < hi)) ? __ldg(p + q) : 0u;
    return RowWindow{__funnelshift_r(l[0], l[1], sh), __funnelshift_r(l[1], l[2], sh), __funnelshift_r(l[2], l[3], sh)};
}

// The bits by which any of the 26 neighbours of the eight voxels kk .. kk + 7 of
// row (i, j) differ from their label; left, right: voxels with such a
// neighbour in the row.
template <bool CHECK>
__device__ __forceinline__ void differ(const uint8_t* __restrict__ base, int64_t mis, int n1, int n2, int n3, int i,
                                       int j, int kk, const unsigned (&left)[2], const unsigned (&right)[2],
                                       unsigned& c0, unsigned& c1, unsigned& d0, unsigned& d1) {
    const int64_t lo = mis, hi = mis + (int64_t)n1 * n2 * n3, s = mis + ((int64_t)i * n2 + j) * n3 + kk - 1;
    const RowWindow c = row_window<CHECK>(base, s, lo, hi);
    c0 = __funnelshift_r(c.w0, c.w1, 8);
    c1 = __funnelshift_r(c.w1, c.w2, 8);
    d0 = d1 = 0u;
#pragma unroll
    for (int di = -1; di <= 1; ++di) {
#pragma unroll
        for (int dj = -1; dj <= 1; ++dj) {
            // a row outside the lattice: the voxels' own row again, which adds nothing
            const bool out = i + di < 0 || i + di >= n1 || j + dj < 0 || j + dj >= n2;
            const int64_t q = out ? s : s + ((int64_t)di * n2 + dj) * n3;
            const RowWindow w = (di == 0 && dj == 0) ? c : row_window<CHECK>(base, q, lo, hi);
            d0 |= (w.w0 ^ c0) & left[0];
            d1 |= (w.w1 ^ c1) & left[1];
            d0 |= __funnelshift_r(w.w0, w.w1, 8) ^ c0;
            d1 |= __funnelshift_r(w.w1, w.w2, 8) ^ c1;
            d0 |= (__funnelshift_r(w.w0, w.w1, 16) ^ c0) & right[0];
            d1 |= (__funnelshift_r(w.w1, w.w2, 16) ^ c1) & right[1];
        }
    }
}

// Cells k0 .. k0 + 7 of the padded row (pi, pj) as bytes (label | flag << 7),
// the wall as 0x7f; cells past the row's end are undefined.
__device__ __forceinline__ uint2 row_cells(const uint8_t* __restrict__ base, int64_t mis, int n1, int n2, int n3,
                                           bool mirror, unsigned pi, unsigned pj, int k0) {
    const unsigned kWalls = 0x7f7f7f7fu;
    if (pi == 0 || pi > (unsigned)n1 || pj == 0 || pj > (unsigned)n2) return make_uint2(kWalls, kWalls);
    const int i = (int)pi - 1, j = (int)pj - 1, kk = k0 - 1;   // the first cell's voxel
    // byte t of the masks: voxel kk + t has a left (right) neighbour in the row; is in the row
    unsigned left[2], right[2], in[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        left[h] = right[h] = in[h] = 0xffffffffu;
        const int f = kk + 4 * h;
        if (f < 1 || f + 4 >= n3) {   // near a row end
            left[h] = right[h] = in[h] = 0u;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if (f + t >= 1) left[h] |= 0xffu << (8 * t);
                if (f + t + 1 < n3) right[h] |= 0xffu << (8 * t);
                if (f + t >= 0 && f + t < n3) in[h] |= 0xffu << (8 * t);
            }
        }
    }
    unsigned c0, c1, d0, d1;
    // all nine windows inside the labels: no bounds to look at
    const int64_t n = (int64_t)n1 * n2 * n3, at = ((int64_t)i * n2 + j) * n3 + kk, reach = ((int64_t)n2 + 1) * n3 + 16;
    if (at >= reach && at + reach <= n) differ<false>(base, mis, n1, n2, n3, i, j, kk, left, right, c0, c1, d0, d1);
    else differ<true>(base, mis, n1, n2, n3, i, j, kk, left, right, c0, c1, d0, d1);
    // flag (bit 7) where no bit of the byte differs
    unsigned f0 = ~(((d0 & kWalls) + kWalls) | d0) & 0x80808080u, f1 = ~(((d1 & kWalls) + kWalls) | d1) & 0x80808080u;
    if (!mirror) {
        const bool inner = i >= 1 && i + 1 < n1 && j >= 1 && j + 1 < n2;
        f0 = inner ? f0 & left[0] & right[0] : 0u;
        f1 = inner ? f1 & left[1] & right[1] : 0u;
    }
    return make_uint2((((c0 & kWalls) | f0) & in[0]) | (kWalls & ~in[0]), (((c1 & kWalls) | f1) & in[1]) | (kWalls & ~in[1]));
}

// four cells of row_cells as nibbles (3-bit label, flag in bit 3)
__device__ __forceinline__ unsigned nibbles(unsigned c) {
    c = (c & 0x07070707u) | ((c >> 4) & 0x08080808u);
    c |= c >> 4;
    return (c & 0xffu) | ((c >> 8) & 0xff00u);
}

template <int BITS>
__global__ void pad_pack_kernel(const uint8_t* __restrict__ labels, int n1, int n2, int n3, int mirror,
                                uint8_t* __restrict__ out, size_t nbytes) {
    const int64_t mis = (int64_t)(reinterpret_cast<uintptr_t>(labels) & 3u);
    const uint8_t* base = labels - mis;
    const unsigned P3 = (unsigned)n3 + 2u, P2 = (unsigned)n2 + 2u;
    const unsigned nvox = (unsigned)(((size_t)n1 + 2) * P2 * P3);   // below 2^32
    const size_t groups = ((size_t)nvox + 7) / 8;
    for (size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x; g < groups; g += (size_t)gridDim.x * blockDim.x) {
        const unsigned p0 = (unsigned)(g * 8);
        unsigned row = p0 / P3;
        int k = (int)(p0 - row * P3);
        // the group's eight cells: one row's, or the end of one and the start of the next (rows may be
        // shorter than the group)
        unsigned long long cells = 0ull;
        for (int t = 0; t < 8;) {
            const unsigned pi = row / P2, pj = row - pi * P2;   // past the last row: pi > n1, wall
            const uint2 c = row_cells(base, mis, n1, n2, n3, mirror != 0, pi, pj, k);
            const unsigned long long v = ((unsigned long long)c.y << 32) | c.x;
            const int n = min(8 - t, (int)P3 - k);
            cells |= (n < 8 ? v & ((1ull << (8 * n)) - 1ull) : v) << (8 * t);
            t += n;
            ++row;
            k = 0;
        }
        const unsigned lo = (unsigned)cells, hi = (unsigned)(cells >> 32);
        if (BITS == 4) {
            const unsigned v = nibbles(lo) | (nibbles(hi) << 16);
            if (g * 4 + 4 <= nbytes) reinterpret_cast<unsigned*>(out)[g] = v;
            else
                for (size_t q = g * 4; q < nbytes; ++q) out[q] = (uint8_t)(v >> (8 * (q - g * 4)));
        } else {
            if (g * 8 + 8 <= nbytes) reinterpret_cast<uint2*>(out)[g] = make_uint2(lo, hi);
            else
                for (size_t q = g * 8; q < nbytes; ++q) out[q] = (uint8_t)(cells >> (8 * (q - g * 8)));
        }
    }
}

template <int NCMAX, int BITS, int B, int M, int MODE, int RULE>
int launch_k(const WalkArgs& a, int grid, void* stream) {
    if (a.naxons == 1 && !a.table_form)
        walk_split_kernel<NCMAX, BITS, B, M, true, RULE, MODE><<<grid, B, 0, (cudaStream_t)stream>>>(a);
    else
        walk_split_kernel<NCMAX, BITS, B, M, false, RULE, MODE><<<grid, B, 0, (cudaStream_t)stream>>>(a);
    return (int)cudaGetLastError();
}

// Launch variants 2.. walk narrow-pulse and PGSE jobs with reflecting
// membranes; the first variant also walks waveforms and the alternative
// membrane rules (rejection sampling, equal-step-length leap).
template <int NCMAX, int BITS, int B, int M>
int launch_modes(const WalkArgs& a, int grid, void* stream) {
    if (a.rule != 0) return (int)cudaErrorInvalidValue;
    if (a.mode == 0) return launch_k<NCMAX, BITS, B, M, 0, 0>(a, grid, stream);
    if (a.mode == 1) return launch_k<NCMAX, BITS, B, M, 1, 0>(a, grid, stream);
    return (int)cudaErrorInvalidValue;
}

template <int NCMAX, int BITS>
int launch_first(const WalkArgs& a, int grid, void* stream) {
    constexpr int B = kVariants[0].block, M = kVariants[0].minb;
    switch (a.mode * 3 + a.rule) {
        case 0: return launch_k<NCMAX, BITS, B, M, 0, 0>(a, grid, stream);
        case 1: return launch_k<NCMAX, BITS, B, M, 0, 1>(a, grid, stream);
        case 2: return launch_k<NCMAX, BITS, B, M, 0, 2>(a, grid, stream);
        case 3: return launch_k<NCMAX, BITS, B, M, 1, 0>(a, grid, stream);
        case 4: return launch_k<NCMAX, BITS, B, M, 1, 1>(a, grid, stream);
        case 5: return launch_k<NCMAX, BITS, B, M, 1, 2>(a, grid, stream);
        case 6: return launch_k<NCMAX, BITS, B, M, 2, 0>(a, grid, stream);
        case 7: return launch_k<NCMAX, BITS, B, M, 2, 1>(a, grid, stream);
        case 8: return launch_k<NCMAX, BITS, B, M, 2, 2>(a, grid, stream);
        default: return (int)cudaErrorInvalidValue;
    }
}

template <int BLOCK, int MINB>
const void* kernel_ptr(int bits) {
    if (bits == 4) return (const void*)walk_split_kernel<8, 4, BLOCK, MINB, false>;
    return (const void*)walk_split_kernel<8, 8, BLOCK, MINB, false>;
}

template <int BLOCK, int MINB>
int launch_v(const WalkArgs& a, int bits, int grid, void* stream) {
    if (bits == 4) return a.nc <= 7 ? launch_modes<8, 4, BLOCK, MINB>(a, grid, stream) : (int)cudaErrorInvalidValue;
    if (bits == 8) return launch_modes<8, 8, BLOCK, MINB>(a, grid, stream);
    return (int)cudaErrorInvalidValue;
}

// Dispatch over the variant table (index v, 0-based).
template <class F>
auto by_variant(int v, F&& f) {
    switch (v) {
        case 0: return f.template operator()<256, 4>();
        case 1: return f.template operator()<256, 3>();
        case 2: return f.template operator()<256, 2>();
        case 3: return f.template operator()<128, 8>();
        default: return f.template operator()<512, 2>();
    }
}

}  // namespace

int split_lattice_bits(int nc) { return nc <= 7 ? 4 : 8; }

size_t padded_lattice_bytes(int n1, int n2, int n3, int bits) {
    const size_t nv = ((size_t)n1 + 2) * ((size_t)n2 + 2) * ((size_t)n3 + 2);
    return (nv * (size_t)bits + 7) / 8;
}

int pack_lattice_padded(const uint8_t* labels, int n1, int n2, int n3, int bits, int mirror, uint8_t* out,
                        void* stream) {
    const size_t nbytes = padded_lattice_bytes(n1, n2, n3, bits);
    size_t grid = (nbytes * 8 / bits / 8 + 255) / 256 + 1;   // a thread per eight cells
    if (grid > 65536) grid = 65536;
    if (bits == 4)
        pad_pack_kernel<4><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(labels, n1, n2, n3, mirror, out, nbytes);
    else
        pad_pack_kernel<8><<<(unsigned)grid, 256, 0, (cudaStream_t)stream>>>(labels, n1, n2, n3, mirror, out, nbytes);
    return (int)cudaGetLastError();
}

int launch_gather_rows(const WalkArgs& a, double* out, size_t fields, void* stream) {
    const size_t n = (size_t)a.timepoints * (kColCount + kNcMax + a.nbvec);
    const unsigned gx = (unsigned)std::min<size_t>((n + 255) / 256, 1024);
    for (int k = 0; k < a.naxons; k += 32768) {   // grid.y holds at most 65535 axons
        WalkArgs b = a;
        b.axons += k;
        gather_rows_kernel<<<dim3(gx, (unsigned)std::min(32768, a.naxons - k)), 256, 0, (cudaStream_t)stream>>>(
            b, out + (size_t)k * fields, fields);
    }
    return (int)cudaGetLastError();
}

int split_variant_count() { return kNumVariants; }
int split_variant_block(int v) { return (v >= 0 && v < kNumVariants) ? kVariants[v].block : -1; }
int split_variant_minb(int v) { return (v >= 0 && v < kNumVariants) ? kVariants[v].minb : -1; }

int launch_walk_split(const WalkArgs& a, int lattice_bits, int variant, int grid, void* stream) {
    if (variant < 0 || variant >= kNumVariants) return (int)cudaErrorInvalidValue;
    if (a.mode < 0 || a.mode > 2 || a.rule < 0 || a.rule > 2) return (int)cudaErrorInvalidValue;
    if (variant == 0) {
        if (lattice_bits == 4) return a.nc <= 7 ? launch_first<8, 4>(a, grid, stream) : (int)cudaErrorInvalidValue;
        if (lattice_bits == 8) return launch_first<8, 8>(a, grid, stream);
        return (int)cudaErrorInvalidValue;
    }
    return by_variant(variant, [&]<int B, int M>() { return launch_v<B, M>(a, lattice_bits, grid, stream); });
}

bool split_variant_walks(int variant, int mode, int rule) { return variant == 0 || (mode != 2 && rule == 0); }

int walk_split_blocks_per_sm(int nc, int lattice_bits, int variant) {
    if (variant < 0 || variant >= kNumVariants) return -1;
    const void* k = by_variant(variant, [&]<int B, int M>() { return kernel_ptr<B, M>(lattice_bits); });
    int n = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kVariants[variant].block, 0);
    return e == cudaSuccess ? n : -1;
}

}  // namespace rms
