// rms_walk_compat.cu -- the FP64, reference-compatible walk (RMS_PREC_COMPAT).
//
// Same per-walker algorithm as the reference kernel `propagate`
// (hpc_code/lib/main.cu:63-384 narrow pulse, main_PGSE.cu:65-410 PGSE): FP64
// positions, FP64 uniforms in the same draw order, the same sub-segment rule,
// mirror walls and Pij decisions, so a walker's voxel and event sequence is
// the CPU oracle's.  This file is compiled with -fmad=false: every product and
// sum is rounded like the reference's own expressions.
//
// What differs from the reference, by design:
//  - cross-walker sums: records staged in shared memory and added up in batches,
//    by a lane per group of columns or per b-value, into per-warp FP64 rows, then
//    one ordered reduction (no CAS atomics, repeatable);
//  - PGSE phase: per walker the displacement sums over each gradient's two
//    lobes are formed from running prefix sums at the lobe edges, instead of
//    an O(Ngrad) update every step into a 16 KB local array
//    (main_PGSE.cu:99-100, 340-346).  phase_j = |g| (g_hat . V_j) dt with
//    V_j = sum_{lobe 1} dx - sum_{lobe 2} dx is the same sum, reassociated;
//  - walls: periodic as an option beside the reference's mirror;
//  - persistent grid: each warp walks a tile of walkers at a time, 32 or fewer
//    (tile_width in rms_api.cpp), tiles strided by the number of warps in the grid.
#include <cuda_runtime.h>
#include <math.h>

#include "philox.cuh"
#include "rms_internal.h"
#include "warp_reduce.cuh"

namespace rms {
namespace {

constexpr double kRefPi = 3.14159265;  // main.cu:34 (the reference's truncated pi)
constexpr int kBlock = 128;

__device__ __forceinline__ unsigned lin3(int i, int j, int k, int n2, int n3) {
    return ((unsigned)i * (unsigned)n2 + (unsigned)j) * (unsigned)n3 + (unsigned)k;
}

// Time to the face ahead on one axis, as the reference forms it (main.cu:200-219):
// d = face - x, beyond a whole step 2, never negative.
__device__ __forceinline__ double face_time(double d, double v) {
    if (fabs(d) > fabs(v)) return 2.0;
    const double q = d / v;
    return (0.0 < q) ? q : 0.0;  // std::max(0.0, q)
}

// a / b rounded to nearest from y = 1 / b rounded to nearest: two residual
// corrections of a * y.  The first leaves a quotient within an ulp, from which
// the second is the correctly rounded one (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 1990, theorem 8.3) -- the division's own result, without forming the
// reciprocal of the same b again for every a.
__device__ __forceinline__ double div_by(double a, double b, double y, double q) {   // q: a * y
    q = __fma_rn(__fma_rn(-q, b, a), y, q);
    return __fma_rn(__fma_rn(-q, b, a), y, q);
}

__device__ __forceinline__ double div_by(double a, double b, double y) { return div_by(a, b, y, __dmul_rn(a, y)); }

// Records in batches of kRec, as the split walk takes them
// (rms_walk_split.cu): every lane stages its walker's displacement and T2
// weight, then lane (r, g) adds six of record r's moments over the tile's
// walkers; lane j of the signals holds one b-value.  One record at a time cost
// a 32-value FP64 reduce-scatter (~270 instructions), and each b-value 10
// shuffles and 5 adds after its cosine.
constexpr int kRec = 8;
// doubles of a staged record: x, y, z, s0 of 32 walkers, then 16 bytes that keep
// the rows of a batch on different banks and hold the bits of the labels
constexpr int kStageRow = 4 * 32 + 2;
__device__ __forceinline__ unsigned* stage_masks(double* row) { return reinterpret_cast<unsigned*>(row + 4 * 32); }

// A value into the warp's row: the warp's first tile stores, later ones add
// (so the rows need no clearing).
__device__ __forceinline__ void put(double* p, double x, bool first) { *p = first ? x : *p + x; }

__device__ __noinline__ void add_moments(double* st, double* row, int nvals, int nrec, unsigned act,
                                         int nw, bool first, int lane) {
    const int r = lane & (kRec - 1), g = lane / kRec;
    __syncwarp();
    double q0 = 0.0, q1 = 0.0, q2 = 0.0, q3 = 0.0, q4 = 0.0, q5 = 0.0;
    const double* v = st + r * kStageRow;
#pragma unroll 2
    for (int w = 0; w < nw; ++w) {
        const double x = v[w], y = v[32 + w], z = v[64 + w], s0 = v[96 + w];
        const double m = g == 1 ? x : (g == 2 ? y : z);
        const double A = g == 0 ? s0 : s0 * m * m, Ax = A * x, Ay = A * y;
        q0 += g == 2 ? s0 : Ax * x;
        q1 += Ax * y;
        q2 += Ax * z;
        q3 += Ay * y;
        q4 += Ay * z;
        q5 += A * z * z;
    }
    if (r >= nrec) return;
    row += (size_t)r * nvals;
    // columns of the group's six products (-1: another group's)
    const int c0 = g == 0 ? 1 : (g == 1 ? 7 : (g == 2 ? 0 : -1));
    const int c1 = g == 0 ? 2 : (g == 1 ? 8 : (g == 2 ? 13 : 15));
    const int c3 = g == 0 ? 4 : (g == 1 ? 10 : (g == 2 ? 17 : -1));
    const int c4 = g == 0 ? 5 : (g == 1 ? 11 : (g == 2 ? 18 : 20));
    if (c0 >= 0) put(row + c0, q0, first);
    put(row + c1, q1, first);
    put(row + c1 + 1, q2, first);
    if (c3 >= 0) put(row + c3, q3, first);
    put(row + c4, q4, first);
    put(row + c4 + 1, q5, first);
    const unsigned* msk = stage_masks(st + r * kStageRow);
    const unsigned m0 = msk[0], m1 = msk[1], m2 = msk[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int c = 2 * g + k;
        const int cnt = __popc(act & ((c & 1) ? m0 : ~m0) & ((c & 2) ? m1 : ~m1) & ((c & 4) ? m2 : ~m2));
        put(row + kColCount + c, (double)cnt, first);
    }
}

// Narrow-pulse signals of a batch (main.cu:374-378).  Lanes beyond the b-values
// of a group of 32 take a share of the walkers (signal_lanes).
__device__ __noinline__ void add_signals(const double* st, const double* __restrict__ qtab,
                                         const double* __restrict__ bvec, int nb, double* row, int nvals, int nrec,
                                         int nw, bool first, int lane) {
    __syncwarp();
    auto group = [&](int jb, bool in, int first_w, int step, auto&& total) {
        const double bx = in ? __ldg(bvec + jb * 3) : 0.0, by = in ? __ldg(bvec + jb * 3 + 1) : 0.0,
                     bz = in ? __ldg(bvec + jb * 3 + 2) : 0.0;
        for (int r = 0; r < nrec; ++r) {
            const double q = in ? __ldg(qtab + (size_t)r * nb + jb) : 0.0;
            const double* v = st + r * kStageRow;
            double s = 0.0;
#pragma unroll 2
            for (int w = first_w; w < nw; w += step)
                s += v[96 + w] * cos(q * (v[w] * bx + v[32 + w] * by + v[64 + w] * bz));
            total(row + (size_t)r * nvals + jb, s);
        }
    };
    int base = 0;
    // a lane to a b-value, while more than half the lanes have one
    for (; nb - base > 16 || (base < nb && nw == 1); base += 32) {
        const int jb = base + lane;
        if (jb < nb) group(jb, true, 0, 1, [&](double* p, double s) { put(p, s, first); });
    }
    if (base < nb) {
        const SignalLanes l = signal_lanes(lane, nb - base, nw);
        const int jb = base + l.item;
        const bool in = jb < nb;
        group(jb, in, l.share, l.shares, [&](double* p, double s) {
            s = share_sum(s, l);
            if (in && l.share == 0) put(p, s, first);
        });
    }
}

// Final T2-weighted PGSE signal of the tile (main_PGSE.cu:348-357), a lane (or
// several) to a gradient: phase_j = |g| (g_hat . V) dt with the walkers' window
// sums V in vscr ([pair * 3 + axis][thread], thread t0 + w).
__device__ __noinline__ void add_pgse(const WalkArgs& a, int nthr, int t0, double s0, int nw, double* sig, bool first,
                                      int lane) {
    __syncwarp();
    for (int base = 0; base < a.ngrad; base += 32) {
        const SignalLanes l = signal_lanes(lane, min(32, a.ngrad - base), nw);
        const int j = min(base + l.item, a.ngrad - 1);
        const double* g = a.grad + 6 * j;
        const double* vv = a.vscr + (size_t)(a.gpair[j] * 3) * nthr + t0;
        const double g2 = g[2], g3 = g[3], g4 = g[4], g5 = g[5];
        double s = 0.0;
        for (int k = 0; k < nw; k += l.shares) {
            const int w = min(k + l.share, nw - 1);
            const double phase = g2 * (vv[w] * g3 + vv[nthr + w] * g4 + vv[2 * (size_t)nthr + w] * g5) * a.dt;
            const double sw = __shfl_sync(0xffffffffu, s0, w);
            s += (k + l.share < nw ? sw : 0.0) * cos(phase);
        }
        s = share_sum(s, l);
        if (base + l.item < a.ngrad && l.share == 0) put(sig + j, s, first);
    }
    // the next tile's walkers clear these sums: every lane has read them by then
    // (a shuffle orders no memory)
    __syncwarp();
}

// What bounds it: FP64 issue (64 lanes per clock and SM) and, below a few warps
// per scheduler, the latency of a step's FP64 chain.  So a step forms no
// quotient it does not need: per axis the face ahead f (an integer kept as a
// double), 1 / v once a step, and the time to a face as (f - x) / v only
// approximately (2^-52) to choose the axis; the exact quotient is formed for the
// axis that is hit, from the same reciprocal.  Where two faces, or a face and
// the step's end, lie within 2^-46 of each other, the segment is decided by the
// exact quotients of all three.  Every value that reaches the walker is the
// reference's expression, rounded as written.
//
// MINB, resident blocks per SM: 4 (narrow pulses 108 registers, PGSE 119), 5 (96, 32
// and 68 bytes spilled) or 6 (80, 156 and 176 bytes); the launch takes the one whose
// rounds of tiles end first (compat_form in rms_api.cpp).
template <int NCMAX, bool TRACE, bool PGSE, int MINB>
__global__ void __launch_bounds__(kBlock, MINB) walk_compat_kernel(const __grid_constant__ WalkArgs a) {
    __shared__ double s_step[NCMAX], s_rstep[NCMAX], s_t2[NCMAX], s_rt2[NCMAX], s_pij[NCMAX * NCMAX];
    __shared__ double s_tc[NCMAX][kBlock];               // residence of the walker per compartment
    __shared__ double s_stage[kBlock / 32][kRec * kStageRow];
    for (int i = threadIdx.x; i < NCMAX * NCMAX; i += blockDim.x) {
        s_pij[i] = (i < a.nc * a.nc) ? a.pij[i] : 0.0;
        if (i < NCMAX) {
            s_step[i] = (i < a.nc) ? a.step[i] : 0.0;
            s_t2[i] = (i < a.nc) ? a.t2[i] : 1.0;
            s_rstep[i] = __drcp_rn(s_step[i]);
            // (0: weight() divides -- an infinite T2, or one so short or long that 1 / T2
            // or a quotient leaves the range in which div_by is the division)
            s_rt2[i] = s_t2[i] > 0x1p-900 && s_t2[i] < 0x1p+900 ? __drcp_rn(s_t2[i]) : 0.0;
        }
    }
    __syncthreads();

    const int lane = threadIdx.x & 31;
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x;
    const int nthr = gridDim.x * blockDim.x;
    const int warp_global = gtid >> 5;
    const int nwarps = nthr >> 5;
    const bool mirror = (a.boundary == 0);
    double* slot = a.slots + (size_t)warp_global * a.timepoints * a.nvals;
    double* st = s_stage[threadIdx.x >> 5];
    const double n0 = (double)a.n1, n1 = (double)a.n2, n2 = (double)a.n3;
    const int l0 = a.n2 * a.n3, l1 = a.n3;               // strides of the label lattice
    // how much nearer a time must be to be surely so.  With a step of a voxel or
    // more (compartment 0 alone may have one, entered by a permeation table) a
    // face beyond a whole step is 2 away, whatever its time: nothing is sure then
    // (as a factor: 1000 walkers x 2000 steps 4.40 ms; with a test of its own 4.55)
    const double near_by = s_step[0] >= 1.0 ? __longlong_as_double(0x7ff0000000000000ll) : 1.0 + 0x1p-46;

    for (int64_t tile = warp_global; tile < a.ntiles; tile += nwarps) {
        const bool first = tile == warp_global;
        const int64_t w = a.walker_begin + tile * a.tile_w + lane;
        bool active = w < a.walker_end && lane < a.tile_w;
        DoubleStream rng;
        rng.init(a.seed, (uint64_t)w);

        // initial position: rejection sampling in the box (main.cu:117-132)
        double xi0 = 0.0, xi1 = 0.0, xi2 = 0.0;
        int lin = 0;
        double g0 = 0.0, g1 = 0.0, g2 = 0.0;             // the voxel
        int ai = 0;
        if (active) {
            long long tries = 0;
            for (;;) {
                xi0 = rng.next() * n0;
                xi1 = rng.next() * n1;
                xi2 = rng.next() * n2;
                const int i0 = (int)floor(xi0), i1 = (int)floor(xi1), i2 = (int)floor(xi2);
                lin = (int)lin3(i0, i1, i2, a.n2, a.n3);
                ai = (int)__ldg(a.labels + lin);
                g0 = (double)i0; g1 = (double)i1; g2 = (double)i2;
                if (ai != 0) break;
                if (++tries >= kInitTryCap) { atomicOr(a.err, kErrInitCap); active = false; break; }
            }
        }
        double xt0 = xi0, xt1 = xi1, xt2 = xi2;
        if (TRACE && active && w < a.trace_n) a.tr_init[w] = lin;

        double tcur = 0.0;                               // residence in compartment ai (the others': s_tc)
#pragma unroll
        for (int k = 0; k < NCMAX; ++k) s_tc[k][threadIdx.x] = 0.0;
        // the T2 weight (main.cu:335-337)
        auto weight = [&]() {
            double s = 0.0;
            s_tc[ai][threadIdx.x] = tcur;
#pragma unroll
            for (int c = 0; c < NCMAX; ++c)
                if (c < a.nc) {
                    const double tc = s_tc[c][threadIdx.x], y = s_rt2[c];
                    s = s + (y > 0.0 ? div_by(tc, s_t2[c], y) : tc / s_t2[c]);
                }
            return active ? exp(-1.0 * s) : 0.0;
        };

        // PGSE: running displacement sum and the lobe-edge events
        double p0 = 0.0, p1 = 0.0, p2 = 0.0;
        int evi = 0;
        int next_ev = (PGSE && a.nevents > 0) ? a.ev_step[0] : -1;
        if (PGSE)
            for (int k = 0; k < a.npairs * 3; ++k) a.vscr[(size_t)k * nthr + gtid] = 0.0;

        int next_rec = 0, rec = 0;   // the next recorded step and its record
        for (int i = 0; i < a.tn; ++i) {                            // main.cu:134
            if (active) {
                double fstep = 1.0;
                unsigned wall0 = 0u, wall1 = 0u;
                uint32_t ev = 0u;
                int nev = 0;
                // direction (main.cu:140-151)
                double vr, vr2;
                rng.next2(vr, vr2);
                const double cos_t = 1.0 - 2.0 * vr;
                const double sin_t = 2.0 * sqrt(vr * (1.0 - vr));
                double sn, cs;
                sincos(2.0 * kRefPi * vr2, &sn, &cs);
                double v0 = sin_t * cs;
                double v1 = sin_t * sn;
                double v2 = cos_t;
                double y0 = __drcp_rn(v0), y1 = __drcp_rn(v1), y2 = __drcp_rn(v2);
                // the face ahead on each axis (no component is zero: both uniforms are odd multiples of 2^-53)
                unsigned ups = (v0 > 0.0 ? 1u : 0u) | (v1 > 0.0 ? 2u : 0u) | (v2 > 0.0 ? 4u : 0u);
                double f0 = (ups & 1u) ? g0 + 1.0 : g0, f1 = (ups & 2u) ? g1 + 1.0 : g1, f2 = (ups & 4u) ? g2 + 1.0 : g2;

                for (int j = 0; (j < a.nite) && (fstep > 0); ++j) {  // main.cu:153
                    const double d0 = f0 - xt0, d1 = f1 - xt1, d2 = f2 - xt2;
                    const double u0 = d0 * y0, u1 = d1 * y1, u2 = d2 * y2;
                    const bool b1 = u1 < u0;
                    const double lo = b1 ? u1 : u0;
                    const bool b2 = u2 < lo;
                    const double u = b2 ? u2 : lo;
                    double tmin = u;
                    int hit = b2 ? 2 : (b1 ? 1 : 0);
                    const double st_ = s_step[ai];                  // main.cu:231-244
                    const double reach = fstep * st_;
                    bool ends = reach * near_by < tmin;
                    if (!ends) {
                        // (a face already passed by rounding is reached at once)
                        const double th = (tmin > 0.0 ? tmin : 0.0) * near_by;   // (0 x inf: no comparison holds)
                        const int near = (int)(u0 <= th) + (int)(u1 <= th) + (int)(u2 <= th);
                        if (reach > th && near == 1) {
                            const double d = hit == 0 ? d0 : (hit == 1 ? d1 : d2);
                            const double v = hit == 0 ? v0 : (hit == 1 ? v1 : v2);
                            const double y = hit == 0 ? y0 : (hit == 1 ? y1 : y2);
                            const double q = div_by(d, v, y, u);
                            tmin = (0.0 < q) ? q : 0.0;
                        } else {
                            // too close to call: the exact quotients, lowest axis on ties
                            tmin = 2.0;
                            hit = -1;
                            const double t0 = face_time(d0, v0), t1 = face_time(d1, v1), t2 = face_time(d2, v2);
                            if (t0 < tmin) { tmin = t0; hit = 0; }
                            if (t1 < tmin) { tmin = t1; hit = 1; }
                            if (t2 < tmin) { tmin = t2; hit = 2; }
                            ends = !(reach >= tmin);
                        }
                    }
                    if (ends) {
                        xt0 = xt0 + reach * v0;
                        xt1 = xt1 + reach * v1;
                        xt2 = xt2 + reach * v2;
                        tcur = tcur + fstep;
                        fstep = 0.0;
                        break;
                    }
                    const double q = div_by(tmin, st_, s_rstep[ai]);
                    fstep = fstep - q;
                    xt0 = xt0 + tmin * v0;
                    xt1 = xt1 + tmin * v1;
                    xt2 = xt2 + tmin * v2;
                    tcur = tcur + q;
                    if (hit < 0) { atomicOr(a.err, kErrStep); break; }

                    // neighbour voxel; lattice wall (main.cu:246-265)
                    const bool up = (ups >> hit) & 1u;
                    const double fh = hit == 0 ? f0 : (hit == 1 ? f1 : f2);
                    const double nh = hit == 0 ? n0 : (hit == 1 ? n1 : n2);
                    const int lh = hit == 0 ? l0 : (hit == 1 ? l1 : 1);
                    const bool wall = up ? fh >= nh : fh <= 0.0;
                    bool cross = false;
                    int aj = ai, lj = lin;
                    if (wall && mirror) {
                        if (up) wall1 |= 1u << hit; else wall0 |= 1u << hit;
                        if (TRACE) ev |= ((1u << 2) | (uint32_t)hit) << (4 * nev++);
                    } else {
                        // membrane (main.cu:272-289); a periodic wall's neighbour is on the far side
                        if (!wall) lj += up ? lh : -lh;
                        else lj += up ? -((int)nh - 1) * lh : ((int)nh - 1) * lh;
                        aj = (int)__ldg(a.labels + (unsigned)lj);
                        const double P = s_pij[ai * a.nc + aj];
                        if (P > 0.999999) {
                            cross = true;
                        } else if (P < 0.000001) {
                            cross = false;
                        } else {
                            cross = rng.next() < P;
                        }
                        if (TRACE)
                            ev |= (((cross ? (wall ? 1u : 3u) : 2u) << 2) | (uint32_t)hit) << (4 * nev++);
                    }
                    // the face ahead next: a voxel further on, or the one behind after a reflection
                    double df = up ? 1.0 : -1.0;
                    if (cross) {
                        if (aj != ai) {
                            s_tc[ai][threadIdx.x] = tcur;
                            tcur = s_tc[aj][threadIdx.x];
                            ai = aj;
                        }
                        lin = lj;
                        if (wall) {
                            const double shift = up ? -nh : nh;
                            df = df + shift;
                            if (hit == 0) { xt0 = xt0 + shift; xi0 = xi0 + shift; }
                            else if (hit == 1) { xt1 = xt1 + shift; xi1 = xi1 + shift; }
                            else { xt2 = xt2 + shift; xi2 = xi2 + shift; }
                        }
                    } else {
                        df = -df;
                        ups ^= 1u << hit;
                        if (hit == 0) { v0 = -v0; y0 = -y0; }
                        else if (hit == 1) { v1 = -v1; y1 = -y1; }
                        else { v2 = -v2; y2 = -y2; }
                    }
                    if (hit == 0) f0 = f0 + df; else if (hit == 1) f1 = f1 + df; else f2 = f2 + df;
                }
                g0 = (ups & 1u) ? f0 - 1.0 : f0;
                g1 = (ups & 2u) ? f1 - 1.0 : f1;
                g2 = (ups & 4u) ? f2 - 1.0 : f2;

                // mirror the origin for each wall hit this step (main.cu:302-310)
                if (wall0 | wall1) {
                    if (wall0 & 1u) xi0 = -xi0;
                    if (wall1 & 1u) xi0 = 2.0 * n0 - xi0;
                    if (wall0 & 2u) xi1 = -xi1;
                    if (wall1 & 2u) xi1 = 2.0 * n1 - xi1;
                    if (wall0 & 4u) xi2 = -xi2;
                    if (wall1 & 4u) xi2 = 2.0 * n2 - xi2;
                }
                if (TRACE && w < a.trace_n) {
                    if (fstep > 0) ev |= 1u << 31;
                    ev |= (uint32_t)nev << 28;
                    a.tr_vox[(size_t)w * a.tn + i] = lin;
                    a.tr_ev[(size_t)w * a.tn + i] = ev;
                    double* tp = a.tr_pos + ((size_t)w * a.tn + i) * 3;
                    tp[0] = xt0; tp[1] = xt1; tp[2] = xt2;
                }
            }

            if (PGSE) {
                // displacement of this step's position (main_PGSE.cu:336-338)
                p0 = p0 + (xt0 - xi0) * a.res;
                p1 = p1 + (xt1 - xi1) * a.res;
                p2 = p2 + (xt2 - xi2) * a.res;
                if (i + 1 == next_ev) {
                    do {
                        const double cf = a.ev_coef[evi];
                        double* vv = a.vscr + (size_t)(a.ev_pair[evi] * 3) * nthr + gtid;
                        vv[0] = vv[0] + cf * p0;
                        vv[nthr] = vv[nthr] + cf * p1;
                        vv[2 * (size_t)nthr] = vv[2 * (size_t)nthr] + cf * p2;
                        ++evi;
                    } while (evi < a.nevents && a.ev_step[evi] == i + 1);
                    next_ev = (evi < a.nevents) ? a.ev_step[evi] : -1;
                }
            }

            // record every tstep steps (main.cu:333-379; i % tstep == 0 as a countdown)
            if (i == next_rec) {
                const int r = rec & (kRec - 1), rec0 = rec - r;   // slot in the batch, the batch's first record
                ++rec;
                next_rec = rec < a.timepoints ? next_rec + a.tstep : -1;
                double* mine = st + r * kStageRow + lane;
                mine[0] = (xt0 - xi0) * a.res;
                mine[32] = (xt1 - xi1) * a.res;
                mine[64] = (xt2 - xi2) * a.res;
                mine[96] = weight();
                const unsigned b0 = __ballot_sync(0xffffffffu, ai & 1), b1 = __ballot_sync(0xffffffffu, ai & 2),
                               b2 = __ballot_sync(0xffffffffu, ai & 4);
                if (lane < 3) stage_masks(st + r * kStageRow)[lane] = lane == 0 ? b0 : (lane == 1 ? b1 : b2);
                if (r == kRec - 1 || rec == a.timepoints) {
                    const unsigned act = __ballot_sync(0xffffffffu, active);
                    double* row = slot + (size_t)rec0 * a.nvals;
                    add_moments(st, row, a.nvals, rec - rec0, act, a.tile_w, first, lane);
                    if (!PGSE && a.nbvec > 0)
                        add_signals(st, a.qtab + (size_t)rec0 * a.nbvec, a.bvec, a.nbvec, row + kRowHead, a.nvals,
                                    rec - rec0, a.tile_w, first, lane);
                    __syncwarp();
                }
            }
        }
        if (PGSE)
            add_pgse(a, nthr, gtid - lane, weight(), a.tile_w, a.sig_slots + (size_t)warp_global * a.ngrad_pad, first,
                     lane);
    }
}

template <class F>
auto by_form(int nc, bool trace, bool pgse, int minb, F&& f) {
    auto blocks = [&]<int NC, bool PG>() {
        if (trace) return f.template operator()<NC, true, PG, 4>();
        if (minb == 6) return f.template operator()<NC, false, PG, 6>();
        if (minb == 5) return f.template operator()<NC, false, PG, 5>();
        return f.template operator()<NC, false, PG, 4>();
    };
    if (nc <= 4) return pgse ? blocks.template operator()<4, true>() : blocks.template operator()<4, false>();
    return pgse ? blocks.template operator()<8, true>() : blocks.template operator()<8, false>();
}

}  // namespace

int launch_walk_compat(const WalkArgs& a, int grid, int block, int minb, bool trace, void* stream) {
    if (block != kBlock) return (int)cudaErrorInvalidValue;
    return by_form(a.nc, trace, a.mode == 1, minb, [&]<int NC, bool TR, bool PG, int MB>() {
        walk_compat_kernel<NC, TR, PG, MB><<<grid, kBlock, 0, (cudaStream_t)stream>>>(a);
        return (int)cudaGetLastError();
    });
}

int walk_compat_blocks_per_sm(int nc, bool trace, bool pgse, int minb) {
    return by_form(nc, trace, pgse, minb, [&]<int NC, bool TR, bool PG, int MB>() {
        int n = 0;
        const cudaError_t e =
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, walk_compat_kernel<NC, TR, PG, MB>, kBlock, 0);
        return e == cudaSuccess ? n : -1;
    });
}

}  // namespace rms
