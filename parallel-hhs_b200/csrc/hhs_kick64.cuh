// hhs_kick64.cuh -- FP64 pair sums of a block of sinks, in the reference's order.
//
// The FP64 kick is bit-exact: a sink's pair terms are added one after another in source
// order (src/kick.cuh:59-155), so a sink's sum is a chain of n dependent additions. The
// terms themselves (a square root and a reciprocal each, about 50 FP64 instructions) do
// not depend on one another. One thread per sink computes both, which leaves a node of
// a few thousand sinks on a dozen CTAs and each thread waiting for its own square roots.
// Here a CTA takes 8 sinks. Seven warps evaluate the terms of 8 sinks x 224 sources at a time
// (a source a thread, loaded once for its sinks) into one of two shared buffers, while the
// eighth adds the 224 terms of the previous stage, one (sink, component) a lane, in order.
// Measured: the kicks of an N=16384 step 132.9 ms with one thread a sink, 24.0 with evaluation
// and addition in turn (by all warps, 8 x 256 terms), 17.4 overlapped; kick_slow of 1367
// particles 225, 24.5 and 22.3 us. What bounds it: the evaluation's latency (a stage takes
// 3100 clocks, 8 terms a thread; its additions 2300).
#pragma once
#include "hhs_pairmath.cuh"

namespace hhs {

constexpr int kK64Threads = 256;
constexpr int kK64Sinks = 8;
constexpr int kK64Sources = 224;        // sources of a stage: one per evaluating thread
constexpr int kK64Row = kK64Sources + 1;

// Rows are an odd number of doubles apart and components 8 (mod 16), so that the adding lanes
// of a half warp read 16 different banks.
struct Kick64Smem {
    double t[2][3][kK64Sinks * kK64Row];
    double sx[kK64Sinks], sy[kK64Sinks], sz[kK64Sinks];
};
static_assert(kK64Sinks * kK64Row % 16 == 8, "components fall on the other half of the banks");

// The (component, sink) whose sum kick64_sums returns in the calling thread; component -1: none.
__device__ __forceinline__ int kick64_component() {
    const int l = (int)threadIdx.x - kK64Sources;
    return l >= 0 && l < 3 * kK64Sinks ? l / kK64Sinks : -1;
}
__device__ __forceinline__ int kick64_sink() { return (int)threadIdx.x & (kK64Sinks - 1); }

// Sum over the sources 0 .. cnt-1 of their pair terms on the nsink <= 8 sinks in k.sx/sy/sz
// (written and synchronised by the caller). index(j) is the array position of source j,
// load(position, x, y, z, m) its values: the position of the stage after next and the values
// of the next are on their way while a stage is evaluated. Every thread of the CTA (256) calls
// it; ends with a CTA barrier.
template <class Index, class Load>
__device__ __forceinline__ double kick64_sums(Kick64Smem& k, int nsink, int cnt, double eps2,
                                              Index&& index, Load&& load) {
    constexpr int C = kK64Sources;
    const int col = threadIdx.x, lane = col & 31;
    const bool eval = col < C;
    const int ad = lane < 3 * kK64Sinks ? lane : 0;
    double acc = 0.0;
    double x = 0.0, y = 0.0, z = 0.0, m = 0.0, xn = 0.0, yn = 0.0, zn = 0.0, mn = 0.0;
    int next = 0;
    if (eval) {
        if (col < cnt) load(index(col), xn, yn, zn, mn);
        if (C + col < cnt) next = index(C + col);
    }
    for (int j0 = 0, st = 0; j0 < cnt + C; j0 += C, st++) {
        if (eval) {
            if (j0 < cnt) {
                x = xn; y = yn; z = zn; m = mn;
                if (j0 + C + col < cnt) load(next, xn, yn, zn, mn);
                if (j0 + 2 * C + col < cnt) next = index(j0 + 2 * C + col);
                // (lanes past the last source repeat the one they hold; their terms are not
                // added)
                double* o = &k.t[st & 1][0][col];
                for (int s = 0; s < nsink; s++, o += kK64Row) {
                    __syncwarp();  // the slow paths of the root and the reciprocal part the lanes
                    const double dx = f64_sub(x, k.sx[s]), dy = f64_sub(y, k.sy[s]),
                                 dz = f64_sub(z, k.sz[s]);
                    const double d2 = f64_add(
                        f64_add(f64_add(f64_mul(dx, dx), f64_mul(dy, dy)), f64_mul(dz, dz)), eps2);
                    // a particle and itself: no term (adding +0 leaves a sum as it is)
                    const double w = f64_mul(m, __drcp_rn(f64_mul(d2, f64_sqrt(d2))));
                    const bool self = d2 == 0.0;
                    o[0] = self ? 0.0 : f64_mul(dx, w);
                    o[kK64Sinks * kK64Row] = self ? 0.0 : f64_mul(dy, w);
                    o[2 * kK64Sinks * kK64Row] = self ? 0.0 : f64_mul(dz, w);
                }
            }
        } else if (st > 0) {
            const double* v = &k.t[(st - 1) & 1][ad / kK64Sinks][(ad % kK64Sinks) * kK64Row];
            const int e = min(C, cnt - (j0 - C));
            int j = 0;
            for (; j + 8 <= e; j += 8) {
                double q[8];
#pragma unroll
                for (int u = 0; u < 8; u++) q[u] = v[j + u];
#pragma unroll
                for (int u = 0; u < 8; u++) acc = f64_add(acc, q[u]);
            }
            for (; j < e; j++) acc = f64_add(acc, v[j]);
        }
        __syncthreads();
    }
    return acc;
}

}  // namespace hhs
