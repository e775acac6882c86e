// hhs_kick64.cuh -- FP64 pair sums of a block of sinks, in the reference's order.
//
// The FP64 kick is bit-exact: a sink's pair terms are added one after another in source
// order (src/kick.cuh:59-155), so a sink's sum is a chain of n dependent additions. The
// terms themselves (a square root and a reciprocal each, about 50 FP64 instructions) do
// not depend on one another. One thread per sink computes both, which leaves a node of
// a few thousand sinks on a dozen CTAs and each thread waiting for its own square roots.
// Here a CTA takes T sinks (8 to 32) and evaluates T x C terms at a time with all its
// threads (lanes along the sources, each source loaded once for its sinks), into shared
// memory; then 3 T threads add the C terms of one (sink, component) each, in order.
// Measured: the kicks of an N=16384 step 132.9 -> 23.8 ms, kick_slow of 1367 particles 225 ->
// 21 us. What bounds it now: of a stage of 8 x 256 terms, 2900 clocks evaluate (8 pairs a
// thread, the latency of their square roots and reciprocals) and 2500 add (256 dependent
// additions).
#pragma once
#include "hhs_pairmath.cuh"

namespace hhs {

constexpr int kK64Threads = 256;
constexpr int kK64MaxT = 32;

// PAIRS terms per stage: T sinks x C = PAIRS / T sources (C <= 256). Rows of a component
// are C + 1 doubles apart and components 8 (mod 16) doubles, so that the adding threads
// of a half warp read 16 different banks.
template <int PAIRS>
struct Kick64Smem {
    static constexpr int kPitch = PAIRS + 2 * kK64MaxT + 8 - (PAIRS + 2 * kK64MaxT) % 16;
    double t[3][kPitch];
    double sx[kK64MaxT], sy[kK64MaxT], sz[kK64MaxT];
};

// Sum over the sources 0 .. cnt-1 of their pair terms on the sinks in k.sx/sy/sz (nsink
// of them, at most T = PAIRS >> cs; written and synchronised by the caller). index(j) is the
// array position of source j, load(position, x, y, z, m) its values: the position of the
// stage after next and the values of the next are on their way while a stage is added up.
// On return thread t < 3 T holds component t >> log2(T) of sink t & (T - 1). Every thread of
// the CTA (256) calls it; ends with a CTA barrier.
template <int PAIRS, class Index, class Load>
__device__ __forceinline__ double kick64_sums(Kick64Smem<PAIRS>& k, int cs, int nsink, int cnt,
                                              double eps2, Index&& index, Load&& load) {
    const int tid = threadIdx.x;
    const int C = 1 << cs, T = PAIRS >> cs, pitch = C + 1;
    const int col = tid & (C - 1), row0 = tid >> cs, rstep = kK64Threads >> cs;
    const bool adds = tid < 3 * T;
    const double* mine = &k.t[tid / T < 3 ? tid / T : 0][(tid & (T - 1)) * pitch];
    double acc = 0.0;
    double x = 0.0, y = 0.0, z = 0.0, m = 0.0;
    if (col < cnt) load(index(col), x, y, z, m);
    int next = C + col < cnt ? index(C + col) : 0;
    for (int j0 = 0; j0 < cnt; j0 += C) {
        if (j0 + col < cnt) {
            for (int s = row0; s < nsink; s += rstep) {
                const double dx = f64_sub(x, k.sx[s]), dy = f64_sub(y, k.sy[s]),
                             dz = f64_sub(z, k.sz[s]);
                const double d2 = f64_add(
                    f64_add(f64_add(f64_mul(dx, dx), f64_mul(dy, dy)), f64_mul(dz, dz)), eps2);
                // a particle and itself: no term (adding +0 leaves a sum as it is)
                const double w = f64_mul(m, __drcp_rn(f64_mul(d2, f64_sqrt(d2))));
                const bool self = d2 == 0.0;
                double* o = &k.t[0][s * pitch + col];
                o[0] = self ? 0.0 : f64_mul(dx, w);
                o[Kick64Smem<PAIRS>::kPitch] = self ? 0.0 : f64_mul(dy, w);
                o[2 * Kick64Smem<PAIRS>::kPitch] = self ? 0.0 : f64_mul(dz, w);
            }
        }
        if (j0 + C + col < cnt) load(next, x, y, z, m);
        if (j0 + 2 * C + col < cnt) next = index(j0 + 2 * C + col);
        __syncthreads();
        if (adds) {
            const int e = min(C, cnt - j0);
            int j = 0;
            for (; j + 8 <= e; j += 8) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = mine[j + u];
#pragma unroll
                for (int u = 0; u < 8; u++) acc = f64_add(acc, v[u]);
            }
            for (; j < e; j++) acc = f64_add(acc, mine[j]);
        }
        __syncthreads();
    }
    return acc;
}

}  // namespace hhs
