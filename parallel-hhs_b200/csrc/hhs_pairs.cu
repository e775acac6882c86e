// hhs_pairs.cu -- one-thread-per-sink pair kernels (timestep, kick), drift, gathers.
//
// These are the plain kernels of the library: the reference's one-thread-per-sink
// structure with source tiles staged through shared memory (src/timestep.cuh:65-99,
// src/kick.cuh:59-155), but on SoA FP64 arrays addressed through index lists, with
// the tail tile loaded correctly (the reference returns before the cooperative load,
// src/timestep.cuh:70) and every launch sized from device-resident counts.
#include <algorithm>
#include <cmath>

#include "hhs_common.cuh"
#include "hhs_kernels.h"
#include "hhs_kick64.cuh"
#include "hhs_pairmath.cuh"
#include "hhs_tsrows.cuh"

using namespace hhs;

namespace {

constexpr int kKickBlock = 128;
constexpr int kSms = 148;  // of a B200

__device__ __forceinline__ int list_at(const int32_t* list, int i) { return ts_list_at(list, i); }

// The stores of a sink-partitioned launch into the peer replicas, then a system-scope
// fence so that the barrier which follows the launch orders them for every peer.
__device__ __forceinline__ void peer_store_ts(const PeerOut& po, int g, double t) {
    if (po.n_peer == 0) return;
    for (int r = 0; r < po.n_peer; r++) po.ts[r][g] = t;
    __threadfence_system();
}
__device__ __forceinline__ void peer_store_v(const PeerOut& po, int g, double vx, double vy,
                                             double vz) {
    if (po.n_peer == 0) return;
    for (int r = 0; r < po.n_peer; r++) {
        po.vx[r][g] = vx; po.vy[r][g] = vy; po.vz[r][g] = vz;
    }
    __threadfence_system();
}

// ---------------------------------------------------------------- timesteps
template <int PREC>
__global__ void __launch_bounds__(kTsThreads, 4)
    k_timesteps(SoA P, const int32_t* __restrict__ list, int n, int T, TsArgs A, PeerOut po) {
    __shared__ TsRows sm;
    const int hi = po.hi < 0 ? n : po.hi;
    const int i0 = po.lo + blockIdx.x * T, nrow = min(T, hi - i0);
    ts_rows<PREC>(P, list, n, i0, nrow, A, sm);
    if ((int)threadIdx.x < nrow) {
        const int g = list_at(list, i0 + threadIdx.x);
        const double t = ts_of_key<PREC>(sm.best[threadIdx.x]);
        P.ts[g] = t;
        peer_store_ts(po, g, t);
    }
}

// ---------------------------------------------------------------- kick, FP64
// Sink s of a split level: s < nf -> fast sink F[s]; else slow sink L[s - nf].
// Sources: slow tiles (every sink), then fast tiles (slow sinks only). Slow sinks
// apply v += aLL*dt then v += aLF*dt (kick_slow then kick_sf(fast->slow),
// src/hold.cuh:138,142); fast sinks apply v += aFL*dt (kick_sf(slow->fast), :143).
__global__ void __launch_bounds__(kKickBlock)
    k_kick_level_fp64(SoA P, const int32_t* __restrict__ F, const int32_t* __restrict__ L,
                      const hhs_partition* __restrict__ counts, double dt, double eps2,
                      PeerOut po) {
    __shared__ double sx[kKickBlock], sy[kKickBlock], sz[kKickBlock], sm[kKickBlock];
    const int nf = counts->n_fast, ns = counts->n_slow, n = nf + ns;
    if (ns == 0) return;
    const int hi = po.hi < 0 ? n : min(po.hi, n);
    if (po.lo + (int)(blockIdx.x * kKickBlock) >= hi) return;
    const int s = po.lo + blockIdx.x * kKickBlock + threadIdx.x;
    const bool active = s < hi;
    const bool slow_sink = s >= nf;
    const int g = active ? (slow_sink ? L[s - nf] : F[s]) : 0;
    const double xi = active ? P.x[g] : 0.0, yi = active ? P.y[g] : 0.0,
                 zi = active ? P.z[g] : 0.0;
    double aLx = 0, aLy = 0, aLz = 0, aFx = 0, aFy = 0, aFz = 0;
    for (int jt = 0; jt < ns; jt += kKickBlock) {
        const int j = jt + threadIdx.x;
        if (j < ns) {
            const int gj = L[j];
            sx[threadIdx.x] = P.x[gj]; sy[threadIdx.x] = P.y[gj]; sz[threadIdx.x] = P.z[gj];
            sm[threadIdx.x] = P.m[gj];
        }
        __syncthreads();
        if (active) {
            const int jn = min(kKickBlock, ns - jt);
            for (int jl = 0; jl < jn; jl++)
                kick_pair_fp64(f64_sub(sx[jl], xi), f64_sub(sy[jl], yi), f64_sub(sz[jl], zi), sm[jl],
                               aLx, aLy, aLz, eps2);
        }
        __syncthreads();
    }
    for (int jt = 0; jt < nf; jt += kKickBlock) {
        const int j = jt + threadIdx.x;
        if (j < nf) {
            const int gj = F[j];
            sx[threadIdx.x] = P.x[gj]; sy[threadIdx.x] = P.y[gj]; sz[threadIdx.x] = P.z[gj];
            sm[threadIdx.x] = P.m[gj];
        }
        __syncthreads();
        if (active && slow_sink) {
            const int jn = min(kKickBlock, nf - jt);
            for (int jl = 0; jl < jn; jl++)
                kick_pair_fp64(f64_sub(sx[jl], xi), f64_sub(sy[jl], yi), f64_sub(sz[jl], zi), sm[jl],
                               aFx, aFy, aFz, eps2);
        }
        __syncthreads();
    }
    if (!active) return;
    double vx = P.vx[g], vy = P.vy[g], vz = P.vz[g];
    vx = f64_add(vx, f64_mul(aLx, dt));
    vy = f64_add(vy, f64_mul(aLy, dt));
    vz = f64_add(vz, f64_mul(aLz, dt));
    if (slow_sink && nf > 0) {
        vx = f64_add(vx, f64_mul(aFx, dt));
        vy = f64_add(vy, f64_mul(aFy, dt));
        vz = f64_add(vz, f64_mul(aFz, dt));
    }
    P.vx[g] = vx; P.vy[g] = vy; P.vz[g] = vz;
    peer_store_v(po, g, vx, vy, vz);
}

// ---------------------------------------------------------------- kick, mixed
// Same sink/source structure. Pair terms in FP32 from double-single relative
// coordinates; per-sink sums Kahan-compensated in FP32 and applied in FP64. The slow
// and fast source sums are kept apart so the update order matches the FP64 form.
__global__ void __launch_bounds__(kKickBlock)
    k_kick_level_mixed(SoA P, const int32_t* __restrict__ F, const int32_t* __restrict__ L,
                       const hhs_partition* __restrict__ counts, double dt, float eps2,
                       PeerOut po) {
    __shared__ float4 sA[kKickBlock];  // xh, yh, zh, m
    __shared__ float4 sB[kKickBlock];  // xl, yl, zl, -
    const int nf = counts->n_fast, ns = counts->n_slow, n = nf + ns;
    if (ns == 0) return;
    const int hi = po.hi < 0 ? n : min(po.hi, n);
    if (po.lo + (int)(blockIdx.x * kKickBlock) >= hi) return;
    const int s = po.lo + blockIdx.x * kKickBlock + threadIdx.x;
    const bool active = s < hi;
    const bool slow_sink = s >= nf;
    const int g = active ? (slow_sink ? L[s - nf] : F[s]) : 0;
    DS xi{0, 0}, yi{0, 0}, zi{0, 0};
    if (active) { xi = ds_split(P.x[g]); yi = ds_split(P.y[g]); zi = ds_split(P.z[g]); }
    float acc[2][3] = {{0, 0, 0}, {0, 0, 0}}, cmp[2][3] = {{0, 0, 0}, {0, 0, 0}};
#pragma unroll 1
    for (int part = 0; part < 2; part++) {
        const int cnt = part == 0 ? ns : nf;
        const int32_t* lst = part == 0 ? L : F;
        const bool use = active && (part == 0 || slow_sink);
        for (int jt = 0; jt < cnt; jt += kKickBlock) {
            const int j = jt + threadIdx.x;
            if (j < cnt) {
                const int gj = lst[j];
                const DS a = ds_split(P.x[gj]), b = ds_split(P.y[gj]), c = ds_split(P.z[gj]);
                sA[threadIdx.x] = make_float4(a.hi, b.hi, c.hi, (float)P.m[gj]);
                sB[threadIdx.x] = make_float4(a.lo, b.lo, c.lo, 0.0f);
            }
            __syncthreads();
            if (use) {
                const int jn = min(kKickBlock, cnt - jt);
                for (int jl = 0; jl < jn; jl++) {
                    const float4 A = sA[jl], B = sB[jl];
                    const float dx = ds_diff(A.x, B.x, xi.hi, xi.lo);
                    const float dy = ds_diff(A.y, B.y, yi.hi, yi.lo);
                    const float dz = ds_diff(A.z, B.z, zi.hi, zi.lo);
                    const float d2 = fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, eps2)));
                    if (d2 == 0.0f) continue;
                    const float ri = rsqrt_nr(d2);
                    const float mr3 = A.w * ri * ri * ri;
                    kahan_add(acc[part][0], cmp[part][0], dx * mr3);
                    kahan_add(acc[part][1], cmp[part][1], dy * mr3);
                    kahan_add(acc[part][2], cmp[part][2], dz * mr3);
                }
            }
            __syncthreads();
        }
    }
    if (!active) return;
    double v[3] = {P.vx[g], P.vy[g], P.vz[g]};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        v[k] += ((double)acc[0][k] - (double)cmp[0][k]) * dt;
        if (slow_sink && nf > 0) v[k] += ((double)acc[1][k] - (double)cmp[1][k]) * dt;
    }
    P.vx[g] = v[0]; P.vy[g] = v[1]; P.vz[g] = v[2];
    peer_store_v(po, g, v[0], v[1], v[2]);
}

// ---------------------------------------------------------------- standalone kicks
// kick_slow / kick_sf of the reference API: sinks sink[0..n), sources src[0..m).
// FP64, unless the sources are few: a CTA per block of 8 sinks, terms evaluated by seven of its warps and added in source
// order by the eighth (hhs_kick64.cuh).
__global__ void __launch_bounds__(kK64Threads, 2)
    k_kick_pair_fp64(SoA K, double* __restrict__ ax_out, double* __restrict__ ay_out,
                     double* __restrict__ az_out, SoA S, int n, int m, double dtfac) {
    extern __shared__ __align__(16) unsigned char k64_smem[];
    auto& k = *reinterpret_cast<Kick64Smem*>(k64_smem);
    const int s0 = blockIdx.x * kK64Sinks, nsink = min(kK64Sinks, n - s0);
    const int tid = threadIdx.x;
    if (tid < nsink) {
        k.sx[tid] = K.x[s0 + tid]; k.sy[tid] = K.y[s0 + tid]; k.sz[tid] = K.z[s0 + tid];
    }
    __syncthreads();
    const double a = kick64_sums(k, nsink, m, 0.0, [](int j) { return j; },
                                 [&](int j, double& x, double& y, double& z, double& mj) {
                                     x = S.x[j]; y = S.y[j]; z = S.z[j]; mj = S.m[j];
                                 });
    const int c = kick64_component(), i = s0 + kick64_sink();
    if (c < 0 || i >= n) return;
    double* out = c == 0 ? ax_out : (c == 1 ? ay_out : az_out);
    double* v = c == 0 ? K.vx : (c == 1 ? K.vy : K.vz);
    if (out) out[i] = a;
    v[i] = f64_add(v[i], f64_mul(a, dtfac));
}

// Mixed: a CTA takes 32 sinks, one a lane, and each of its 8 warps an eighth of the sources, 32
// at a time, converted to double-single pairs in the warp's own shared memory (no CTA barrier
// until the end). Two sources are evaluated at once in f32x2 arithmetic, each pair term as
// before (1/d from rsqrtf with one Newton step) into Kahan-compensated FP32 sums, one for the
// even and one for the odd sources of each warp; these are added in FP64 in a fixed order.
// Measured: kick_slow of 10923 particles 926 -> 209 us (one thread a sink before: 86 CTAs, every
// thread waiting for its own chain of compensated additions). The FMA pipe bounds it: 34 packed
// operations for two pairs, 12 of them the compensated sums.
__device__ __forceinline__ void kahan_add2(float2& s, float2& c, float2 t) {
    const float2 m1 = make_float2(-1.0f, -1.0f);
    const float2 y = __ffma2_rn(c, m1, t);
    const float2 u = __fadd2_rn(s, y);
    c = __ffma2_rn(y, m1, __ffma2_rn(s, m1, u));
    s = u;
}

constexpr int kPmWarps = 8;
__global__ void __launch_bounds__(32 * kPmWarps, 3)
    k_kick_pair_mixed(SoA K, double* __restrict__ ax_out, double* __restrict__ ay_out,
                      double* __restrict__ az_out, SoA S, int n, int m, double dtfac) {
    // source pairs: (x hi), (y hi) | (z hi), (mass) | (x lo), (y lo) | (z lo)
    __shared__ float4 src[kPmWarps][16][4];
    __shared__ double sum[kPmWarps][3][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    DS xi{0, 0}, yi{0, 0}, zi{0, 0};
    if (i < n) { xi = ds_split(K.x[i]); yi = ds_split(K.y[i]); zi = ds_split(K.z[i]); }
    const float2 nxh = f2dup(-xi.hi), nyh = f2dup(-yi.hi), nzh = f2dup(-zi.hi), nxl = f2dup(-xi.lo),
                 nyl = f2dup(-yi.lo), nzl = f2dup(-zi.lo);
    float2 acc[3], cmp[3];
#pragma unroll
    for (int k = 0; k < 3; k++) acc[k] = cmp[k] = make_float2(0.0f, 0.0f);
    const int j1 = (int)((long long)m * (warp + 1) / kPmWarps);
    int j0 = (int)((long long)m * warp / kPmWarps);
    double sx = 0.0, sy = 0.0, sz = 0.0, sm = 0.0;
    // Past the slice, its last source without mass: a pair of the sink with a place of its own
    // (the origin, say) could overflow where no source does, and 0 times that is a NaN.
    auto load = [&](int j) {
        const int k = min(j, j1 - 1);
        sx = S.x[k]; sy = S.y[k]; sz = S.z[k];
        sm = j < j1 ? S.m[k] : 0.0;
    };
    if (j0 < j1) load(j0 + lane);
    for (; j0 < j1; j0 += 32) {
        __syncwarp();  // the previous sources are read
        {
            const DS a = ds_split(sx), b = ds_split(sy), c = ds_split(sz);
            float* q = reinterpret_cast<float*>(src[warp][lane >> 1]) + (lane & 1);
            q[0] = a.hi; q[2] = b.hi; q[4] = c.hi; q[6] = (float)sm;
            q[8] = a.lo; q[10] = b.lo; q[12] = c.lo;
        }
        __syncwarp();
        load(j0 + 32 + lane);  // on its way while these are evaluated
        const int np = min(32, j1 - j0) + 1 >> 1;
#pragma unroll 2
        for (int p = 0; p < np; p++) {
            const float4 Q0 = src[warp][p][0], Q1 = src[warp][p][1], Q2 = src[warp][p][2];
            const float2 zl = *reinterpret_cast<const float2*>(&src[warp][p][3]);
            const float2 dx = __fadd2_rn(__fadd2_rn(make_float2(Q0.x, Q0.y), nxh),
                                         __fadd2_rn(make_float2(Q2.x, Q2.y), nxl));
            const float2 dy = __fadd2_rn(__fadd2_rn(make_float2(Q0.z, Q0.w), nyh),
                                         __fadd2_rn(make_float2(Q2.z, Q2.w), nyl));
            const float2 dz = __fadd2_rn(__fadd2_rn(make_float2(Q1.x, Q1.y), nzh),
                                         __fadd2_rn(zl, nzl));
            float2 d2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
            // a particle and itself: no term
            const float2 w = make_float2(d2.x == 0.0f ? 0.0f : Q1.z, d2.y == 0.0f ? 0.0f : Q1.w);
            d2.x = d2.x == 0.0f ? 1.0f : d2.x;
            d2.y = d2.y == 0.0f ? 1.0f : d2.y;
            const float2 ri = rsqrt_nr2(d2);
            const float2 mr3 = __fmul2_rn(__fmul2_rn(__fmul2_rn(w, ri), ri), ri);
            kahan_add2(acc[0], cmp[0], __fmul2_rn(dx, mr3));
            kahan_add2(acc[1], cmp[1], __fmul2_rn(dy, mr3));
            kahan_add2(acc[2], cmp[2], __fmul2_rn(dz, mr3));
        }
    }
#pragma unroll
    for (int k = 0; k < 3; k++)
        sum[warp][k][lane] = ((double)acc[k].x - (double)cmp[k].x) +
                             ((double)acc[k].y - (double)cmp[k].y);
    __syncthreads();
    if (warp < 3 && i < n) {  // component `warp` of sink i
        double a = 0.0;
#pragma unroll
        for (int w = 0; w < kPmWarps; w++) a += sum[w][warp][lane];
        double* out = warp == 0 ? ax_out : (warp == 1 ? ay_out : az_out);
        double* v = warp == 0 ? K.vx : (warp == 1 ? K.vy : K.vz);
        if (out) out[i] = a;
        v[i] += a * dtfac;
    }
}

// Many sinks and few sources (few_sources): a thread per sink, which adds its terms one after another.
// FP64: the order, and so the bits, of the form above.
__global__ void __launch_bounds__(kKickBlock)
    k_kick_few_fp64(SoA K, double* __restrict__ ax_out, double* __restrict__ ay_out,
                    double* __restrict__ az_out, SoA S, int n, int m, double dtfac) {
    __shared__ double sx[kKickBlock], sy[kKickBlock], sz[kKickBlock], sm[kKickBlock];
    const int i = blockIdx.x * kKickBlock + threadIdx.x;
    const bool active = i < n;
    const double xi = active ? K.x[i] : 0.0, yi = active ? K.y[i] : 0.0,
                 zi = active ? K.z[i] : 0.0;
    double ax = 0, ay = 0, az = 0;
    for (int jt = 0; jt < m; jt += kKickBlock) {
        const int j = jt + threadIdx.x;
        if (j < m) {
            sx[threadIdx.x] = S.x[j]; sy[threadIdx.x] = S.y[j]; sz[threadIdx.x] = S.z[j];
            sm[threadIdx.x] = S.m[j];
        }
        __syncthreads();
        if (active) {
            const int jn = min(kKickBlock, m - jt);
            for (int jl = 0; jl < jn; jl++)
                kick_pair_fp64(f64_sub(sx[jl], xi), f64_sub(sy[jl], yi), f64_sub(sz[jl], zi), sm[jl],
                               ax, ay, az);
        }
        __syncthreads();
    }
    if (!active) return;
    if (ax_out) { ax_out[i] = ax; ay_out[i] = ay; az_out[i] = az; }
    K.vx[i] = f64_add(K.vx[i], f64_mul(ax, dtfac));
    K.vy[i] = f64_add(K.vy[i], f64_mul(ay, dtfac));
    K.vz[i] = f64_add(K.vz[i], f64_mul(az, dtfac));
}

__global__ void __launch_bounds__(kKickBlock)
    k_kick_few_mixed(SoA K, double* __restrict__ ax_out, double* __restrict__ ay_out,
                     double* __restrict__ az_out, SoA S, int n, int m, double dtfac) {
    __shared__ float4 sA[kKickBlock], sB[kKickBlock];
    const int i = blockIdx.x * kKickBlock + threadIdx.x;
    const bool active = i < n;
    DS xi{0, 0}, yi{0, 0}, zi{0, 0};
    if (active) { xi = ds_split(K.x[i]); yi = ds_split(K.y[i]); zi = ds_split(K.z[i]); }
    float acc[3] = {0, 0, 0}, cmp[3] = {0, 0, 0};
    for (int jt = 0; jt < m; jt += kKickBlock) {
        const int j = jt + threadIdx.x;
        if (j < m) {
            const DS a = ds_split(S.x[j]), b = ds_split(S.y[j]), c = ds_split(S.z[j]);
            sA[threadIdx.x] = make_float4(a.hi, b.hi, c.hi, (float)S.m[j]);
            sB[threadIdx.x] = make_float4(a.lo, b.lo, c.lo, 0.0f);
        }
        __syncthreads();
        if (active) {
            const int jn = min(kKickBlock, m - jt);
            for (int jl = 0; jl < jn; jl++) {
                const float4 A = sA[jl], B = sB[jl];
                const float dx = ds_diff(A.x, B.x, xi.hi, xi.lo);
                const float dy = ds_diff(A.y, B.y, yi.hi, yi.lo);
                const float dz = ds_diff(A.z, B.z, zi.hi, zi.lo);
                const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                if (d2 == 0.0f) continue;
                const float ri = rsqrt_nr(d2);
                const float mr3 = A.w * ri * ri * ri;
                kahan_add(acc[0], cmp[0], dx * mr3);
                kahan_add(acc[1], cmp[1], dy * mr3);
                kahan_add(acc[2], cmp[2], dz * mr3);
            }
        }
        __syncthreads();
    }
    if (!active) return;
    const double a0 = (double)acc[0] - cmp[0], a1 = (double)acc[1] - cmp[1],
                 a2 = (double)acc[2] - cmp[2];
    if (ax_out) { ax_out[i] = a0; ay_out[i] = a1; az_out[i] = a2; }
    K.vx[i] += a0 * dtfac;
    K.vy[i] += a1 * dtfac;
    K.vz[i] += a2 * dtfac;
}

// ---------------------------------------------------------------- drift / gathers
// pos += vel*h (src/drift.cuh:24-26) over the slow list of a split level.
__global__ void k_drift_slow(SoA P, const int32_t* __restrict__ L,
                             const hhs_partition* __restrict__ counts, double h) {
    const int ns = counts->n_slow;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) {
        const int g = L[s];
        P.x[g] = f64_add(P.x[g], f64_mul(P.vx[g], h));
        P.y[g] = f64_add(P.y[g], f64_mul(P.vy[g], h));
        P.z[g] = f64_add(P.z[g], f64_mul(P.vz[g], h));
    }
}

__global__ void k_drift(SoA P, int n, double h) {
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
        P.x[g] = f64_add(P.x[g], f64_mul(P.vx[g], h));
        P.y[g] = f64_add(P.y[g], f64_mul(P.vy[g], h));
        P.z[g] = f64_add(P.z[g], f64_mul(P.vz[g], h));
    }
}

// prev[parent_id[i]] <- cur[i] for pos, vel, m, timestep (src/update_system.cuh:14-23)
__global__ void k_update_system(SoA prev, SoA cur, const int32_t* __restrict__ parent, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = parent[i];
        prev.x[p] = cur.x[i]; prev.y[p] = cur.y[i]; prev.z[p] = cur.z[i];
        prev.vx[p] = cur.vx[i]; prev.vy[p] = cur.vy[i]; prev.vz[p] = cur.vz[i];
        prev.m[p] = cur.m[i];
        prev.ts[p] = cur.ts[i];
    }
}

// Copy of the split (src/split.cuh:341-356): fast[k] <- total[F[k]], slow[k] <- total[L[k]]
// for pos, vel, m, timestep, id, with parent_id = the source index.
__global__ void k_gather_split(SoA T, SoA Ls, int32_t* __restrict__ lpar, SoA Fs,
                               int32_t* __restrict__ fpar, const int32_t* __restrict__ L,
                               const int32_t* __restrict__ F,
                               const hhs_partition* __restrict__ counts) {
    const int nf = counts->n_fast, ns = counts->n_slow;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nf + ns;
         k += gridDim.x * blockDim.x) {
        const bool fast = k < nf;
        const int d = fast ? k : k - nf;
        const int g = fast ? F[d] : L[d];
        SoA& D = fast ? Fs : Ls;
        D.x[d] = T.x[g]; D.y[d] = T.y[g]; D.z[d] = T.z[g];
        D.vx[d] = T.vx[g]; D.vy[d] = T.vy[g]; D.vz[d] = T.vz[g];
        D.m[d] = T.m[g]; D.ts[d] = T.ts[g];
        D.id[d] = T.id[g];
        (fast ? fpar : lpar)[d] = g;
    }
}

inline int grid_for(int n, int block) { return (n + block - 1) / block; }
inline int grid_stride(int n, int block) {
    int g = grid_for(n, block);
    return g < kSms * 8 ? (g > 0 ? g : 1) : kSms * 8;
}

}  // namespace

hhs_status launch_timesteps(const SoA& P, const int32_t* list, int n, double eta,
                            hhs_precision prec, cudaStream_t stream, const PeerOut& po) {
    if (n <= 0) return HHS_OK;
    if (po.lo < 0 || po.n_peer < 0 || po.n_peer > kMaxPeers) return HHS_ERR_INVALID_ARG;
    const int hi = po.hi < 0 ? n : po.hi;
    if (hi > n || po.lo > hi) return HHS_ERR_INVALID_ARG;
    if (hi == po.lo) return HHS_OK;  // an empty shard
    const double eta_s2 = eta / 1.41421356237309504880;  // eta / M_SQRT2
    const TsArgs A{eta, eta_s2, (float)(1.0 / eta_s2), (float)(1.0 / eta)};
    // rows of a CTA: the rows share the columns' conversion, but every SM should have its four
    // CTAs (16384 particles: 261 us with 32 rows, 363 with 64; 32768: 823 with 32, 992 with 64)
    const int rows = hi - po.lo, T = rows <= 32 * kSms ? 8 : (rows <= 64 * kSms ? 16 : kTsMaxRows);
    if (prec == HHS_PREC_FP64)
        k_timesteps<HHS_PREC_FP64><<<grid_for(rows, T), kTsThreads, 0, stream>>>(P, list, n, T, A, po);
    else
        k_timesteps<HHS_PREC_MIXED><<<grid_for(rows, T), kTsThreads, 0, stream>>>(P, list, n, T, A, po);
    HHS_LAUNCH_CHECK();
    return HHS_OK;
}

hhs_status launch_kick_level(const SoA& P, const int32_t* fast_list,
                             const int32_t* slow_list, const hhs_partition* counts,
                             int n_max, double dt, double eps2, hhs_precision prec,
                             cudaStream_t stream, const PeerOut& po) {
    if (n_max <= 0) return HHS_OK;
    if (po.lo < 0 || po.n_peer < 0 || po.n_peer > kMaxPeers) return HHS_ERR_INVALID_ARG;
    // hi >= 0: a shard whose bounds the caller took from the host copy of the counts
    const int hi = po.hi < 0 ? n_max : po.hi;
    if (hi > n_max || po.lo > hi) return HHS_ERR_INVALID_ARG;
    if (hi == po.lo) return HHS_OK;
    const int grid = grid_for(hi - po.lo, kKickBlock);
    if (prec == HHS_PREC_FP64)
        k_kick_level_fp64<<<grid, kKickBlock, 0, stream>>>(P, fast_list, slow_list, counts, dt,
                                                           eps2, po);
    else
        k_kick_level_mixed<<<grid, kKickBlock, 0, stream>>>(P, fast_list, slow_list, counts, dt,
                                                            (float)eps2, po);
    HHS_LAUNCH_CHECK();
    return HHS_OK;
}

// Whether a thread per sink is the faster form for n sinks and m sources. Its time is m source
// visits one after another; the other forms take whole rounds of CTAs for 8 (FP64) or 32 sinks each,
// which few sources leave mostly idle. The models below are fits of the measured microseconds
// (thread / CTA), FP64: 4096 x 10 6.2 / 8.3, x 64 14.4 / 8.3, 32768 x 10 6.2 / 43, x 300 55 / 74, x 1500
// 258 / 207, 100000 x 100 36 / 140, x 300 99 / 213; mixed: 32768 x 10 6.2 / 8.3, x 64 10.3 / 10.3,
// x 224 24.6 / 14.8, 100000 x 20 8.3 / 18.5, x 100 23 / 25, x 300 62 / 49.
static bool few_sources(int n, int m, hhs_precision prec) {
    const double dn = n, dm = m;
    if (prec == HHS_PREC_FP64) {
        const double rounds = std::ceil(dn / (kK64Sinks * 2 * kSms)), stages = (m + kK64Sources - 1) / kK64Sources;
        return 2.5 + 0.17 * dm * std::max(1.0, dn / 55000.0) < rounds * (1.0 + 1.9 * stages);
    }
    return 3.6 + 0.0915 * dm * std::max(1.0, dn / 48000.0) < 1.4 + 1.26e-4 * dn + 1.3e-6 * dn * dm;
}

hhs_status launch_kick_pair(const SoA& sink, double* ax, double* ay, double* az,
                            const SoA& src, int n_sink, int n_src, double dtfac,
                            hhs_precision prec, cudaStream_t stream) {
    if (n_sink <= 0) return HHS_OK;
    if (few_sources(n_sink, n_src, prec)) {
        const int grid = grid_for(n_sink, kKickBlock);
        if (prec == HHS_PREC_FP64)
            k_kick_few_fp64<<<grid, kKickBlock, 0, stream>>>(sink, ax, ay, az, src, n_sink, n_src, dtfac);
        else
            k_kick_few_mixed<<<grid, kKickBlock, 0, stream>>>(sink, ax, ay, az, src, n_sink, n_src, dtfac);
    } else if (prec == HHS_PREC_FP64) {
        constexpr int bytes = (int)sizeof(Kick64Smem);
        HHS_CUDA_TRY(cudaFuncSetAttribute(k_kick_pair_fp64,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        k_kick_pair_fp64<<<grid_for(n_sink, kK64Sinks), kK64Threads, bytes, stream>>>(
            sink, ax, ay, az, src, n_sink, n_src, dtfac);
    } else
        k_kick_pair_mixed<<<grid_for(n_sink, 32), 32 * kPmWarps, 0, stream>>>(
            sink, ax, ay, az, src, n_sink, n_src, dtfac);
    HHS_LAUNCH_CHECK();
    return HHS_OK;
}

hhs_status launch_drift_slow(const SoA& P, const int32_t* slow_list,
                             const hhs_partition* counts, int n_max, double h,
                             cudaStream_t stream) {
    if (n_max <= 0) return HHS_OK;
    k_drift_slow<<<grid_stride(n_max, 256), 256, 0, stream>>>(P, slow_list, counts, h);
    HHS_LAUNCH_CHECK();
    return HHS_OK;
}

hhs_status launch_drift(const SoA& P, int n, double h, cudaStream_t stream) {
    if (n <= 0) return HHS_OK;
    k_drift<<<grid_stride(n, 256), 256, 0, stream>>>(P, n, h);
    HHS_LAUNCH_CHECK();
    return HHS_OK;
}

hhs_status launch_update_system(const SoA& prev, const SoA& cur, const int32_t* parent_id,
                                int n, cudaStream_t stream) {
    if (n <= 0) return HHS_OK;
    k_update_system<<<grid_stride(n, 256), 256, 0, stream>>>(prev, cur, parent_id, n);
    HHS_LAUNCH_CHECK();
    return HHS_OK;
}

hhs_status launch_gather_split(const SoA& total, const SoA& slow, int32_t* slow_parent,
                               const SoA& fast, int32_t* fast_parent,
                               const int32_t* slow_list, const int32_t* fast_list,
                               const hhs_partition* counts, int n_max, cudaStream_t stream) {
    if (n_max <= 0) return HHS_OK;
    k_gather_split<<<grid_stride(n_max, 256), 256, 0, stream>>>(
        total, slow, slow_parent, fast, fast_parent, slow_list, fast_list, counts);
    HHS_LAUNCH_CHECK();
    return HHS_OK;
}
