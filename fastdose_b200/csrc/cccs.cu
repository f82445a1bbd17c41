// cccs.cu -- collapsed-cone convolution/superposition in beam's-eye view.
//
// Restates d_DoseComputeCollective (FastDoseLib/src/DoseComp.cu:217-392).  For
// every forward zenith bin theta (theta <= pi/2) and azimuth phi, the rays of
// all BEV pixels -- translates of one base ray starting at (0.5, 0.5, 0) in
// normalised BEV units -- march slice by slice through voxel boundaries.  Per
// segment of path length p (physical, with divergence) in voxel v:
//     dose[v] += (A/a * XA + B/b * XB) * p * rho[v]       (g == 1, quirk Q1)
//     sum_p[v] += p * rho[v]
//     X <- T[v] (1 - e^{-k p rho}) + e^{-k p rho} X          for (k, X) in {(a, XA), (b, XB)}
// with lateral wrap-around and the recursion reset on crossing an edge (Q4).
// After all azimuths of a slice, dose_bev[s] += sum_phi dose / (sum_p_lastphi + 1e-4)
// (Q2: the path sum of the last azimuth only).
//
// B200 design.  (Batches of 8 x 8, 12 x 12 and 16 x 16 maps take the
// voxel-stationary march further down; this paragraph is about the instances
// for the other maps.)  The reference runs one block per beamlet with one thread per
// pixel and a block barrier after every ray step, azimuths in sequence.  Here a
// block owns one beamlet (schedule 0: all zenith bins in turn) or one
// (beamlet, zenith bin) (schedule 1), and each WARP owns one azimuth: its 32
// lanes carry all P rays (P/32 independent recursions per lane, which the
// scheduler interleaves), every lane computes the shared base-ray step itself
// (the warp stays converged, no broadcast), and the only barriers are the
// three per slice that stage the slice's Terma/density pair into shared memory
// and reduce the azimuths.  Within one step the rays of a beamlet deposit into
// distinct voxels (a shift permutation), so the warp-private deposit buffer
// needs only a __syncwarp between steps.
//
// Boundary decisions (next voxel boundary, slice snap, lateral wrap) use
// correctly rounded float operations in the order the reference writes them,
// starting from cone directions computed on the host; the CPU oracle performs
// the identical operations, so both march the same segments bit for bit.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <vector>

#include "fd2_internal.cuh"

namespace fd2 {

namespace {

constexpr int kStepCap = 1 << 20;  // per-slice step cap (the watchdog bound)
constexpr int kMapThreads = 256;     // the common-map instances are compiled for at most 8 azimuth warps
constexpr int kSpreadThreads = 768;  // and the spread ones (kWpa > 1) for blocks of up to 24 warps
constexpr int kMaxCluster = 4;       // blocks of a spread cluster

struct RayGeom {  // per-beamlet scalars the march needs
    float hx, hy;      // fmap_size / 2
    float bsx, bsy;    // beamlet_size
    float ls, lim_min, inv_sad;
    float ffx, ffy;    // fmap size as float
    int fx, fy, P, L;
};

// 1/x on the special-function unit (PTX rcp.approx.ftz.f32).
__device__ __forceinline__ float rcp_sfu(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A cone direction with what the boundary step needs of it, formed once per
// (zenith, azimuth) pass: the sign of each component and the reciprocal of its
// magnitude (+inf for a zero component).
struct ConeDir {
    float3 d, sg, ra;
};

__device__ __forceinline__ ConeDir make_cone_dir(float3 d) {
    ConeDir k;
    k.d = d;
    k.sg = make_float3(d.x < 0.0f ? -1.0f : 1.0f, d.y < 0.0f ? -1.0f : 1.0f, d.z < 0.0f ? -1.0f : 1.0f);
    k.ra = make_float3(rcp_sfu(fabsf(d.x)), rcp_sfu(fabsf(d.y)), rcp_sfu(fabsf(d.z)));
    return k;
}

// The reference's step to the next boundary along one axis (its build uses
// -use_fast_math, whose a/b is a * rcp.approx(b)):
//     (ceil(c + 1e-3) - c) / d    for d > 0,
//     (floor(c - 1e-3) - c) / d   otherwise.
// With s = sign(d) and u = s c (exact), floor(c - 1e-3) - c = -(ceil(u + 1e-3) - u)
// (round-to-nearest is symmetric under negation) and the sign cancels against
// d's, so both cases are (ceil(u + 1e-3) - u) * rcp(|d|): one rounding
// function and no division per step.  u + 1e-3 and ceil(...) - u are single
// fused operations on the exact product s c, so they round as the
// reference's additions do.  A zero component gives rcp(0) = +inf, so an axis
// the ray does not move along never limits the step (the reference divides
// by zero there and the ray becomes NaN and never ends its slice).
__device__ __forceinline__ float step_to_boundary(float c, float s, float ra) {
    const float up = ceilf(__fmaf_rn(c, s, 1e-3f));
    return __fmul_rn(__fmaf_rn(-c, s, up), ra);
}

// d_nextPoint (DoseComp.cu:76-111): the next voxel-boundary point of the base ray.
__device__ __forceinline__ bool next_point(float3 c, const ConeDir& k, float3& np) {
    const float3 d = k.d;
    float sx = step_to_boundary(c.x, k.sg.x, k.ra.x), sy = step_to_boundary(c.y, k.sg.y, k.ra.y),
          sz = step_to_boundary(c.z, k.sg.z, k.ra.z);
    float take = fminf(fminf(sx, sy), sz);
    np = make_float3(__fmaf_rn(take, d.x, c.x), __fmaf_rn(take, d.y, c.y), __fmaf_rn(take, d.z, c.z));
    bool flag = fabsf(__fsub_rn(np.z, roundf(np.z))) < 1e-4f;
    if (flag) {
        np = make_float3(__fmaf_rn(sz, d.x, c.x), __fmaf_rn(sz, d.y, c.y), roundf(__fmaf_rn(sz, d.z, c.z)));
    }
    return flag;
}

// Lateral voxel column of the segment midpoint (d_calcCoords, DoseComp.cu:147-164).
//
// The reference's r = fmodf(m, ff), plus ff when negative, is computed
// without fmodf: q = floor(m / ff) (the division may round q one off near a
// multiple of ff), r = m - q ff in one fused operation, then one correction by
// +-ff.  For m >= 0 the fused result is exact (the true remainder, or it minus
// or plus ff, all representable by Sterbenz's lemma) and the correction lands
// on the exact remainder, which is what fmodf returns.  For m < 0 the
// reference rounds fmod + ff once; the fused operation rounds the same exact
// value once, or, when q is one off, produces the exact fmod (Sterbenz) and the
// correction rounds fmod + ff once.  Both paths give the reference's float.
__device__ __forceinline__ int mid_index(float b, float n, float ff, int f) {
    const float m = __fmul_rn(__fadd_rn(b, n), 0.5f);
    const float q = floorf(__fdiv_rn(m, ff));
    float r = __fmaf_rn(-q, ff, m);
    if (r < 0.0f)
        r = __fadd_rn(r, ff);
    else if (r >= ff)
        r = __fsub_rn(r, ff);
    const int i = (int)floorf(r);
    return i < f ? i : f - 1;
}

__device__ __forceinline__ bool crosses_edge(float b, float n, float ff) {
    return floorf(__fdividef(b, ff)) != floorf(__fdividef(n, ff));
}

// 4 bytes from global to shared memory without passing through registers
// (PTX cp.async), committed as one group per call site; and the wait for all
// of this thread's groups.
__device__ __forceinline__ void cp_async4(float* smem_dst, const float* gsrc) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// 2^x on the special-function unit (PTX ex2.approx.ftz.f32).  The attenuation
// e^(-k p) is evaluated as 2^(-(k log2 e) p) with k log2 e formed once per
// zenith bin: one multiply and one MUFU operation per exponential.
__device__ __forceinline__ float exp2_sfu(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Segment length sqrt(l2) as l2 * rsqrt(l2) with the SFU reciprocal square
// root (PTX rsqrt.approx.ftz.f32); l2 > 0 for every segment the march takes.
__device__ __forceinline__ float rsqrt_sfu(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float seg_length(float l2) { return l2 * rsqrt_sfu(l2); }

// Could the midpoints of the segment c..n of two rays of a step, whole voxels
// apart, round to the same voxel?  (The base ray's midpoint close to a boundary;
// margins as in path_axis.)
__device__ __forceinline__ bool may_meet(float c, float n, float ff) {
    const float m = __fmul_rn(__fadd_rn(c, n), 0.5f);
    const float eps = 4e-6f + 3e-7f * (fabsf(c) + ff);
    return !(fabsf(m - floorf(m) - 0.5f) < 0.5f - eps);
}

__device__ __forceinline__ void named_barrier(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Block: n_phi warps (kWpa per azimuth of the block).  Dynamic shared memory:
// float2 tr[P] (Terma, density of the current slice) followed by float2
// dp[n_phi][P] (per-azimuth dose and path sums).  RPL = rays per lane (P <= 32 * RPL).
// kCols: every map of the batch is F x F with 25 <= F <= 32 -- lane l owns column
// l, so the x half of the voxel work is done once per lane and the y half once per
// row and shared by shuffles; RPL * kWpa >= F.  (With the arithmetic for several
// lanes a column, of narrower maps, it spilled 300 bytes instead of 156: 30 beams of
// 32 x 32, 8 azimuths 12.4 ms, 8.9 without.)
//
// kWpa > 1 spreads a (beamlet, zenith bin) that would leave most of the device
// idle: kWpa warps share an azimuth's rays, RPL each, and the azimuths are
// divided over the blocks of a cluster, which reduce them through each other's
// shared memory.  The rays of a step deposit into distinct voxels, whichever
// warp marches them, so one barrier of the azimuth's warps per step keeps the
// deposits of a voxel in step order, as with one warp; where rounding could let
// two rays of a step meet (a midpoint within some 1e-5 of a boundary), the warps
// deposit in turn.  The dose is the same bit for bit.
template <int RPL, bool kCols = false, bool kTab = false, int kWpa = 1>
__global__ void __launch_bounds__(kWpa > 1 ? kSpreadThreads : (kCols || kTab ? kMapThreads : 768),
                                  kWpa > 1 ? 1 : ((kCols || kTab) && RPL <= 8 ? 4 : (kCols || kTab ? 3 : 1)))
    cccs_kernel(const fd2_beam_t* __restrict__ beams,
                                                   const float* const* __restrict__ terma,
                                                   const float* const* __restrict__ dens,
                                                   float* const* __restrict__ dose,
                                                   const float4* __restrict__ dirs,  // [beam][n_tf][n_phi]
                                                   ConeParams cp, int split, float* __restrict__ split_out,
                                                   size_t split_stride, DeviceStatus* status,
                                                   const int* __restrict__ order) {
    extern __shared__ float2 smem[];
    __shared__ int s_ctrl[2];  // next slice index, abort flag
    int* s_next = &s_ctrl[0];
    int* s_abort = &s_ctrl[1];
    if (threadIdx.x == 0) *s_abort = 0;
    const int n_tf = cp.n_theta_fwd, n_phi = cp.n_phi;
    // order (optional, one block per beamlet only): the beamlet each block
    // marches, longest first, so the launch ends on short blocks
    namespace cg = cooperative_groups;
    const int n_cl = kWpa > 1 ? (int)cg::this_cluster().num_blocks() : 1;
    const int rank = kWpa > 1 ? (int)cg::this_cluster().block_rank() : 0;
    // kept apart from blockIdx.x where kWpa is 1: with one expression for both
    // the F = 20 instance spills 52 bytes instead of 44 and the F = 8 one 72
    // instead of none (24 beams of 20 x 20 maps: 141.4 against 140.4 ms)
    const int unit = blockIdx.x / n_cl;
    const int bi = split ? (kWpa > 1 ? unit : blockIdx.x) / n_tf : (order ? order[blockIdx.x] : blockIdx.x);
    const int t0 = split ? (kWpa > 1 ? unit : blockIdx.x) % n_tf : 0;
    const int t1 = split ? t0 + 1 : n_tf;
    const fd2_beam_t& b = beams[bi];
    RayGeom g;
    g.fx = b.fmap_size[0];
    g.fy = b.fmap_size[1];
    g.P = g.fx * g.fy;
    g.L = (int)b.long_dim;
    g.ffx = (float)g.fx;
    g.ffy = (float)g.fy;
    g.hx = g.fx * 0.5f;
    g.hy = g.fy * 0.5f;
    g.bsx = b.beamlet_size[0];
    g.bsy = b.beamlet_size[1];
    g.ls = b.long_spacing;
    g.lim_min = b.lim_min;
    g.inv_sad = 1.0f / b.sad;
    const size_t pitch = b.TermaBEV_pitch / sizeof(float);

    // kTab: per block, the (column, row) table entries of ray j of each lane
    // (x entry = column, y entry = F + row; all ones past the map), and per
    // azimuth warp the step's 2F halves
    __shared__ uint32_t s_pairs[kTab ? kWpa * RPL * 32 : 1];
    __shared__ float2 s_htab[kTab ? (kWpa > 1 ? kSpreadThreads / 32 : 8) * 64 : 1];
    if constexpr (kTab) {
        for (int i = threadIdx.x; i < kWpa * RPL * 32; i += blockDim.x)  // ray i / 32 of lane i % 32 is cell i
            s_pairs[i] = i < g.P ? (uint32_t)(i % g.fx) | (uint32_t)(g.fx + i / g.fx) << 16 : 0xffffffffu;
    }  // visible after the first slice's barrier

    float2* tr = smem;
    float2* dp = smem + g.P;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // this warp's azimuth in its block and its share of that azimuth's rays
    const int az = warp / kWpa, sub = warp % kWpa;
    const int n_az = n_phi / n_cl, phi = rank * n_az + az;
    float2* mydp = dp + (size_t)az * g.P;
    const float* __restrict__ T = terma[bi];
    const float* __restrict__ R = dens[bi];
    float* __restrict__ D = dose[bi];

    // per-ray constant pixel coordinates
    float fix[RPL], fiy[RPL];
    bool act[RPL];
    if constexpr (!kCols) {
#pragma unroll
        for (int j = 0; j < RPL; j++) {
            int r = j * 32 + lane;
            act[j] = r < g.P;
            fix[j] = (float)(r % g.fx);
            fiy[j] = (float)(r / g.fx);
        }
    }
    // kCols: this lane's column, and the row whose y half it computes for the others
    const bool clane = kCols && lane < g.fx;
    const float fcol = clane ? (float)lane : 0.0f, frow = fcol;

    // The slice most likely to come next (s + 1, or slice 0 of the next zenith
    // pass), copied by cp.async into s_stage (Terma, then density) during the
    // march and used only if that slice is the one taken.  Each thread copies
    // and later reads the same pixels, so no barrier stands between the two.
    constexpr int kStageP = 1024;
    __shared__ float s_stage[2 * kStageP];
    int st_s = -1;

    for (int t = t0; t < t1; t++) {
        const float Aa = cp.A_a[t], Bb = cp.B_b[t];
        const float ka = -cp.a[t] * 1.4426950408889634f, kb = -cp.b[t] * 1.4426950408889634f;  // -k log2(e)
        const float4 d4 = dirs[((size_t)bi * n_tf + t) * n_phi + phi];
        const ConeDir cd = make_cone_dir(make_float3(d4.x, d4.y, d4.z));
        float3 c = make_float3(0.5f, 0.5f, 0.0f);
        float fs = (c.z * g.ls + g.lim_min) * g.inv_sad;  // divergence factor at c, carried step to step
        float XA[RPL], XB[RPL];
#pragma unroll
        for (int j = 0; j < RPL; j++) XA[j] = XB[j] = 0.0f;

        // The slice of every pass is the rounded z of the first azimuth's base
        // ray (DoseComp.cu:300): when that ray ends a slice within 1e-3 below
        // the next plane it steps over it, and the reference skips that slice
        // for this zenith bin; the other azimuths keep marching from wherever
        // they stopped.
        if (threadIdx.x == 0) *s_next = 0;
        __syncthreads();  // the previous pass has finished; s_next is visible
        int s = *s_next;
        while (s < g.L) {
            cp_async_wait_all();  // this thread's staged pixels have landed
            for (int v = threadIdx.x; v < g.P; v += blockDim.x)
                tr[v] = s == st_s ? make_float2(s_stage[v], s_stage[kStageP + v])
                                  : make_float2(__ldg(T + (size_t)s * pitch + v), __ldg(R + (size_t)s * pitch + v));
            for (int v = kWpa > 1 ? 32 * sub + lane : lane; v < g.P; v += 32 * kWpa) mydp[v] = make_float2(0.0f, 0.0f);
            __syncthreads();
            st_s = s + 1 < g.L ? s + 1 : (t + 1 < t1 ? 0 : -1);
            if (st_s >= 0)
                for (int v = threadIdx.x; v < g.P; v += blockDim.x) {
                    cp_async4(&s_stage[v], T + (size_t)st_s * pitch + v);
                    cp_async4(&s_stage[kStageP + v], R + (size_t)st_s * pitch + v);
                }
            cp_async_commit();

            int guard = 0;
            for (;;) {
                float3 np;
                const bool flag = next_point(c, cd, np);
                const float fe = (np.z * g.ls + g.lim_min) * g.inv_sad;
                const float dzp = (np.z - c.z) * g.ls;
                auto rays = [&]() {
                    if constexpr (kCols) {
                        const float btx = __fadd_rn(c.x, fcol), ntx = __fadd_rn(np.x, fcol);
                        const int cx = mid_index(btx, ntx, g.ffx, g.fx);
                        const bool wrapx = crosses_edge(btx, ntx, g.ffx);
                        const float dxp = (ntx - g.hx) * g.bsx * fe - (btx - g.hx) * g.bsx * fs;
                        const float dxz2 = dxp * dxp + dzp * dzp;
                        const float bty = __fadd_rn(c.y, frow), nty = __fadd_rn(np.y, frow);
                        const int ycode = mid_index(bty, nty, g.ffy, g.fy) | (crosses_edge(bty, nty, g.ffy) ? 64 : 0);
                        const float dyq = (nty - g.hy) * g.bsy * fe - (bty - g.hy) * g.bsy * fs;
                        // kWpa: formed at every step, or the rows' numbers and predicates are
                        // kept over the steps and spill (32 x 32, one beam of 8 azimuths 1.77
                        // ms, 1.74 so)
                        int y0 = 0;
                        if constexpr (kWpa > 1) asm volatile("mov.b32 %0, %1;" : "=r"(y0) : "r"(sub * RPL));
#pragma unroll
                        for (int j = 0; j < RPL; j++) {
                            const int y = y0 + j;
                            const bool on = clane && y < g.fy;
                            const int yc = __shfl_sync(0xffffffffu, ycode, on ? y : 0);
                            const float dyp = __shfl_sync(0xffffffffu, dyq, on ? y : 0);
                            const int mi = on ? cx + g.fx * (yc & 63) : 0;
                            const bool wrap = wrapx || (yc & 64);
                            const float l2 = dxz2 + dyp * dyp;
                            const float len = seg_length(l2);
                            const float2 trv = tr[mi];
                            const float p = len * trv.y;
                            const float ea = exp2_sfu(ka * p), eb = exp2_sfu(kb * p);
                            const float dep = (Aa * XA[j] + Bb * XB[j]) * p;
                            if (on) {
                                float2 acc = mydp[mi];
                                acc.x += dep;
                                acc.y += p;
                                mydp[mi] = acc;
                            }
                            XA[j] = wrap ? 0.0f : __fmaf_rn(ea, XA[j] - trv.x, trv.x);
                            XB[j] = wrap ? 0.0f : __fmaf_rn(eb, XB[j] - trv.x, trv.x);
                        }
                    } else if constexpr (kTab) {
                        // F x F map, F <= 24: the rays of lane l are the cells l + 32 j,
                        // so all 32 lanes carry rays whatever F.  The step's 2F halves
                        // (x of each column, y of each row) are evaluated once, one per
                        // lane and round, into the warp's half table {+-|offset|,
                        // bytes into the slice}, the edge crossing as the sign bit;
                        // each ray then reads its column's and its row's entry.
                        float2* ht = s_htab + 64 * warp;
                        for (int h = lane; h < 2 * g.fx; h += 32) {
                            const bool yh = h >= g.fx;
                            const float off = (float)(yh ? h - g.fx : h);
                            const float hb = __fadd_rn(yh ? c.y : c.x, off), hn = __fadd_rn(yh ? np.y : np.x, off);
                            const float ff = yh ? g.ffy : g.ffx, hh = yh ? g.hy : g.hx, bs = yh ? g.bsy : g.bsx;
                            const int hi = mid_index(hb, hn, ff, yh ? g.fy : g.fx);
                            const float hq = fabsf((hn - hh) * bs * fe - (hb - hh) * bs * fs);
                            const float hs = crosses_edge(hb, hn, ff) ? -hq : hq;
                            const int bytes = (int)sizeof(float2) * (yh ? hi * g.fx : hi);
                            ht[h] = make_float2(hs, __int_as_float(bytes));
                        }
                        __syncwarp();
                        const float dz2 = dzp * dzp;
#pragma unroll
                        for (int j = 0; j < RPL; j++) {
                            const uint32_t pr = s_pairs[32 * (kWpa > 1 ? sub * RPL + j : j) + lane];
                            const bool on = pr != 0xffffffffu;
                            const float2 xe = ht[on ? (pr & 0xffffu) : 0], ye = ht[on ? (pr >> 16) : 0];
                            const bool wrap = (__float_as_int(xe.x) | __float_as_int(ye.x)) < 0;
                            const int mb = __float_as_int(xe.y) + __float_as_int(ye.y);
                            const float dxz2 = xe.x * xe.x + dz2;
                            const float l2 = dxz2 + ye.x * ye.x;
                            const float len = seg_length(l2);
                            const float2 trv = *reinterpret_cast<const float2*>(reinterpret_cast<const char*>(tr) + mb);
                            const float p = len * trv.y;
                            const float ea = exp2_sfu(ka * p), eb = exp2_sfu(kb * p);
                            const float dep = (Aa * XA[j] + Bb * XB[j]) * p;
                            if (on) {
                                float2* acc_p = reinterpret_cast<float2*>(reinterpret_cast<char*>(mydp) + mb);
                                float2 acc = *acc_p;
                                acc.x += dep;
                                acc.y += p;
                                *acc_p = acc;
                            }
                            XA[j] = wrap ? 0.0f : __fmaf_rn(ea, XA[j] - trv.x, trv.x);
                            XB[j] = wrap ? 0.0f : __fmaf_rn(eb, XB[j] - trv.x, trv.x);
                        }
                    } else {
#pragma unroll
                    for (int j = 0; j < RPL; j++) {
                        const float btx = __fadd_rn(c.x, fix[j]), ntx = __fadd_rn(np.x, fix[j]);
                        const float bty = __fadd_rn(c.y, fiy[j]), nty = __fadd_rn(np.y, fiy[j]);
                        const int cx = mid_index(btx, ntx, g.ffx, g.fx);
                        const int cy = mid_index(bty, nty, g.ffy, g.fy);
                        const int mi = cx + cy * g.fx;
                        const bool wrap = crosses_edge(btx, ntx, g.ffx) || crosses_edge(bty, nty, g.ffy);
                        // physical segment length (d_calcLineSeg, DoseComp.cu:114-144)
                        const float dxp = (ntx - g.hx) * g.bsx * fe - (btx - g.hx) * g.bsx * fs;
                        const float dyp = (nty - g.hy) * g.bsy * fe - (bty - g.hy) * g.bsy * fs;
                        const float l2 = dxp * dxp + dyp * dyp + dzp * dzp;
                        const float len = seg_length(l2);
                        const float2 trv = tr[act[j] ? mi : 0];
                        const float p = len * trv.y;
                        const float ea = exp2_sfu(ka * p), eb = exp2_sfu(kb * p);
                        const float dep = (Aa * XA[j] + Bb * XB[j]) * p;
                        if (act[j]) {
                            float2 acc = mydp[mi];
                            acc.x += dep;
                            acc.y += p;
                            mydp[mi] = acc;
                        }
                        XA[j] = wrap ? 0.0f : __fmaf_rn(ea, XA[j] - trv.x, trv.x);
                        XB[j] = wrap ? 0.0f : __fmaf_rn(eb, XB[j] - trv.x, trv.x);
                    }
                    }
                };
                if constexpr (kWpa > 1) {
                    // the azimuth's warps in turn when two of its rays might meet in a voxel
                    const bool turns = may_meet(c.x, np.x, g.ffx) || may_meet(c.y, np.y, g.ffy);
                    for (int turn = turns ? 0 : sub;; turn++) {
                        if (turn == sub) rays();
                        named_barrier(1 + az, 32 * kWpa);
                        if (!turns || turn == kWpa - 1) break;
                    }
                } else {
                    rays();
                }
                c = np;
                fs = fe;
                __syncwarp();
                if (flag) break;
                if (++guard >= kStepCap) {
                    if (lane == 0) {
                        atomicExch(&status->code, (int)FD2_ERR_WATCHDOG);
                        if constexpr (kWpa > 1)
                            *cg::this_cluster().map_shared_rank(s_abort, 0) = 1;
                        else
                            *s_abort = 1;
                    }
                    break;
                }
            }
            if (threadIdx.x == 0 && (kWpa == 1 || rank == 0)) {
                // the first azimuth's plane after this slice; it always lies ahead
                const int nxt = (int)roundf(c.z);
                *s_next = nxt > s ? nxt : g.L;
            }
            if constexpr (kWpa > 1) {
                cg::this_cluster().sync();
                const int* ctrl = cg::this_cluster().map_shared_rank(s_ctrl, 0);
                const int s_new = ctrl[1] ? g.L : ctrl[0];
                // this block's share of the pixels, over all blocks' azimuths in order
                const float2* part[kMaxCluster];
#pragma unroll
                for (int r = 0; r < kMaxCluster; r++)
                    part[r] = cg::this_cluster().map_shared_rank(dp, r < n_cl ? r : 0);
                for (int v = rank * blockDim.x + threadIdx.x; v < g.P; v += n_cl * blockDim.x) {
                    float sum = 0.0f, last_sum_p = 0.0f;
#pragma unroll
                    for (int r = 0; r < kMaxCluster; r++)
                        if (r < n_cl)
                            for (int w = 0; w < n_az; w++) {
                                const float2 d = part[r][(size_t)w * g.P + v];
                                sum += d.x;
                                last_sum_p = d.y;
                            }
                    split_out[(size_t)unit * split_stride + (size_t)s * g.P + v] = sum / (last_sum_p + 1e-4f);
                }
                cg::this_cluster().sync();  // every block's sums and rank 0's s_next are read
                s = s_new;
                continue;
            }
            __syncthreads();
            const int s_new = *s_abort ? g.L : *s_next;
            // reduce azimuths in order; normalise by the last azimuth's path sum
            for (int v = threadIdx.x; v < g.P; v += blockDim.x) {
                float sum = 0.0f, last_sum_p;
                for (int w = 0; w < n_phi; w++) sum += dp[(size_t)w * g.P + v].x;
                last_sum_p = dp[(size_t)(n_phi - 1) * g.P + v].y;
                const float val = sum / (last_sum_p + 1e-4f);
                if (split)
                    split_out[(size_t)blockIdx.x * split_stride + (size_t)s * g.P + v] = val;
                else
                    // this block alone owns beam bi's dose and each (s, v) stays with
                    // one thread, so a fire-and-forget add gives D + val in pass order
                    // without waiting for D's old value
                    atomicAdd(D + (size_t)s * pitch + v, val);
            }
            __syncthreads();  // the sums and the slice are read; s_next was read by every thread
            s = s_new;
        }
    }
    cp_async_wait_all();  // a staged slice that was not taken
}

// dose_bev[s][v] += sum_t planes[t][s][v] (zenith bins in order)
__global__ void cccs_split_reduce(const fd2_beam_t* __restrict__ beams, float* const* __restrict__ dose,
                                  const float* __restrict__ planes, size_t stride, int n_tf) {
    const int bi = blockIdx.y;
    const fd2_beam_t& b = beams[bi];
    const int P = b.fmap_size[0] * b.fmap_size[1];
    const size_t n = (size_t)P * b.long_dim;
    const size_t pitch = b.TermaBEV_pitch / sizeof(float);
    float* D = dose[bi];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        size_t s = i / P, v = i % P;
        float acc = 0.0f;
        for (int t = 0; t < n_tf; t++) acc += planes[((size_t)bi * n_tf + t) * stride + i];
        D[s * pitch + v] += acc;
    }
}

// ---------------------------------------------------------------------------
// The voxel-stationary march of common square maps (F x F, F = G * R).
//
// Within one step every ray of an azimuth moves by the same whole number of
// voxels, so the map as seen by the rays is a cyclic shift of the map of
// voxels.  A lane therefore keeps its VOXELS in registers for a whole slice --
// lane v + F g holds column v, rows R g .. R g + R - 1: Terma, density and the
// dose sum -- and the ray states (XA, XB) move instead: a step that enters the
// next column rotates them by one lane (shuffles), one that enters the next row
// by one register.  A ray step then touches no memory, and the rows of a lane
// pair up in the packed FP32 instructions of sm_100 (fma/mul/add.rn.f32x2),
// which take one issue slot for two rays.
//
// What all rays of an azimuth share does not depend on the slice data: the base
// ray's points and when the shift changes.  One warp computes these path
// records for all azimuths, one azimuth per lane, into shared memory: the step
// chain of next_point is issued once per block instead of once per azimuth
// warp, and it runs while the other warps reduce the previous slice.  Two
// barriers per slice.
//
// kOwnPath is for launches of few blocks, where the chain of one block is the
// time: the other warps wait for those records, and a step's loads and votes are
// not hidden by other blocks.  There every warp computes its azimuth's path as it
// goes, beside the arithmetic of the rays, and the registers of a whole SM are
// taken.  The same operations on the same floats: the dose is the same bit for bit.
// One beam's zenith bins, rays in place / records / own path: 16 x 16, 6 azimuths,
// 0.125 cm pixels 1.81 / 2.11 / 1.65 ms; 12 x 12 2.12 / 1.82 / 1.42; 8 x 8 1.38 /
// 1.37 / 1.11.
//
// The lateral offset and the edge crossing of a column or row are the
// reference's own roundings, evaluated once per column and row (only the rays on
// the first and last column and row can cross an edge).  Where rounding
// could put a ray's segment midpoint into the neighbour of the voxel the shift
// gives it (a midpoint within some 1e-5 of a boundary), or a segment spans
// several voxels, the record asks for march_exact_step, which evaluates every
// ray's voxel and crossing as the reference does (about 0.1 % of the steps).
//
// Bound: instruction issue, and the slowest azimuth of each slice at the
// barrier.  CCCS time on one B200 against the march that kept the rays in place
// and the slice in shared memory: 100-beam torso plan, 15 070 beamlets of
// 16 x 16: 332 ms (356.9); one beam of 100 beamlets on the 64^3 slab: 1.53 ms
// (2.15); 360 beamlets of 12 x 12, 4 azimuths: 3.3 ms (5.4); of 8 x 8, 8
// azimuths: 2.5 ms (3.6).  Measured slower: the last azimuth's path sums in
// shared memory instead of registers (366 ms; every slice waits for that warp),
// a warp of its own for the paths with one barrier a slice (356 ms at 72
// registers and 4 blocks), the edge crossings in the path records (longer
// chain in the one warp that the others wait for).
// ---------------------------------------------------------------------------
constexpr int kMarchWarps = 8;   // azimuths a block may have
constexpr int kMarchSteps = 40;  // path records of an azimuth per round; a slice with more takes several rounds
constexpr float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the add's rounding mode

// Two floats in one 64-bit register pair, and the packed operations on them.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pk(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 up(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

// floor, ceil and round of |x| < 2^22 as adds of kMagic in the directed
// rounding mode (FMA pipe) instead of conversions (special-function pipe).
__device__ __forceinline__ float floor_biased(float x) { return __fadd_rd(x, kMagic); }
__device__ __forceinline__ int biased_int(float b) { return __float_as_int(b) - __float_as_int(kMagic); }
__device__ __forceinline__ float round_biased(float x) { return __fsub_rn(__fadd_rn(x, kMagic), kMagic); }

// step_to_boundary and next_point with the roundings as biased adds: the same
// floats for |c| < 2^22 (Reach::admits bounds the path).
__device__ __forceinline__ float step_to_boundary_biased(float c, float s, float ra) {
    const float up = __fsub_rn(__fadd_ru(__fmaf_rn(c, s, 1e-3f), kMagic), kMagic);
    return __fmul_rn(__fmaf_rn(-c, s, up), ra);
}
__device__ __forceinline__ bool next_point_biased(float3 c, const ConeDir& k, float3& np) {
    const float3 d = k.d;
    const float sx = step_to_boundary_biased(c.x, k.sg.x, k.ra.x), sy = step_to_boundary_biased(c.y, k.sg.y, k.ra.y),
                sz = step_to_boundary_biased(c.z, k.sg.z, k.ra.z);
    const float take = fminf(fminf(sx, sy), sz);
    np = make_float3(__fmaf_rn(take, d.x, c.x), __fmaf_rn(take, d.y, c.y), __fmaf_rn(take, d.z, c.z));
    // (a tie rounds to even here and away from zero in roundf; the test's 1e-4 is far from a tie)
    const bool flag = fabsf(__fsub_rn(np.z, round_biased(np.z))) < 1e-4f;
    if (flag)
        np = make_float3(__fmaf_rn(sz, d.x, c.x), __fmaf_rn(sz, d.y, c.y), round_biased(__fmaf_rn(sz, d.z, c.z)));
    return flag;
}

// Bits of a path record's code.
enum : int {
    kRecEnd = 1,                      // the step ends the slice
    kRecExact = 2,                    // march_exact_step
    kRecMoveX = 4, kRecMoveY = 8,     // the shift changed by one column / row before this step
};

// Shared memory of a march block.  A map's cell (column v, row r) is at
// v * S + r: a lane's rows are consecutive, and with S = F + 4 (F a multiple of
// 8) eight neighbouring lanes' 16-byte accesses hit distinct banks.
template <int F, int kW>
struct MarchShared {
    static constexpr int S = F + 4;
    float4 rec[kW][kMarchSteps];  // next point x, y; divergence factor there; (depth of the step)^2
    int code[kW][kMarchSteps];
    alignas(16) float T[2][F * S];         // this slice and the one staged behind it
    alignas(16) float R[2][F * S];
    alignas(16) float dose[kW][F * S];  // each azimuth's sums of the slice
    alignas(16) float path[F * S];               // the last azimuth's path sums
    alignas(16) float xa[kW][F * S], xb[kW][F * S];  // ray states in march_exact_step
    alignas(16) float row[kW][2][F];    // the step's lateral offset of each row
    float3 c[kW];                 // chain state: point, voxel shift,
    int2 k[kW];
    ConeDir dir[kW];              // direction,
    int count[kW];                // records of this round,
    int next, more, abort;                 // next slice; some azimuth has more rounds; step cap hit
};

// Per-beamlet and per-pass values of a march.
struct MarchRay {
    float bsx, bsy, ls, lim_min, inv_sad;
    float ka, kb, Aa, Bb;
};

__device__ __forceinline__ int pos_mod(int a, int f) {
    const int r = a % f;
    return r < 0 ? r + f : r;
}

// One axis of a path record: the voxel shift of the segment c..n, and whether
// the shift may not hold for every ray.
template <int F>
__device__ __forceinline__ int path_axis(float c, float n, bool& exact) {
    const float m = __fmul_rn(__fadd_rn(c, n), 0.5f);
    const float fl = floor_biased(m);
    // a ray's midpoint differs from the base ray's by at most 1.2e-7 of its
    // coordinate, and the remainder by F rounds by at most 2e-6 more
    const float eps = 4e-6f + 3e-7f * (fabsf(c) + F);
    exact = exact || fabsf(m - __fsub_rn(fl, kMagic) - 0.5f) > 0.5f - eps || fabsf(n - c) > 1.5f;
    return biased_int(fl);
}

// The record of the step c..n of a base ray at voxel shift k0, and the shift kn
// along it; whether it asks for march_exact_step.
template <int F>
__device__ __forceinline__ bool path_record(const MarchRay& g, float3 c, float3 n, int2 k0, int2& kn, float4& rec) {
    bool exact = false;
    kn = make_int2(path_axis<F>(c.x, n.x, exact), 0);
    kn.y = path_axis<F>(c.y, n.y, exact);
    const float dz = (n.z - c.z) * g.ls;
    rec = make_float4(n.x, n.y, (n.z * g.ls + g.lim_min) * g.inv_sad, __fmul_rn(dz, dz));
    return exact || abs(kn.x - k0.x) > 1 || abs(kn.y - k0.y) > 1;
}

// The first azimuth's plane after slice s; it always lies ahead.
__device__ __forceinline__ int plane_after(float z, int s, int L) {
    const int nxt = (int)roundf(z);
    return nxt > s ? nxt : L;
}

// One round of every azimuth's path (lane = azimuth) from the chain state in
// shared memory.  `open`: the lane's slice is not finished.
template <int F, int kW>
__device__ __forceinline__ void march_paths(MarchShared<F, kW>& sm, const MarchRay& g, int n_phi, int s, int L, bool open) {
    const int w = threadIdx.x & 31;
    int n = 0;
    if (w < n_phi && open) {
        float3 c = sm.c[w];
        int2 k0 = sm.k[w];
        const ConeDir k = sm.dir[w];
        bool flag = false;
        while (!flag && n < kMarchSteps) {
            float3 np;
            int2 kn;
            flag = next_point_biased(c, k, np);
            const bool exact = path_record<F>(g, c, np, k0, kn, sm.rec[w][n]);
            sm.code[w][n++] = (flag ? kRecEnd : 0) | (exact ? kRecExact : 0) | (kn.x != k0.x ? kRecMoveX : 0) |
                              (kn.y != k0.y ? kRecMoveY : 0);
            c = np;
            k0 = kn;
        }
        sm.k[w] = k0;
        sm.c[w] = c;
        open = !flag;
        if (w == 0 && flag) {
            sm.next = plane_after(c.z, s, L);
        }
    }
    if (w < n_phi) sm.count[w] = n;
    const bool more = __any_sync(0xffffffffu, w < n_phi && open);
    if (w == 0) sm.more = more;
}

// A step in which some ray's voxel may not be the shifted one: every ray's
// voxel and edge crossing as the reference computes them, from b to n.  The
// warp's states and sums are in shared memory, each at its voxel: the states
// come in at the old shift (ox, oy), taken modulo F, and leave at the new one,
// which is returned.  Rays of one step can only meet in a voxel next to their
// own, so four passes, one per parity of column and row, keep the additions
// apart and their order fixed.
template <int F, int G, int R, int kW>
__device__ __noinline__ int2 march_exact_step(MarchShared<F, kW>& sm, int buf, const MarchRay& g, float2 b, float2 n,
                                              float fs, float fe, float dz2, int ox, int oy, bool last) {
    constexpr int S = MarchShared<F, kW>::S;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, v = lane % F, grp = lane / F;
    const bool on = grp < G;
    const float ff = (float)F, hh = 0.5f * F;
    const int kx = pos_mod(biased_int(floor_biased(__fmul_rn(__fadd_rn(b.x, n.x), 0.5f))), F);
    const int ky = pos_mod(biased_int(floor_biased(__fmul_rn(__fadd_rn(b.y, n.y), 0.5f))), F);
    const int lx = pos_mod(v - kx, F);
    const float bx = __fadd_rn(b.x, (float)lx), nx = __fadd_rn(n.x, (float)lx);
    const int ix = mid_index(bx, nx, ff, F);
    const bool wx = crosses_edge(bx, nx, ff);
    const float dx = (nx - hh) * g.bsx * fe - (bx - hh) * g.bsx * fs;
    const float dxz2 = dx * dx + dz2;
    float *dose = sm.dose[warp], *xa = sm.xa[warp], *xb = sm.xb[warp];
    float XA[R], XB[R];
    __syncwarp();
#pragma unroll
    for (int j = 0; j < R; j++) {
        const int from = pos_mod(lx + ox, F) * S + pos_mod(grp * R + j - ky + oy, F);
        XA[j] = on ? xa[from] : 0.0f;
        XB[j] = on ? xb[from] : 0.0f;
    }
    __syncwarp();
    for (int pass = 0; pass < 4; pass++) {
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int row = grp * R + j;
            if (on && pass == ((v & 1) | (row & 1) << 1)) {
                const int ly = pos_mod(row - ky, F);
                const float by = __fadd_rn(b.y, (float)ly), ny = __fadd_rn(n.y, (float)ly);
                const int q = ix * S + mid_index(by, ny, ff, F);
                const float dy = (ny - hh) * g.bsy * fe - (by - hh) * g.bsy * fs;
                const float p = seg_length(dxz2 + dy * dy) * sm.R[buf][q];
                const float t = sm.T[buf][q];
                dose[q] = __fmaf_rn(g.Aa * XA[j] + g.Bb * XB[j], p, dose[q]);
                if (last) sm.path[q] += p;
                const bool wrap = wx || crosses_edge(by, ny, ff);
                xa[v * S + row] = wrap ? 0.0f : __fmaf_rn(exp2_sfu(g.ka * p), XA[j] - t, t);
                xb[v * S + row] = wrap ? 0.0f : __fmaf_rn(exp2_sfu(g.kb * p), XB[j] - t, t);
            }
        }
        __syncwarp();
    }
    return make_int2(kx, ky);
}

// A lane's R consecutive cells to and from shared memory, in pairs.
template <int R>
__device__ __forceinline__ void load_cells(const float* p, F2 (&o)[R / 2]) {
    if constexpr (R % 4 == 0) {
#pragma unroll
        for (int q = 0; q < R / 2; q += 2) {
            const float4 a = *reinterpret_cast<const float4*>(p + 2 * q);
            o[q] = pk(a.x, a.y);
            o[q + 1] = pk(a.z, a.w);
        }
    } else {
#pragma unroll
        for (int q = 0; q < R / 2; q++) {
            const float2 a = *reinterpret_cast<const float2*>(p + 2 * q);
            o[q] = pk(a.x, a.y);
        }
    }
}
template <int R>
__device__ __forceinline__ void store_cells(float* p, const F2 (&o)[R / 2]) {
    if constexpr (R % 4 == 0) {
#pragma unroll
        for (int q = 0; q < R / 2; q += 2)
            *reinterpret_cast<float4*>(p + 2 * q) = make_float4(up(o[q]).x, up(o[q]).y, up(o[q + 1]).x, up(o[q + 1]).y);
    } else {
#pragma unroll
        for (int q = 0; q < R / 2; q++) *reinterpret_cast<float2*>(p + 2 * q) = up(o[q]);
    }
}

// kW: azimuths the shared memory is for.  80 registers: four blocks of 6 azimuths
// an SM, six of up to 4 (with the shared memory of 8 azimuths only five fit: 1800
// beams of 16 x 16, 4 azimuths 14.7 ms, 12.0 so, 12.1 with the rays in place).
template <int F, int G, int R, int kW, bool kOwnPath>
__global__ void __launch_bounds__(32 * kW, kOwnPath ? 1 : (kW <= 4 ? 6 : 3))
    cccs_march_kernel(const fd2_beam_t* __restrict__ beams, const float* const* __restrict__ terma,
                      const float* const* __restrict__ dens, float* const* __restrict__ dose,
                      const float4* __restrict__ dirs,  // [beam][n_tf][n_phi]
                      ConeParams cp, int split, float* __restrict__ split_out, size_t split_stride, DeviceStatus* status,
                      const int* __restrict__ order) {
    static_assert(F == G * R && G > 1 && R % 2 == 0 && F * G <= 32, "a lane holds R rows of a column in pairs");
    constexpr unsigned kAll = 0xffffffffu;
    constexpr int P = F * F, S = MarchShared<F, kW>::S;
    __shared__ MarchShared<F, kW> sm;
    const int n_tf = cp.n_theta_fwd, n_phi = cp.n_phi;
    // split: one block per (zenith bin, beamlet), the widest bin (most steps per
    // slice) first; else one block per beamlet in `order` (longest first)
    const int nb = gridDim.x / n_tf;
    const int bi = split ? blockIdx.x % nb : (order ? order[blockIdx.x] : blockIdx.x);
    const int t0 = split ? n_tf - 1 - blockIdx.x / nb : 0;
    const int t1 = split ? t0 + 1 : n_tf;
    const fd2_beam_t& bm = beams[bi];
    const int L = (int)bm.long_dim;
    const size_t pitch = bm.TermaBEV_pitch / sizeof(float);
    const float* __restrict__ T = terma[bi];
    const float* __restrict__ Rho = dens[bi];
    float* __restrict__ D = dose[bi];
    MarchRay g;
    g.bsx = bm.beamlet_size[0];
    g.bsy = bm.beamlet_size[1];
    g.ls = bm.long_spacing;
    g.lim_min = bm.lim_min;
    g.inv_sad = 1.0f / bm.sad;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int v = lane % F, grp = lane / F;
    const bool on = grp < G, last = warp == n_phi - 1;
    const bool yl = grp == 1;  // group 0 evaluates the columns' offsets, group 1 the rows'
    const int cell = (v * S + (on ? grp * R : 0));
    if (threadIdx.x == 0) sm.abort = 0;
    if (L <= 0) return;

    // thread i of the block copies pixels i, i + blockDim, ... of a slice
    auto stage = [&](int s, int buf) {
        for (int i = threadIdx.x; i < P; i += blockDim.x) {
            const int q = i % F * S + i / F;
            cp_async4(&sm.T[buf][q], T + (size_t)s * pitch + i);
            cp_async4(&sm.R[buf][q], Rho + (size_t)s * pitch + i);
        }
        cp_async_commit();
    };
    // the azimuths of slice s in order, normalised by the last one's path sum;
    // done by the warps that compute no path (the first does)
    const int rt0 = n_phi > 1 && !kOwnPath ? 32 : 0;
    auto reduce = [&](int t, int s) {
        for (int i = threadIdx.x - rt0; i < P; i += blockDim.x - rt0) {
            const int q = i % F * S + i / F;
            float sum = 0.0f;
            for (int w = 0; w < n_phi; w++) sum += sm.dose[w][q];
            const float val = sum / (sm.path[q] + 1e-4f);
            if (split)
                split_out[((size_t)bi * n_tf + t) * split_stride + (size_t)s * P + i] = val;
            else
                // this block alone owns beam bi's dose and each (s, i) stays with
                // one thread, so a fire-and-forget add gives D + val in pass order
                // without waiting for D's old value
                atomicAdd(D + (size_t)s * pitch + i, val);
        }
    };

    int buf = 0, staged = 0;
    stage(0, 0);
    int prev_s = -1, prev_t = 0;  // the slice whose sums wait to be reduced
    for (int t = t0; t < t1; t++) {
        g.ka = -cp.a[t] * 1.4426950408889634f;  // -k log2(e)
        g.kb = -cp.b[t] * 1.4426950408889634f;
        g.Aa = cp.A_a[t];
        g.Bb = cp.B_b[t];
        const F2 ka2 = pk(g.ka, g.ka), kb2 = pk(g.kb, g.kb), Aa2 = pk(g.Aa, g.Aa), Bb2 = pk(g.Bb, g.Bb);
        const float4 d4 = dirs[((size_t)bi * n_tf + t) * n_phi + warp];
        if (warp == 0 && lane < n_phi) {
            const float4 q4 = dirs[((size_t)bi * n_tf + t) * n_phi + lane];
            sm.dir[lane] = make_cone_dir(make_float3(q4.x, q4.y, q4.z));
            sm.c[lane] = make_float3(0.5f, 0.5f, 0.0f);
            sm.k[lane] = make_int2(0, 0);
        }
        // a move in x takes a state from lane ux, one in y the row carried over
        // from another group's lane uy; the ray on this lane's column (group 0) or
        // row `v` (group 1) changes by -step
        const bool xp = d4.x >= 0.0f, yp = d4.y >= 0.0f, yp_all = __any_sync(kAll, yp);
        const int ux = (xp ? (v == 0 ? F - 1 : v - 1) : (v == F - 1 ? 0 : v + 1)) + grp * F;
        const int uy = (yp ? (grp == 0 ? G - 1 : grp - 1) : (grp + 1 >= G ? 0 : grp + 1)) * F + v;
        const float step = (yl ? yp : xp) ? 1.0f : -1.0f;
        const float bs = yl ? g.bsy : g.bsx;
        float lf = (float)v;   // the ray on this lane's column or row
        float cb = 0.5f;       // the base ray's coordinate of this lane's axis
        F2 XA[R / 2], XB[R / 2];
#pragma unroll
        for (int q = 0; q < R / 2; q++) XA[q] = XB[q] = pk(0.0f, 0.0f);
        float fs = (0.0f * g.ls + g.lim_min) * g.inv_sad;  // divergence factor at the step's start
        // The slice of every pass is the rounded z of the first azimuth's base
        // ray (DoseComp.cu:300): when that ray ends a slice within 1e-3 below
        // the next plane it steps over it, and the reference skips that slice
        // for this zenith bin; the other azimuths keep marching from wherever
        // they stopped.
        int s = 0, par = 0;
        // kOwnPath: the azimuth's own path state
        const ConeDir cd = make_cone_dir(make_float3(d4.x, d4.y, d4.z));
        float3 c = make_float3(0.5f, 0.5f, 0.0f);
        int2 k0 = make_int2(0, 0);
        while (s < L) {
            F2 Tv[R / 2], Rv[R / 2], Dv[R / 2], Pv[R / 2];
            int s_next = L;
            auto load_slice = [&]() {
                load_cells<R>(&sm.T[buf][cell], Tv);
                load_cells<R>(&sm.R[buf][cell], Rv);
#pragma unroll
                for (int q = 0; q < R / 2; q++) {
                    if (!on) Tv[q] = Rv[q] = pk(0.0f, 0.0f);
                    Dv[q] = Pv[q] = pk(0.0f, 0.0f);
                }
            };
            auto store_sums = [&]() {
                if (on) {
                    store_cells<R>(&sm.dose[warp][cell], Dv);
                    if (last) store_cells<R>(&sm.path[cell], Pv);
                }
            };
            // the states to the shift of the coming step
            auto move = [&](bool move_x, bool move_y) {
                if (move_x) {
#pragma unroll
                    for (int q = 0; q < R / 2; q++) {
                        const float2 a = up(XA[q]), b = up(XB[q]);
                        XA[q] = pk(__shfl_sync(kAll, a.x, ux), __shfl_sync(kAll, a.y, ux));
                        XB[q] = pk(__shfl_sync(kAll, b.x, ux), __shfl_sync(kAll, b.y, ux));
                    }
                }
                if (move_y) {
                    if (R == 2 || kOwnPath ? yp_all : __any_sync(kAll, yp)) {
                        const float ea = __shfl_sync(kAll, up(XA[R / 2 - 1]).y, uy);
                        const float eb = __shfl_sync(kAll, up(XB[R / 2 - 1]).y, uy);
#pragma unroll
                        for (int q = R / 2 - 1; q >= 0; q--) {
                            XA[q] = pk(q ? up(XA[q ? q - 1 : 0]).y : ea, up(XA[q]).x);
                            XB[q] = pk(q ? up(XB[q ? q - 1 : 0]).y : eb, up(XB[q]).x);
                        }
                    } else {
                        const float ea = __shfl_sync(kAll, up(XA[0]).x, uy);
                        const float eb = __shfl_sync(kAll, up(XB[0]).x, uy);
#pragma unroll
                        for (int q = 0; q < R / 2; q++) {
                            const bool e = q == R / 2 - 1;
                            XA[q] = pk(up(XA[q]).y, e ? ea : up(XA[e ? q : q + 1]).x);
                            XB[q] = pk(up(XB[q]).y, e ? eb : up(XB[e ? q : q + 1]).x);
                        }
                    }
                }
            };
            // lateral offset over the step of the ray on this lane's column or row, its
            // edge crossing as the sign (the offset enters the length squared); rows'
            // offsets go to the warp's table, columns' come by shuffle
            auto offset = [&](float cn, float fe) {
                const float b = __fadd_rn(cb, lf), e = __fadd_rn(cn, lf);
                float d = fabsf((e - 0.5f * F) * bs * fe - (b - 0.5f * F) * bs * fs);
                d = floor_biased(__fdividef(b, (float)F)) != floor_biased(__fdividef(e, (float)F)) ? -d : d;
                if (yl) sm.row[warp][par][v] = d;
                return __shfl_sync(kAll, d, v);
            };
            // the rays of a step, at the offsets of the column and of the table
            auto rays = [&](float dx, float dz2) {
                const float dxz2 = dx * dx + dz2;
                F2 dy[R / 2];
                load_cells<R>(&sm.row[warp][par][on ? grp * R : 0], dy);
                const F2 dxz = pk(dxz2, dxz2);
#pragma unroll
                for (int q = 0; q < R / 2; q++) {
                    const F2 l2 = fma2(dy[q], dy[q], dxz);
                    const float2 l2s = up(l2);
                    const F2 p = mul2(mul2(l2, pk(rsqrt_sfu(l2s.x), rsqrt_sfu(l2s.y))), Rv[q]);
                    const float2 xa = up(mul2(p, ka2)), xb = up(mul2(p, kb2));
                    Dv[q] = fma2(fma2(Bb2, XB[q], mul2(Aa2, XA[q])), p, Dv[q]);
                    if (last) Pv[q] = add2(Pv[q], p);
                    XA[q] = fma2(pk(exp2_sfu(xa.x), exp2_sfu(xa.y)), sub2(XA[q], Tv[q]), Tv[q]);
                    XB[q] = fma2(pk(exp2_sfu(xb.x), exp2_sfu(xb.y)), sub2(XB[q], Tv[q]), Tv[q]);
                }
                // rays that crossed an edge start anew
                const bool wx = __float_as_int(dx) < 0;
                if (__any_sync(kAll, wx)) {
#pragma unroll
                    for (int q = 0; q < R / 2; q++) {
                        XA[q].v = wx ? 0ull : XA[q].v;
                        XB[q].v = wx ? 0ull : XB[q].v;
                    }
                }
                const bool w0 = __float_as_int(up(dy[0]).x) < 0, w1 = __float_as_int(up(dy[R / 2 - 1]).y) < 0;
                XA[0] = pk(w0 ? 0.0f : up(XA[0]).x, up(XA[0]).y);
                XB[0] = pk(w0 ? 0.0f : up(XB[0]).x, up(XB[0]).y);
                XA[R / 2 - 1] = pk(up(XA[R / 2 - 1]).x, w1 ? 0.0f : up(XA[R / 2 - 1]).y);
                XB[R / 2 - 1] = pk(up(XB[R / 2 - 1]).x, w1 ? 0.0f : up(XB[R / 2 - 1]).y);
            };
            // one step, whose shift changed by a column and a row
            auto ray_step = [&](const float4& rec, bool move_x, bool move_y) {
                move(move_x, move_y);
                if (yl ? move_y : move_x) lf -= step;
                lf = lf < 0.0f ? lf + F : (lf >= F ? lf - F : lf);
                const float cn = yl ? rec.y : rec.x;
                const float dx = offset(cn, rec.z);
                cb = cn;
                fs = rec.z;
                __syncwarp();
                rays(dx, rec.w);
                par ^= 1;
            };
            // a step from b to n in which some ray's voxel may not be the shifted one;
            // the states come at shift o and leave at the one returned
            auto exact_step = [&](float2 b, float2 n, float f0, float f1, float dz2, int ox, int oy) {
                if (on) {
                    store_cells<R>(&sm.dose[warp][cell], Dv);
                    store_cells<R>(&sm.xa[warp][cell], XA);
                    store_cells<R>(&sm.xb[warp][cell], XB);
                    if (last) store_cells<R>(&sm.path[cell], Pv);
                }
                const int2 k = march_exact_step<F, G, R, kW>(sm, buf, g, b, n, f0, f1, dz2, ox, oy, last);
                if (on) {
                    load_cells<R>(&sm.dose[warp][cell], Dv);
                    load_cells<R>(&sm.xa[warp][cell], XA);
                    load_cells<R>(&sm.xb[warp][cell], XB);
                    if (last) load_cells<R>(&sm.path[cell], Pv);
                }
                __syncwarp();
                return k;
            };
            if constexpr (kOwnPath) {
                if (s != staged) {  // the slice after the last one was skipped
                    cp_async_wait_all();
                    stage(s, buf);
                }
                cp_async_wait_all();
                __syncthreads();  // the slice stands, the last one's sums are used
                load_slice();
                staged = s + 1 < L ? s + 1 : (t + 1 < t1 ? 0 : -1);
                if (staged >= 0) stage(staged, buf ^ 1);
                bool flag = false;
                for (int guard = 0; !flag; guard++) {
                    if (guard >= kStepCap) {
                        if (lane == 0) {
                            atomicExch(&status->code, (int)FD2_ERR_WATCHDOG);
                            sm.abort = 1;
                        }
                        break;
                    }
                    float3 np;
                    int2 kn;
                    float4 rec;
                    flag = next_point_biased(c, cd, np);
                    if (path_record<F>(g, c, np, k0, kn, rec)) {
                        const int2 k = exact_step(make_float2(c.x, c.y), make_float2(np.x, np.y), fs, rec.z, rec.w,
                                                  pos_mod(k0.x, F), pos_mod(k0.y, F));
                        lf = (float)pos_mod(v - (yl ? k.y : k.x), F);
                        cb = yl ? rec.y : rec.x;
                        fs = rec.z;
                    } else {
                        ray_step(rec, kn.x != k0.x, kn.y != k0.y);
                    }
                    c = np;
                    k0 = kn;
                }
                store_sums();
                if (threadIdx.x == 0) sm.next = plane_after(c.z, s, L);
                __syncthreads();  // the slice's sums stand
                if (sm.abort) {
                    cp_async_wait_all();
                    return;
                }
                s_next = sm.next;
                reduce(t, s);
            } else {
                for (int round = 0;; round++) {
                    if (warp == 0) {
                        bool open = true;
                        if (round > 0) {  // azimuths still inside the slice: their last record does not end it
                            open = lane < n_phi && sm.count[lane] > 0 && !(sm.code[lane][sm.count[lane] - 1] & kRecEnd);
                            if ((long long)round * kMarchSteps >= kStepCap) {
                                open = false;
                                if (lane == 0) {
                                    atomicExch(&status->code, (int)FD2_ERR_WATCHDOG);
                                    sm.abort = 1;
                                }
                            }
                        }
                        __syncwarp();
                        march_paths<F, kW>(sm, g, n_phi, s, L, open);
                    }
                    if (round == 0) {
                        if (prev_s >= 0 && (warp > 0 || n_phi == 1)) reduce(prev_t, prev_s);
                        cp_async_wait_all();  // this thread's pixels of the slice have landed
                    }
                    __syncthreads();
                    if (sm.abort) return;  // the same for all: written before the barrier only
                    if (round == 0) load_slice();
                    const bool more = sm.more;
                    if (!more) {
                        s_next = sm.next;
                        // the next slice to come (or slice 0 of the next zenith pass)
                        const int st = s_next < L ? s_next : (t + 1 < t1 ? 0 : -1);
                        if (st >= 0) stage(st, buf ^ 1);
                    }
                    const int n = sm.count[warp];
                    for (int i = 0; i < n; i++) {
                        for (; i < n; i++) {
                            const int code = sm.code[warp][i];
                            if (__any_sync(kAll, code & kRecExact)) break;
                            const float4 rec = sm.rec[warp][i];
                            const bool mx = __any_sync(kAll, code & kRecMoveX), my = __any_sync(kAll, code & kRecMoveY);
                            move(mx, my);
                            if (yl ? my : mx) lf -= step;
                            lf = lf < 0.0f ? lf + F : (lf >= F ? lf - F : lf);
                            const float cn = yl ? rec.y : rec.x;
                            const float dx = offset(cn, rec.z);
                            cb = cn;
                            fs = rec.z;
                            __syncwarp();
                            rays(dx, rec.w);
                            par ^= 1;
                        }
                        if (i >= n) break;
                        const float4 rec = sm.rec[warp][i];
                        const int o = pos_mod(v - (int)lf, F);  // the shift: of x in group 0, of y in group 1
                        const int2 k = exact_step(make_float2(__shfl_sync(kAll, cb, 0), __shfl_sync(kAll, cb, F)),
                                                  make_float2(rec.x, rec.y), fs, rec.z, rec.w, __shfl_sync(kAll, o, 0),
                                                  __shfl_sync(kAll, o, F));
                        lf = (float)pos_mod(v - (yl ? k.y : k.x), F);
                        cb = yl ? rec.y : rec.x;
                        fs = rec.z;
                    }
                    if (!more) break;
                    __syncthreads();  // the round's records are used
                }
                store_sums();
                __syncthreads();  // the slice's sums stand, its records and data are used
                prev_s = s;
                prev_t = t;
            }
            buf ^= 1;
            s = s_next;
        }
    }
    if constexpr (kOwnPath)
        cp_async_wait_all();  // a slice staged and not taken
    else if (prev_s >= 0 && (warp > 0 || n_phi == 1))
        reduce(prev_t, prev_s);
}

template <int RPL, bool kCols, bool kTab = false>
int launch_instance(unsigned blocks, int threads, size_t shm, cudaStream_t st, const fd2_beam_t* d_beams,
                    const float* const* T, const float* const* R, float* const* D, const float4* dirs,
                    const ConeParams& cp, int split, float* planes, size_t plane_stride, DeviceStatus* status,
                    const int* order) {
    FD2_CHECK_CUDA(cudaFuncSetAttribute(cccs_kernel<RPL, kCols, kTab>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)shm));
    cccs_kernel<RPL, kCols, kTab><<<blocks, threads, shm, st>>>(d_beams, T, R, D, dirs, cp, split, planes,
                                                                 plane_stride, status, order);
    FD2_CHECK_CUDA(cudaGetLastError());
    return FD2_OK;
}

template <int F, int G, int R>
int launch_voxel_march(unsigned blocks, int n_phi, cudaStream_t st, const fd2_beam_t* d_beams,
                       const float* const* T, const float* const* Rho, float* const* D, const float4* dirs,
                       const ConeParams& cp, int split, float* planes, size_t plane_stride, DeviceStatus* status,
                       const int* order, int sm_count) {
    // kOwnPath up to some 20 warps an SM: later its blocks, one of more than 4
    // azimuths an SM, run one after the other (16 x 16, 6 azimuths, own path / records:
    // 2.2 blocks an SM 2.09 / 2.52 ms at 0.125 cm and 0.69 / 0.81 at 0.5; 3.8 blocks
    // 2.10 / 2.62 and 1.05 / 0.85).  8 x 8 maps leave room for two blocks.  Blocks of
    // whole beamlets are all long: only as many as run at once.
    const uint64_t half_blocks = split ? (F == 8 ? 12 : (n_phi <= 4 ? 10 : 5)) : (F == 8 || n_phi <= 4 ? 4 : 2);  // per SM
    const bool own_path = 2 * (uint64_t)blocks <= half_blocks * sm_count;
    (own_path ? cccs_march_kernel<F, G, R, kMarchWarps, true>
     : n_phi <= 4 ? cccs_march_kernel<F, G, R, 4, false>
                  : cccs_march_kernel<F, G, R, kMarchWarps, false>)<<<blocks, 32 * n_phi, 0, st>>>(
        d_beams, T, Rho, D, dirs, cp, split, planes, plane_stride, status, order);
    FD2_CHECK_CUDA(cudaGetLastError());
    return FD2_OK;
}

// Lateral reach of a batch's rays in voxels: what bounds the integers and the
// biased roundings of the voxel-stationary march.
struct Reach {
    double tan_x = 0, tan_y = 0;    // of the cone directions
    double slice = 0, total = 0;    // largest lateral advance per slice, and over a beam
    bool finite = true;
    Reach(const ConeAngles& a) {
        for (int t = 0; t < a.n_theta_fwd; t++)
            for (int f = 0; f < a.n_phi; f++) {
                const double r = std::fabs(std::tan((double)a.theta[t]));
                tan_x = std::max(tan_x, r * std::fabs(std::cos((double)a.phi[f])));
                tan_y = std::max(tan_y, r * std::fabs(std::sin((double)a.phi[f])));
            }
    }
    void add(const fd2_beam_t& b) {
        const double sx = std::fabs(b.long_spacing * tan_x / b.beamlet_size[0]),
                     sy = std::fabs(b.long_spacing * tan_y / b.beamlet_size[1]);
        if (!(sx < 1e30 && sy < 1e30)) finite = false;  // (NaN too)
        slice = std::max({slice, sx, sy});
        total = std::max(total, std::max(sx, sy) * b.long_dim);
    }
    // voxel indices fit 15 bits, and the 1e-4 slack of the slice rule moves a
    // ray sideways by a fraction of a voxel
    bool admits() const { return finite && slice < 500.0 && total < 15000.0; }
};

// The march for a batch.  map: the common map side F when every map of the
// batch is F x F, else 0; reach_ok: Reach::admits.  Common sides of 8, 12 and
// 16 take the voxel-stationary march (1..8 azimuth warps); other common sides
// up to 24 the half-table instance and up to 32 the shared-column instance
// (4..8 azimuth warps); anything else the general per-ray instance.
int launch_march(int map, bool reach_ok, int sm_count, int maxP, int n_phi, unsigned blocks, cudaStream_t st,
                 const fd2_beam_t* d_beams, const float* const* T, const float* const* R, float* const* D,
                 const float4* dirs, const ConeParams& cp, int split, float* planes, size_t plane_stride, DeviceStatus* status,
                 const int* order = nullptr) {
    const int threads = 32 * n_phi;
    const size_t shm = (size_t)(1 + n_phi) * maxP * sizeof(float2);
    const bool warps_ok = threads >= 128 && threads <= kMapThreads;
    if (reach_ok && n_phi <= kMarchWarps) {
        if (map == 16)
            return launch_voxel_march<16, 2, 8>(blocks, n_phi, st, d_beams, T, R, D, dirs, cp, split, planes,
                                                plane_stride, status, order, sm_count);
        if (map == 12)
            return launch_voxel_march<12, 2, 6>(blocks, n_phi, st, d_beams, T, R, D, dirs, cp, split, planes,
                                                plane_stride, status, order, sm_count);
        if (map == 8)
            return launch_voxel_march<8, 4, 2>(blocks, n_phi, st, d_beams, T, R, D, dirs, cp, split, planes,
                                               plane_stride, status, order, sm_count);
    }
    if (map > 0 && map <= 24 && warps_ok) {  // half-table instance: rays per lane = ceil(F^2 / 32)
        const int P = map * map;
        if (P <= 64)
            return launch_instance<2, false, true>(blocks, threads, shm, st, d_beams, T, R, D, dirs, cp, split,
                                                          planes, plane_stride, status, order);
        if (P <= 160)
            return launch_instance<5, false, true>(blocks, threads, shm, st, d_beams, T, R, D, dirs, cp, split,
                                                          planes, plane_stride, status, order);
        if (P <= 256)
            return launch_instance<8, false, true>(blocks, threads, shm, st, d_beams, T, R, D, dirs, cp, split,
                                                          planes, plane_stride, status, order);
        if (P <= 416)
            return launch_instance<13, false, true>(blocks, threads, shm, st, d_beams, T, R, D, dirs, cp,
                                                           split, planes, plane_stride, status, order);
        return launch_instance<18, false, true>(blocks, threads, shm, st, d_beams, T, R, D, dirs, cp, split,
                                                       planes, plane_stride, status, order);
    }
    if (map > 0 && map <= 32 && warps_ok)  // 25 to 32: one lane per column, up to 32 rows each
        return launch_instance<32, true>(blocks, threads, shm, st, d_beams, T, R, D, dirs, cp, split, planes,
                                         plane_stride, status, order);
    if (maxP <= 256)
        return launch_instance<8, false>(blocks, threads, shm, st, d_beams, T, R, D, dirs, cp, split, planes,
                                                plane_stride, status, order);
    return launch_instance<32, false>(blocks, threads, shm, st, d_beams, T, R, D, dirs, cp, split, planes,
                                             plane_stride, status, order);
}

// The spread march: 17 x 17 to 32 x 32 maps, where an azimuth's rays keep a warp
// busy for hundreds of instructions a step, in a batch under schedule 1 whose
// (beamlet, zenith bin) pairs leave SMs without a block.  A device (or a slice of
// one) that has no room for the clusters refuses the launch: *taken is false
// then, and the plain march gives the same dose.
template <int RPL, bool kCols, bool kTab, int kWpa>
int launch_spread(unsigned blocks, int cluster, int n_phi, size_t maxP, cudaStream_t st, const fd2_beam_t* d_beams,
                  const float* const* T, const float* const* R, float* const* D, const float4* dirs,
                  const ConeParams& cp, float* planes, size_t plane_stride, DeviceStatus* status, bool* taken) {
    const size_t shm = (size_t)(1 + n_phi / cluster) * maxP * sizeof(float2);
    FD2_CHECK_CUDA(cudaFuncSetAttribute(cccs_kernel<RPL, kCols, kTab, kWpa>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)shm));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks * cluster);
    cfg.blockDim = dim3(32 * kWpa * (n_phi / cluster));
    cfg.dynamicSmemBytes = shm;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    *taken = cudaLaunchKernelEx(&cfg, cccs_kernel<RPL, kCols, kTab, kWpa>, d_beams, T, R, D, dirs, cp, 1, planes,
                                plane_stride, status, (const int*)nullptr) == cudaSuccess;
    if (!*taken) cudaGetLastError();
    return FD2_OK;
}

// Blocks per cluster of the spread march: the azimuths are divided evenly and
// the clusters stay within two blocks an SM; 0 when it is not taken.  Blocks of 512
// threads run one an SM, the rest of two in a second wave: that stays the faster
// where a plain block has more rays a lane than registers for them (maps over 20:
// 24 x 24, 8 azimuths, 18 beams 2.9 / 4.7 ms), below only while the second wave is
// short (20 x 20, 0.3 cm: 13 beams 2.42 / 2.56 ms, 18 beams 2.79 / 2.55, 30 beams of
// 4 bins 1.87 / 1.46; 0.1 cm: 13 beams 5.98 / 7.06, 18 beams 6.2 / 7.05).
int spread_cluster(int map, int n_phi, unsigned blocks, int sm_count) {
    if (map < 17 || map > 32 || n_phi < 4 || n_phi > 8) return 0;
    for (int c : {kMaxCluster, 2}) {
        const unsigned quarters = map <= 20 && 32 * 4 * (n_phi / c) > 384 ? 6 : 8;  // blocks per 4 SMs
        if (n_phi % c == 0 && 4 * blocks * (unsigned)c <= quarters * (unsigned)sm_count) return c;
    }
    return 0;
}

// common map side of a batch (F when every map is F x F), else 0
int common_map(int side, const fd2_beam_t& b) {
    const int fx = (int)b.fmap_size[0], fy = (int)b.fmap_size[1];
    if (fx != fy) return 0;
    return side < 0 ? fx : (side == fx ? side : 0);
}

}  // namespace

// Forward zenith bins of a kernel and its azimuths.
static ConeAngles forward_angles(const fd2_cccs_kernel* k) {
    ConeAngles ang{};
    for (int t = 0; t < k->n_theta; t++)
        if ((double)k->theta[t] <= 1.5707963267948966) ang.theta[ang.n_theta_fwd++] = k->theta[t];  // DoseComp.cu:265
    ang.n_phi = k->n_phi;
    for (int f = 0; f < k->n_phi; f++) ang.phi[f] = k->phi[f];
    return ang;
}

// What of a batch selects its kernel beside the map's pixels and the cones.
struct BatchForm {
    int map = -1;        // common map side, else 0
    bool reach = false;  // Reach::admits
    int cluster = 0;     // spread_cluster under schedule 1
};
static BatchForm batch_form(const fd2_context* ctx, size_t n_beams, const fd2_beam_t* h_beams, const ConeAngles& ang) {
    BatchForm f;
    Reach reach(ang);
    for (size_t i = 0; i < n_beams; i++) {
        if (f.map != 0) f.map = common_map(f.map, h_beams[i]);
        reach.add(h_beams[i]);
    }
    f.reach = reach.admits();
    f.cluster = spread_cluster(f.map, ang.n_phi, (unsigned)(n_beams * ang.n_theta_fwd), ctx->sm_count);
    return f;
}

int cccs_form(const fd2_context* ctx, size_t n_beams, const fd2_beam_t* h_beams, const fd2_cccs_kernel* k) {
    const BatchForm f = batch_form(ctx, n_beams, h_beams, forward_angles(k));
    return f.cluster | (f.map > 0 ? 0 : 8) | (f.reach ? 0 : 16);
}

int launch_cccs_host(fd2_context* ctx, size_t n_beams, const fd2_beam_t* h_beams, const fd2_beam_t* d_beams,
                     const float* const* d_terma, const float* const* d_dens, float* const* d_dose,
                     const fd2_cccs_kernel* k, int schedule, cudaStream_t stream, const int* d_order) {
    if (n_beams == 0) return FD2_OK;
    ConeParams cp{};
    std::vector<int> fwd;
    for (int t = 0; t < k->n_theta; t++)
        if ((double)k->theta[t] <= 1.5707963267948966) fwd.push_back(t);  // forward only, DoseComp.cu:265
    if (fwd.empty()) return FD2_OK;
    cp.n_theta_fwd = (int)fwd.size();
    cp.n_phi = k->n_phi;
    for (size_t i = 0; i < fwd.size(); i++) {
        int t = fwd[i];
        cp.a[i] = k->a[t];
        cp.b[i] = k->b[t];
        cp.A_a[i] = k->A[t] / k->a[t];
        cp.B_b[i] = k->B[t] / k->b[t];
    }
    int maxP = 0, maxL = 0;
    for (size_t i = 0; i < n_beams; i++) {
        FD2_REQUIRE(h_beams[i].TermaBEV_pitch == h_beams[i].DensityBEV_pitch, FD2_ERR_INVALID_ARGUMENT,
                    "dose_compute: Terma and density pitches differ");
        maxP = std::max(maxP, (int)(h_beams[i].fmap_size[0] * h_beams[i].fmap_size[1]));
        maxL = std::max(maxL, (int)h_beams[i].long_dim);
    }
    FD2_REQUIRE(maxP > 0 && maxP <= 1024, FD2_ERR_INVALID_ARGUMENT, "dose_compute: fmap of %d pixels (1..1024)", maxP);
    // direction table [beam][theta_fwd][phi] as float4, evaluated on the device
    const ConeAngles ang = forward_angles(k);
    size_t dir_bytes = n_beams * fwd.size() * k->n_phi * sizeof(float4);
    size_t plane_stride = (size_t)maxP * maxL;
    size_t plane_bytes = schedule == 1 ? n_beams * fwd.size() * plane_stride * sizeof(float) : 0;
    void* scratch = nullptr;
    FD2_TRY(ctx_scratch(ctx, dir_bytes + plane_bytes + 256, stream, &scratch));
    float4* d_dirs = (float4*)scratch;
    float* d_planes = (float*)((char*)scratch + ((dir_bytes + 255) / 256) * 256);
    FD2_TRY(launch_cone_dirs(d_beams, n_beams, ang, d_dirs, stream));
    // slices a zenith pass skips must contribute zero
    if (plane_bytes) FD2_CHECK_CUDA(cudaMemsetAsync(d_planes, 0, plane_bytes, stream));
    const unsigned blocks = (unsigned)(schedule == 1 ? n_beams * fwd.size() : n_beams);
    const BatchForm form = batch_form(ctx, n_beams, h_beams, ang);
    const int map = form.map, cluster = schedule == 1 ? form.cluster : 0;
    bool taken = false;
    if (cluster && map <= 24)
        FD2_TRY((launch_spread<5, false, true, 4>(blocks, cluster, k->n_phi, maxP, stream, d_beams, d_terma, d_dens, d_dose,
                                                  d_dirs, cp, d_planes, plane_stride, ctx->d_status, &taken)));
    else if (cluster && k->n_phi / cluster <= 3)
        FD2_TRY((launch_spread<4, true, false, 8>(blocks, cluster, k->n_phi, maxP, stream, d_beams, d_terma, d_dens, d_dose,
                                                  d_dirs, cp, d_planes, plane_stride, ctx->d_status, &taken)));
    else if (cluster)
        FD2_TRY((launch_spread<8, true, false, 4>(blocks, cluster, k->n_phi, maxP, stream, d_beams, d_terma, d_dens, d_dose,
                                                  d_dirs, cp, d_planes, plane_stride, ctx->d_status, &taken)));
    if (!taken)
        FD2_TRY(launch_march(map, form.reach, ctx->sm_count, maxP, k->n_phi, blocks, stream, d_beams, d_terma, d_dens, d_dose, d_dirs, cp,
                             schedule, d_planes, plane_stride, ctx->d_status, schedule == 1 ? nullptr : d_order));
    ctx->launches += 2;  // direction table + march
    if (schedule == 1) {
        dim3 grid(std::max(1, std::min(64, (int)((plane_stride + 255) / 256))), (unsigned)n_beams);
        cccs_split_reduce<<<grid, 256, 0, stream>>>(d_beams, d_dose, d_planes, plane_stride, (int)fwd.size());
        FD2_CHECK_CUDA(cudaGetLastError());
        ctx->launches += 1;
    }
    return FD2_OK;
}

size_t cccs_scratch_bytes(size_t n_beams, const fd2_beam_t* h_beams, const fd2_cccs_kernel* k, int schedule) {
    size_t n_fwd = 0;
    for (int t = 0; t < k->n_theta; t++)
        if ((double)k->theta[t] <= 1.5707963267948966) n_fwd++;
    size_t maxP = 0, maxL = 0;
    for (size_t i = 0; i < n_beams; i++) {
        maxP = std::max(maxP, (size_t)h_beams[i].fmap_size[0] * h_beams[i].fmap_size[1]);
        maxL = std::max(maxL, (size_t)h_beams[i].long_dim);
    }
    const size_t dir_bytes = n_beams * n_fwd * k->n_phi * sizeof(float4);
    const size_t plane_bytes = schedule == 1 ? n_beams * n_fwd * maxP * maxL * sizeof(float) : 0;
    return dir_bytes + plane_bytes + 256;
}

void cccs_longest_first(size_t n_beams, const fd2_beam_t* h_beams, int* order) {
    std::vector<int> idx(n_beams);
    for (size_t i = 0; i < n_beams; i++) idx[i] = (int)i;
    std::stable_sort(idx.begin(), idx.end(),
                     [&](int a, int b) { return h_beams[a].long_dim > h_beams[b].long_dim; });
    std::copy(idx.begin(), idx.end(), order);
}

// Automatic schedule: split the zenith bins across blocks when the beamlets
// alone cannot fill the device (fewer than ~4 blocks per SM).
int cccs_auto_schedule(const fd2_context* ctx, size_t n_beams) {
    return n_beams < (size_t)ctx->sm_count * 4 ? 1 : 0;
}

}  // namespace fd2

extern "C" int fd2_dose_compute(fd2_context* ctx, size_t fmap_npixels, size_t n_beams, const fd2_beam_t* d_beams,
                                float* const* d_terma, float* const* d_density_bev, float* const* d_dose,
                                const fd2_cccs_kernel* kernel, void* stream) {
    FD2_REQUIRE(ctx && d_beams && d_terma && d_density_bev && d_dose && kernel, FD2_ERR_INVALID_ARGUMENT,
                "dose_compute: null argument");
    FD2_REQUIRE(fmap_npixels > 0 && fmap_npixels <= 1024, FD2_ERR_INVALID_ARGUMENT,
                "dose_compute: fmap_npixels %zu outside 1..1024", fmap_npixels);
    if (n_beams == 0) return FD2_OK;
    // the cone directions are evaluated on the host from the beam descriptors
    std::vector<fd2_beam_t> hb(n_beams);
    cudaStream_t st = (cudaStream_t)stream;
    FD2_CHECK_CUDA(cudaMemcpyAsync(hb.data(), d_beams, n_beams * sizeof(fd2_beam_t), cudaMemcpyDeviceToHost, st));
    FD2_CHECK_CUDA(cudaStreamSynchronize(st));
    return fd2::launch_cccs_host(ctx, n_beams, hb.data(), d_beams, (const float* const*)d_terma,
                                 (const float* const*)d_density_bev, d_dose, kernel,
                                 fd2::cccs_auto_schedule(ctx, n_beams), st, nullptr);
}

extern "C" int fd2_cccs_cone_directions(fd2_context* ctx, const fd2_cccs_kernel* k, size_t n_beams,
                                        const fd2_beam_t* h_beams, float* h_out, size_t n_out) {
    FD2_REQUIRE(ctx && k && h_beams && h_out, FD2_ERR_INVALID_ARGUMENT, "cone_directions: null argument");
    const fd2::ConeAngles ang = fd2::forward_angles(k);
    const size_t n = n_beams * ang.n_theta_fwd * ang.n_phi;
    FD2_REQUIRE(n_out >= 4 * n, FD2_ERR_CAPACITY, "cone_directions: need %zu floats", 4 * n);
    if (!n) return FD2_OK;
    fd2_beam_t* d_beams = nullptr;
    float4* d_out = nullptr;
    FD2_CHECK_CUDA(cudaMalloc(&d_beams, n_beams * sizeof(fd2_beam_t)));
    cudaError_t e = cudaMalloc(&d_out, n * sizeof(float4));
    if (e == cudaSuccess) e = cudaMemcpy(d_beams, h_beams, n_beams * sizeof(fd2_beam_t), cudaMemcpyHostToDevice);
    int rc = FD2_OK;
    if (e == cudaSuccess) rc = fd2::launch_cone_dirs(d_beams, n_beams, ang, d_out, ctx->stream);
    if (e == cudaSuccess && rc == FD2_OK) e = cudaStreamSynchronize(ctx->stream);
    if (e == cudaSuccess && rc == FD2_OK) e = cudaMemcpy(h_out, d_out, n * sizeof(float4), cudaMemcpyDeviceToHost);
    cudaFree(d_beams);
    if (d_out) cudaFree(d_out);
    if (rc) return rc;
    FD2_CHECK_CUDA(e);
    return FD2_OK;
}

// ---------------------------------------------------------------------------
// fd2_dose_compute_static: the CCCS march without any device allocation.
//
// fd2_dose_compute keeps its cone-direction table (and, for batches too small
// to fill the device, per-zenith planes) in the context's scratch buffer,
// which grows with cudaMalloc when a larger batch arrives.  Some hosts cannot
// allow that: a treatment-planning service that hands out every byte of device
// memory from its own pool sized at start-up, or a caller whose device memory
// is owned by another runtime that forbids foreign allocations once its pools
// are set.  Those callers get this entry point: no context, no cudaMalloc, no
// cudaFree, no allocating library.  What it needs beyond the caller's buffers
// -- the status word and the direction table -- lives in one fixed array in
// device global memory, defined below.  Its address belongs to the CUDA
// context that loaded this library's device code, so it is looked up with
// cudaGetSymbolAddress on the first call in each context (once per device
// under the runtime's primary context) and kept under that context's id.
//
// Limits: n_beams * n_forward_theta * n_phi * 16 bytes of directions must fit
// FD2_DOSE_STATIC_DIR_BYTES (256 KiB: 256 beams of an 8 x 8 cone kernel);
// larger batches are rejected with FD2_ERR_CAPACITY before any device work.
// Only schedule 0 runs (every zenith bin of a beamlet in one block, no
// planes), whose dose equals schedule 1's bit for bit.
//
// Every call shares the one array on its device: two calls whose work
// overlaps on the device (different streams, or different host threads with
// no ordering between them) overwrite each other's direction table and status
// word.  Serialise them (same stream, or synchronise in between).

// [0, 256): status word, cleared by every call before its launches (the only
// part that must start at zero); [256, 256 + FD2_DOSE_STATIC_DIR_BYTES):
// direction table [beam][theta_fwd][phi] as float4, fully rewritten by every call.
static __device__ __align__(256) unsigned char fd2_static_scratch[256 + FD2_DOSE_STATIC_DIR_BYTES];

namespace {

constexpr size_t kStaticStatusBytes = 256;  // fd2::DeviceStatus, padded to keep the table aligned
constexpr size_t kStaticDirBytes = FD2_DOSE_STATIC_DIR_BYTES;
constexpr size_t kBeamChunk = 32;  // beam descriptors read back per copy, on the host stack
static_assert(sizeof(fd2::DeviceStatus) <= kStaticStatusBytes, "status word outgrew its slot");

// Looked-up addresses, one per CUDA context.  A context is named by its
// driver-assigned id, which is never reused within a process: a second context
// on the same device, or the primary context recreated after cudaDeviceReset,
// gets a new id and so a fresh lookup (the module may load at another address).
struct StaticAddr {
    unsigned long long ctx_id;
    void* addr;
};
std::vector<StaticAddr> g_static_addr;
std::mutex g_static_mu;

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);
CtxGetCurrentFn g_ctx_get_current = nullptr;
CtxGetIdFn g_ctx_get_id = nullptr;
std::once_flag g_ctx_fns_once;

// The id of the context current on this thread; false when none is current
// yet or the driver does not offer the query.  The driver functions come
// through the runtime's entry-point table, so the library does not link the
// driver library itself.
bool current_context_id(unsigned long long* id) {
    std::call_once(g_ctx_fns_once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_ctx_get_current = (CtxGetCurrentFn)f;
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            g_ctx_get_id = (CtxGetIdFn)f;
    });
    if (!g_ctx_get_current || !g_ctx_get_id) return false;
    CUcontext c = nullptr;
    if (g_ctx_get_current(&c) != CUDA_SUCCESS || c == nullptr) return false;
    return g_ctx_get_id(c, id) == CUDA_SUCCESS;
}

// The device address of fd2_static_scratch in the current context.  Host
// code only sees a stand-in for the array's name, so the address is looked up
// with cudaGetSymbolAddress (which also makes the device's primary context
// current if none is) the first time a context calls, then reused.
int static_scratch_address(unsigned char** out) {
    unsigned long long id = 0;
    if (current_context_id(&id)) {
        std::lock_guard<std::mutex> lock(g_static_mu);
        for (const StaticAddr& s : g_static_addr)
            if (s.ctx_id == id) {
                *out = (unsigned char*)s.addr;
                return FD2_OK;
            }
    }
    void* p = nullptr;
    FD2_CHECK_CUDA(cudaGetSymbolAddress(&p, fd2_static_scratch));
    FD2_REQUIRE(p != nullptr && ((uintptr_t)p & 255) == 0, FD2_ERR_CUDA,
                "dose_compute_static: scratch address %p not 256-byte aligned", p);
    if (current_context_id(&id)) {
        std::lock_guard<std::mutex> lock(g_static_mu);
        g_static_addr.push_back({id, p});
    }
    *out = (unsigned char*)p;
    return FD2_OK;
}

}  // namespace

extern "C" int fd2_dose_compute_static(size_t fmap_npixels, size_t n_beams, const fd2_beam_t* d_beams,
                                       float* const* d_terma, float* const* d_density_bev, float* const* d_dose,
                                       const fd2_cccs_kernel* kernel, int* status_out, void* stream) {
    using namespace fd2;
    FD2_REQUIRE(d_beams && d_terma && d_density_bev && d_dose && kernel, FD2_ERR_INVALID_ARGUMENT,
                "dose_compute_static: null argument");
    FD2_REQUIRE(fmap_npixels > 0 && fmap_npixels <= 1024, FD2_ERR_INVALID_ARGUMENT,
                "dose_compute_static: fmap_npixels %zu outside 1..1024", fmap_npixels);
    if (n_beams == 0) return FD2_OK;
    const fd2_cccs_kernel* k = kernel;
    ConeParams cp{};
    ConeAngles ang{};
    for (int t = 0; t < k->n_theta; t++) {
        if ((double)k->theta[t] > 1.5707963267948966) continue;  // forward bins only, DoseComp.cu:265
        const int i = cp.n_theta_fwd++;
        cp.a[i] = k->a[t];
        cp.b[i] = k->b[t];
        cp.A_a[i] = k->A[t] / k->a[t];
        cp.B_b[i] = k->B[t] / k->b[t];
        ang.theta[i] = k->theta[t];
    }
    if (cp.n_theta_fwd == 0) return FD2_OK;
    cp.n_phi = ang.n_phi = k->n_phi;
    ang.n_theta_fwd = cp.n_theta_fwd;
    for (int f = 0; f < k->n_phi; f++) ang.phi[f] = k->phi[f];
    const size_t per_beam = (size_t)cp.n_theta_fwd * cp.n_phi * sizeof(float4);
    FD2_REQUIRE(n_beams <= kStaticDirBytes / per_beam, FD2_ERR_CAPACITY,
                "dose_compute_static: %zu beams x %d cones need %zu bytes of direction table; the fixed scratch "
                "holds %zu bytes (at most %zu beams of this kernel per call)",
                n_beams, cp.n_theta_fwd * cp.n_phi, n_beams * per_beam, kStaticDirBytes, kStaticDirBytes / per_beam);

    // map sizes of the batch, read back in chunks through a small stack buffer
    cudaStream_t st = (cudaStream_t)stream;
    fd2_beam_t hb[kBeamChunk];
    Reach reach(ang);
    int maxP = 0;
    int map = -1;
    for (size_t i0 = 0; i0 < n_beams; i0 += kBeamChunk) {
        const size_t m = std::min(kBeamChunk, n_beams - i0);
        FD2_CHECK_CUDA(cudaMemcpyAsync(hb, d_beams + i0, m * sizeof(fd2_beam_t), cudaMemcpyDeviceToHost, st));
        FD2_CHECK_CUDA(cudaStreamSynchronize(st));
        for (size_t i = 0; i < m; i++) {
            FD2_REQUIRE(hb[i].TermaBEV_pitch == hb[i].DensityBEV_pitch, FD2_ERR_INVALID_ARGUMENT,
                        "dose_compute_static: Terma and density pitches differ");
            maxP = std::max(maxP, (int)(hb[i].fmap_size[0] * hb[i].fmap_size[1]));
            map = map == 0 ? 0 : common_map(map, hb[i]);
            reach.add(hb[i]);
        }
    }
    FD2_REQUIRE(maxP > 0 && maxP <= 1024, FD2_ERR_INVALID_ARGUMENT,
                "dose_compute_static: fmap of %d pixels (1..1024)", maxP);

    int device = 0, sm_count = 0;
    FD2_CHECK_CUDA(cudaGetDevice(&device));
    FD2_CHECK_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
    unsigned char* base = nullptr;
    FD2_TRY(static_scratch_address(&base));
    DeviceStatus* d_status = (DeviceStatus*)base;
    float4* d_dirs = (float4*)(base + kStaticStatusBytes);
    FD2_CHECK_CUDA(cudaMemsetAsync(d_status, 0, sizeof(DeviceStatus), st));
    FD2_TRY(launch_cone_dirs(d_beams, n_beams, ang, d_dirs, st));
    const float* const* T = (const float* const*)d_terma;
    const float* const* R = (const float* const*)d_density_bev;
    FD2_TRY(launch_march(map, reach.admits(), sm_count, maxP, cp.n_phi, (unsigned)n_beams, st, d_beams, T, R, d_dose,
                         d_dirs, cp, 0, nullptr, 0, d_status));
    if (status_out)
        FD2_CHECK_CUDA(cudaMemcpyAsync(status_out, &d_status->code, sizeof(int), cudaMemcpyDefault, st));
    return FD2_OK;
}
