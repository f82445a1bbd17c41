// resample.cu -- BEV -> PVCS resampling: dense trilinear volumes and the
// per-beamlet sparse dose columns of the dose-loading matrix.
//
// Dense: d_BEV2PVCS (FastDoseLib/src/TermaComp.cu:124-150) and
// d_BEV2PVCS_SuperSampling (FastDoseLib/src/geom.cu:412-474).  Each voxel centre
// (or ss^3 sub-voxel sample) is rotated into the beam frame, projected onto the
// divergent BEV grid and sampled trilinearly (texel centres at i+0.5, zero
// outside), as the reference's linear/border texture does.
//
// Sparse columns: d_voxelInterp (IMRTOpt/src/IMRTgeom.cu:370-468).  A voxel within
// extent + half its diagonal of the beamlet axis takes the mean of ss^3 point
// samples of the beamlet's BEV dose; samples outside the fluence map laterally
// are skipped, samples outside [0, long_dim) in depth read zero.  The reference
// evaluates every (voxel, beamlet) pair of a beam into a dense
// [beamlets x voxels] matrix and then converts it with cusparseDenseToSparse;
// here each beamlet visits only the voxels of a conservative box around its
// frustum, tests them against a cheap bound, and emits its nonzeros straight
// into CSR order (voxel index ascending) with a block-wide scan.
#include <algorithm>
#include <cmath>

#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>

#include "fd2_internal.cuh"
#include "resample.cuh"

namespace fd2 {

namespace {

__device__ __forceinline__ float3 rot(const float* R, float3 v) {
    return make_float3(R[0] * v.x + R[1] * v.y + R[2] * v.z, R[3] * v.x + R[4] * v.y + R[5] * v.z,
                       R[6] * v.x + R[7] * v.y + R[8] * v.z);
}

__device__ __forceinline__ float bev_fetch(const float* __restrict__ bev, int fx, int fy, int L, int i, int j, int k) {
    if ((unsigned)i >= (unsigned)fx || (unsigned)j >= (unsigned)fy || (unsigned)k >= (unsigned)L) return 0.0f;
    return __ldg(bev + (size_t)i + (size_t)fx * ((size_t)j + (size_t)fy * k));
}

// The eight texels of cell (i, j, k), zero outside the grid.  A cell inside
// takes them without the tests of each.  Index: int where the grid's texels can
// be counted in it.
template <typename Index>
__device__ __forceinline__ void bev_cell(const float* __restrict__ bev, int fx, int fy, int L, int i, int j, int k,
                                         float (&t)[8]) {
    if ((unsigned)i < (unsigned)(fx - 1) && (unsigned)j < (unsigned)(fy - 1) && (unsigned)k < (unsigned)(L - 1)) {
        const Index p = (Index)i + (Index)fx * ((Index)j + (Index)fy * (Index)k), plane = (Index)fx * fy;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float* row = bev + (p + (q & 1 ? (Index)fx : 0) + (q & 2 ? plane : 0));
            t[2 * q] = __ldg(row);
            t[2 * q + 1] = __ldg(row + 1);
        }
    } else {
#pragma unroll
        for (int q = 0; q < 8; q++) t[q] = bev_fetch(bev, fx, fy, L, i + (q & 1), j + (q >> 1 & 1), k + (q >> 2));
    }
}

__device__ __forceinline__ float cell_blend(const float (&t)[8], float ax, float ay, float az) {
    float c00 = t[0] * (1 - ax) + t[1] * ax;
    float c10 = t[2] * (1 - ax) + t[3] * ax;
    float c01 = t[4] * (1 - ax) + t[5] * ax;
    float c11 = t[6] * (1 - ax) + t[7] * ax;
    return (c00 * (1 - ay) + c10 * ay) * (1 - az) + (c01 * (1 - ay) + c11 * ay) * az;
}

// Trilinear sample at (u, v, w), texel centres at i + 0.5, zero outside.
__device__ __forceinline__ float bev_trilinear(const float* __restrict__ bev, int fx, int fy, int L, float u, float v,
                                               float w) {
    const float xb = u - 0.5f, yb = v - 0.5f, zb = w - 0.5f;
    const float fi = floorf(xb), fj = floorf(yb), fk = floorf(zb);
    float t[8];
    bev_cell<size_t>(bev, fx, fy, L, (int)fi, (int)fj, (int)fk, t);
    return cell_blend(t, xb - fi, yb - fj, zb - fk);
}

// The same at cell coordinates (x, y, z) = (u, v, w) - 0.5 of any finite size:
// they are clamped just outside the grid, where all texels are zero, so that
// their floors are exact adds of 1.5 * 2^23 rounding down.
template <typename Index>
__device__ __forceinline__ float bev_trilinear_near(const float* __restrict__ bev, int fx, int fy, int L, float x, float y,
                                                    float z) {
    constexpr float kBias = 12582912.0f;
    x = fminf(fmaxf(x, -2.0f), fx + 1.0f);
    y = fminf(fmaxf(y, -2.0f), fy + 1.0f);
    z = fminf(fmaxf(z, -2.0f), L + 1.0f);
    const float bx = __fadd_rd(x, kBias), by = __fadd_rd(y, kBias), bz = __fadd_rd(z, kBias);
    float t[8];
    bev_cell<Index>(bev, fx, fy, L, __float_as_int(bx) - __float_as_int(kBias), __float_as_int(by) - __float_as_int(kBias),
             __float_as_int(bz) - __float_as_int(kBias), t);
    return cell_blend(t, x - (bx - kBias), y - (by - kBias), z - (bz - kBias));
}

// PVCS point -> normalised BEV coordinates (x lateral, y depth, z lateral).
__device__ __forceinline__ float3 to_bev_grid(const ColumnInfo& ci, float3 p) {
    float3 v = rot(ci.R, make_float3(p.x - ci.src[0], p.y - ci.src[1], p.z - ci.src[2]));
    float k = v.y * ci.inv_sad;
    return make_float3(v.x / (ci.bsx * k) + ci.hx, (v.y - ci.lim_min) * ci.inv_ls, v.z / (ci.bsy * k) + ci.hy);
}

// Dense volume: a warp takes 32 voxels of a row, a thread up to kDenseZ planes of
// them.  Most of the volume lies outside the beam, so the pass is bound by
// finding that out and writing zeros: a voxel more than half a texel off the map
// or the depths, where the trilinear sample is zero, is told by four comparisons
// without the two divisions (the margin of 0.01 texels is far more than they
// round).
// Fewer than kDenseZ planes where the volume would leave SMs without a block:
// 64 x 64 x 51 12.3 us with 8 planes, 8.2 with one.
constexpr int kDenseZ = 8;

__global__ void __launch_bounds__(256) bev2pvcs_kernel(ColumnInfo ci, const float* __restrict__ bev,
                                                       float* __restrict__ out, size_t pitch, int nx, int ny, int nz,
                                                       float vx, float vy, float vz, int planes) {
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    if (x >= nx || y >= ny) return;
    const float tx = (ci.hx + 0.51f) * fabsf(ci.bsx * ci.inv_sad), tz = (ci.hy + 0.51f) * fabsf(ci.bsy * ci.inv_sad);
    const float y0 = ci.lim_min - 0.51f * ci.ls, y1 = ci.lim_min + (ci.L + 0.51f) * ci.ls;
    for (int z0 = blockIdx.z * planes; z0 < nz; z0 += gridDim.z * planes)
#pragma unroll 4
        for (int z = z0; z < min(z0 + planes, nz); z++) {
            const float3 p = make_float3((x + 0.5f) * vx, (y + 0.5f) * vy, (z + 0.5f) * vz);
            const float3 v = rot(ci.R, make_float3(p.x - ci.src[0], p.y - ci.src[1], p.z - ci.src[2]));
            float val = 0.0f;
            if (fabsf(v.x) <= tx * fabsf(v.y) && fabsf(v.z) <= tz * fabsf(v.y) && v.y >= y0 && v.y <= y1) {
                const float3 cn = to_bev_grid(ci, p);
                val = bev_trilinear(bev, ci.fx, ci.fy, ci.L, cn.x, cn.z, cn.y);
            }
            out[(size_t)x + pitch * ((size_t)y + (size_t)ny * z)] = val;
        }
}

// Supersampled volume.  Only the voxels within `extent` of the beam axis that may
// touch the map and the BEV depths are sampled, about 0.5 % of a 200 x 200 x 160
// volume for 2 cm.  A voxel's place in the beam frame is formed in double, its
// samples' offsets from it in float.  Leaving out what lies beside the map matters
// where the extent is the larger: 200 x 200 x 160, 16 x 16 map of 0.25 cm, 5^3
// samples, 8 cm 517 -> 96 us, 60 cm 5300 -> 92 us.
struct SsFrame {
    float vx, vy, vz, extent;
    float mx, mz;      // lateral half width of the map per unit of depth, half a texel more (past which samples
                       // are zero) and its rounding
    float hv, slack;   // half diagonal of a voxel; allowance for rounding
    float sx, sz;      // texels per unit of lateral distance over depth
    SsFrame(const ColumnInfo& ci, const fd2_volume_t& v, float extent_)  // on the host, once a launch
        : vx(v.voxel_size[0]), vy(v.voxel_size[1]), vz(v.voxel_size[2]), extent(extent_) {
        mx = (ci.hx + 0.51f) * std::fabs(ci.bsx * ci.inv_sad);
        mz = (ci.hy + 0.51f) * std::fabs(ci.bsy * ci.inv_sad);
        hv = 0.5f * std::sqrt(vx * vx + vy * vy + vz * vz);
        slack = 1e-3f + 1e-4f * (4.0f * hv + std::fabs(extent));
        sx = 1.0f / (ci.bsx * ci.inv_sad);
        sz = 1.0f / (ci.bsy * ci.inv_sad);
    }
    __device__ __forceinline__ float3 at(const ColumnInfo& ci, float x, float y, float z) const {  // voxels -> beam frame
        return rot(ci.R, make_float3(x * vx - ci.src[0], y * vy - ci.src[1], z * vz - ci.src[2]));
    }
    // could a point within d of v lie on the map and the depths?
    __device__ __forceinline__ bool near_map(const ColumnInfo& ci, float3 v, float d) const {
        const float y = fabsf(v.y) + d;
        return !(fabsf(v.x) > mx * y + d) && !(fabsf(v.z) > mz * y + d) && !(v.y < ci.lim_min - ci.ls - d) &&
               !(v.y > ci.lim_min + (ci.L + 1) * ci.ls + d);
    }
    __device__ __forceinline__ bool sampled(const ColumnInfo& ci, int x, int y, int z) const {
        const float3 v = at(ci, x + 0.5f, y + 0.5f, z + 0.5f);
        return !(v.x * v.x + v.z * v.z > extent * extent) && near_map(ci, v, hv + slack);
    }
    // beam-frame offset of sample s of ss^3 from the voxel centre
    __device__ __forceinline__ float3 offset(const ColumnInfo& ci, int ss, int s) const {
        const float inv = 1.0f / ss;
        const int jk = (int)((s + 0.5f) * inv), k = (int)((jk + 0.5f) * inv);  // s / ss and s / ss^2, s <= 4096
        const float a = ((s - jk * ss + 0.5f) * inv - 0.5f) * vx, b = ((jk - k * ss + 0.5f) * inv - 0.5f) * vy,
                    c = ((k + 0.5f) * inv - 0.5f) * vz;
        return rot(ci.R, make_float3(a, b, c));
    }
};

// A voxel's centre in the beam frame, and the BEV dose at an offset from it.
struct SsVoxel {
    float cx, cy, cw, cz;  // cw: depth behind the first slice
    __device__ __forceinline__ SsVoxel(const ColumnInfo& ci, const SsFrame& f, int x, int y, int z) {
        const double px = (x + 0.5) * f.vx - ci.src[0], py = (y + 0.5) * f.vy - ci.src[1], pz = (z + 0.5) * f.vz - ci.src[2];
        cx = (float)(ci.R[0] * px + ci.R[1] * py + ci.R[2] * pz);
        const double dy = ci.R[3] * px + ci.R[4] * py + ci.R[5] * pz;
        cy = (float)dy;
        cw = (float)(dy - ci.lim_min);
        cz = (float)(ci.R[6] * px + ci.R[7] * py + ci.R[8] * pz);
    }
    template <typename Index>
    __device__ __forceinline__ float sample(const ColumnInfo& ci, const SsFrame& f, const float* __restrict__ bev,
                                            float3 o) const {
        const float uy = cy + o.y;
        float r = __fdividef(1.0f, uy);
        r = fmaf(r, fmaf(-uy, r, 1.0f), r);
        return bev_trilinear_near<Index>(bev, ci.fx, ci.fy, ci.L, fmaf((cx + o.x) * r, f.sx, ci.hx) - 0.5f,
                                         fmaf((cz + o.z) * r, f.sz, ci.hy) - 0.5f, fmaf(cw + o.y, ci.inv_ls, -0.5f));
    }
};

// Few samples a voxel: a thread takes a voxel.  A warp a voxel leaves most lanes
// idle up to 2^3 samples, and the listing below costs a small volume more than 3^3
// samples in turn.  2 cm, this form / the warps: 64 x 64 x 51, 1 sample 7 / 34 us,
// 2^3 11 / 35, 3^3 19 / 33; 200 x 200 x 160, 1 sample 23 / 36, 2^3 27 / 37; 3^3 from
// 2^19 voxels on is the warps' (100 x 100 x 80: 30 us, 200 x 200 x 160: 37).
template <typename Index>
__global__ void __launch_bounds__(256) bev2pvcs_ss_thread_kernel(ColumnInfo ci, const float* __restrict__ bev,
                                                                 float* __restrict__ out, size_t pitch, int nx, int ny,
                                                                 int nz, SsFrame f, int ss) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y,
              z = blockIdx.z * blockDim.z + threadIdx.z;
    if (x >= nx || y >= ny || z >= nz || !f.sampled(ci, x, y, z)) return;
    const SsVoxel c(ci, f, x, y, z);
    const float inv = 1.0f / ss;
    float acc = 0.0f;
    for (int k = 0; k < ss; k++)
        for (int j = 0; j < ss; j++)
#pragma unroll 3
            for (int i = 0; i < ss; i++)
                acc += c.sample<Index>(ci, f, bev, rot(ci.R, make_float3(((i + 0.5f) * inv - 0.5f) * f.vx,
                                                                         ((j + 0.5f) * inv - 0.5f) * f.vy,
                                                                         ((k + 0.5f) * inv - 0.5f) * f.vz)));
    if (!(acc < 1e-4f)) out[(size_t)x + pitch * ((size_t)y + (size_t)ny * z)] = acc / (float)(ss * ss * ss);
}

// More samples: the work is found first.  The volume is cut into tiles of
// 4 x 4 x 4 voxels, a block's first warp tests `per` tiles (32, fewer for small
// volumes, whose tiles would else lie with a few blocks), and the block lists a
// hit tile's voxels.  A warp then takes a voxel, its lanes the ss^3 samples: they
// fall into a few texel cells, so that a load touches two or three cache lines,
// where 32 voxels side by side touched up to sixteen and the pass was bound by
// their lookups.  2 cm, 5^3 samples, a thread a voxel / 32 tiles a block / as now:
// 200 x 200 x 160 111 / 56 / 56 us, 100 x 100 x 80 103 / 66 / 43, 64 x 64 x 51
// 58 / 58 / 50.
constexpr int kSsThreads = 256, kSsTile = 4, kSsTileVox = kSsTile * kSsTile * kSsTile;
constexpr int kSsRounds = 4;  // samples per lane whose offsets are kept in registers (ss <= 5)

template <typename Index>
__global__ void __launch_bounds__(kSsThreads, 3) bev2pvcs_ss_kernel(ColumnInfo ci, const float* __restrict__ bev,
                                                                 float* __restrict__ out, size_t pitch, int nx, int ny,
                                                                 int nz, SsFrame f, int ss, int per) {
    __shared__ int s_vox[kSsTileVox];
    __shared__ int3 s_tile[32];
    __shared__ unsigned s_hits;
    __shared__ int s_n;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tx = (nx + kSsTile - 1) / kSsTile, ty = (ny + kSsTile - 1) / kSsTile, tz = (nz + kSsTile - 1) / kSsTile;
    const long long tiles = (long long)tx * ty * tz, groups = (tiles + per - 1) / per;
    const int n_s = ss * ss * ss;
    float3 off[kSsRounds];
#pragma unroll
    for (int q = 0; q < kSsRounds; q++) off[q] = f.offset(ci, ss, lane + 32 * q);
    for (long long g = blockIdx.x; g < groups; g += gridDim.x) {
        if (warp == 0) {
            // neighbouring tiles go to different blocks: tile numbers times a prime
            // beyond their count
            const long long i = g * per + lane, tile = i * 2654435761LL % tiles;
            const int yz = (int)(tile / tx), x = ((int)(tile - (long long)yz * tx)) * kSsTile, z = yz / ty * kSsTile,
                      y = yz % ty * kSsTile;
            const float3 v = f.at(ci, x + 0.5f * kSsTile, y + 0.5f * kSsTile, z + 0.5f * kSsTile);
            const float ht = kSsTile * f.hv, r = fabsf(f.extent) + ht + f.slack;
            const unsigned hits = __ballot_sync(0xffffffffu, lane < per && i < tiles && !(v.x * v.x + v.z * v.z > r * r) &&
                                                                 f.near_map(ci, v, ht + f.slack));
            s_tile[lane] = make_int3(x, y, z);
            if (lane == 0) s_hits = hits;
        }
        __syncthreads();
        const unsigned hits = s_hits;
        for (unsigned m = hits; m; m &= m - 1) {
            const int3 t0 = s_tile[__ffs(m) - 1];
            if (threadIdx.x == 0) s_n = 0;
            __syncthreads();
            if (threadIdx.x < kSsTileVox) {
                const int q = threadIdx.x, x = t0.x + q % kSsTile, y = t0.y + q / kSsTile % kSsTile,
                          z = t0.z + q / (kSsTile * kSsTile);
                if (x < nx && y < ny && z < nz && f.sampled(ci, x, y, z))
                    s_vox[atomicAdd(&s_n, 1)] = q;  // any order: each voxel's sum is its own
            }
            __syncthreads();
            const int n = s_n;
            for (int w = warp; w < n; w += kSsThreads / 32) {
                const int q = s_vox[w];
                const int x = t0.x + q % kSsTile, y = t0.y + q / kSsTile % kSsTile, z = t0.z + q / (kSsTile * kSsTile);
                const SsVoxel c(ci, f, x, y, z);
                float acc = 0.0f;
#pragma unroll
                for (int k = 0; k < kSsRounds; k++)
                    if (lane + 32 * k < n_s) acc += c.sample<Index>(ci, f, bev, off[k]);
                for (int k = lane + 32 * kSsRounds; k < n_s; k += 32) acc += c.sample<Index>(ci, f, bev, f.offset(ci, ss, k));
#pragma unroll
                for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                if (lane == 0 && !(acc < 1e-4f))
                    out[(size_t)x + pitch * ((size_t)y + (size_t)ny * z)] = acc / (float)n_s;
            }
            __syncthreads();  // s_vox and s_n are used again
        }
        __syncthreads();  // s_tile and s_hits are used again
    }
}

// Conservative candidate test for a voxel centre c: could any point within
// hdiag of c carry a nonzero column value?
__device__ __forceinline__ bool candidate(const ColumnInfo& ci, float3 c, float hdiag, float extent) {
    float3 v = rot(ci.R, make_float3(c.x - ci.src[0], c.y - ci.src[1], c.z - ci.src[2]));
    const float slack = 1e-3f;
    if (sqrtf(v.x * v.x + v.z * v.z) > hdiag + extent + slack) return false;
    float ymax = v.y + hdiag + slack;
    if (ymax < ci.lim_min || v.y - hdiag - slack >= ci.lim_min + ci.L * ci.ls) return false;
    float k = ymax * ci.inv_sad;
    if (fabsf(v.x) - hdiag - slack > ci.hx * ci.bsx * k) return false;
    if (fabsf(v.z) - hdiag - slack > ci.hy * ci.bsy * k) return false;
    return true;
}

// Mean of ss^3 point samples (d_voxelInterp), or 0 when the voxel centre is
// farther than extent + hdiag from the beamlet axis.  Sample positions are
// affine in the sub-sample indices, so the beam-frame coordinates are stepped
// incrementally; one reciprocal of the depth per sample gives the divergent
// lateral scale.  SS > 0: ss == SS known at compile time, the innermost line
// of samples unrolled -- independent samples whose loads are predicated
// rather than branched around; SS == 0: any ss, consecutive samples that land
// in the same texel reuse it.  Both add the same values in the same order.
template <int SS>
__device__ __forceinline__ float column_value(const ColumnInfo& ci, const float* __restrict__ bev, int x, int y,
                                              int z, float3 vs, float hdiag, float extent, int ss_rt) {
    const int ss = SS > 0 ? SS : ss_rt;
    const float3 c = make_float3((x + 0.5f) * vs.x, (y + 0.5f) * vs.y, (z + 0.5f) * vs.z);
    const float3 v = rot(ci.R, make_float3(c.x - ci.src[0], c.y - ci.src[1], c.z - ci.src[2]));
    if (sqrtf(v.x * v.x + v.z * v.z) > hdiag + extent) return 0.0f;
    const float inv = 1.0f / ss;
    const float ffx = (float)ci.fx, ffy = (float)ci.fy;
    const float a = inv * vs.x, b = inv * vs.y, cz = inv * vs.z;
    const float3 dI = make_float3(ci.R[0] * a, ci.R[3] * a, ci.R[6] * a);
    const float3 dJ = make_float3(ci.R[1] * b, ci.R[4] * b, ci.R[7] * b);
    const float3 dK = make_float3(ci.R[2] * cz, ci.R[5] * cz, ci.R[8] * cz);
    const float3 p0 = make_float3((x + 0.5f * inv) * vs.x - ci.src[0], (y + 0.5f * inv) * vs.y - ci.src[1],
                                  (z + 0.5f * inv) * vs.z - ci.src[2]);
    const float3 u0 = rot(ci.R, p0);
    const float sx = 1.0f / (ci.bsx * ci.inv_sad), sz = 1.0f / (ci.bsy * ci.inv_sad);
    const int plane = ci.fx * ci.fy;
    int last = -1;
    float last_v = 0.0f, acc = 0.0f;
    for (int kk = 0; kk < ss; kk++) {
        const float3 uk = make_float3(u0.x + kk * dK.x, u0.y + kk * dK.y, u0.z + kk * dK.z);
        for (int jj = 0; jj < ss; jj++) {
            const float3 ukj = make_float3(uk.x + jj * dJ.x, uk.y + jj * dJ.y, uk.z + jj * dJ.z);
            if constexpr (SS > 0) {
#pragma unroll
                for (int ii = 0; ii < SS; ii++) {
                    const float ux = ukj.x + ii * dI.x, uy = ukj.y + ii * dI.y, uz = ukj.z + ii * dI.z;
                    const float r = __fdividef(1.0f, uy);
                    const float cnx = ux * r * sx + ci.hx, cnz = uz * r * sz + ci.hy;
                    const int tx = __float2int_rd(cnx), ty = __float2int_rd(cnz);
                    const int tz = __float2int_rd((uy - ci.lim_min) * ci.inv_ls);
                    const bool in = !(cnx < 0.0f || cnx > ffx || cnz < 0.0f || cnz > ffy) && tx < ci.fx &&
                                    ty < ci.fy && (unsigned)tz < (unsigned)ci.L;
                    if (in) acc += __ldg(bev + (tx + ci.fx * ty + plane * tz));
                }
            } else {
                for (int ii = 0; ii < ss; ii++) {
                    const float ux = ukj.x + ii * dI.x, uy = ukj.y + ii * dI.y, uz = ukj.z + ii * dI.z;
                    const float r = __fdividef(1.0f, uy);
                    const float cnx = ux * r * sx + ci.hx, cnz = uz * r * sz + ci.hy;
                    if (cnx < 0.0f || cnx > ffx || cnz < 0.0f || cnz > ffy) continue;
                    const int tx = __float2int_rd(cnx), ty = __float2int_rd(cnz);
                    const int tz = __float2int_rd((uy - ci.lim_min) * ci.inv_ls);
                    if (tx >= ci.fx || ty >= ci.fy || (unsigned)tz >= (unsigned)ci.L) continue;
                    const int idx = tx + ci.fx * ty + plane * tz;
                    if (idx != last) {
                        last = idx;
                        last_v = __ldg(bev + idx);
                    }
                    acc += last_v;
                }
            }
        }
    }
    return acc * (inv * inv * inv);
}

constexpr int kColThreads = 256;
constexpr int kPerThread = 4;
constexpr int kColChunk = kColThreads * kPerThread;

// Voxels of the row (y, z) of a beamlet's box that can be candidates: the
// candidate test requires the voxel centre within r0 = hdiag + extent + slack
// of the beamlet axis, and along a row the squared distance to the axis is a
// quadratic in x, so the admissible x form one interval.  It is solved in
// double and widened by one voxel on each side, so it contains every x the
// float test accepts; the exact test still runs on each voxel of it.
__device__ __forceinline__ void row_interval(const ColumnInfo& ci, int y, int z, float3 vs, float r0, int& xa,
                                             int& xb) {
    const double cx0 = 0.5 * vs.x - ci.src[0], cy = (y + 0.5) * vs.y - ci.src[1], cz = (z + 0.5) * vs.z - ci.src[2];
    const double A0 = ci.R[0] * cx0 + ci.R[1] * cy + ci.R[2] * cz, A1 = (double)ci.R[0] * vs.x;
    const double C0 = ci.R[6] * cx0 + ci.R[7] * cy + ci.R[8] * cz, C1 = (double)ci.R[6] * vs.x;
    const double a = A1 * A1 + C1 * C1, b = A0 * A1 + C0 * C1, c = A0 * A0 + C0 * C0 - (double)r0 * r0;
    xa = ci.box[0];
    xb = ci.box[3];
    if (a < 1e-12) {  // row parallel to the beamlet axis
        if (c > 1e-6 * r0 * r0) xb = xa;
        return;
    }
    const double disc = b * b - a * c;
    if (disc < 0.0) {
        xb = xa;
        return;
    }
    const double s = sqrt(disc);
    const double lo = (-b - s) / a, hi = (-b + s) / a;
    xa = max(xa, (int)floor(lo) - 1);
    xb = min(xb, (int)ceil(hi) + 2);
    if (xb < xa) xb = xa;
}

// Pass 1: number of candidate voxels of each beamlet (its row capacity).
__global__ void __launch_bounds__(kColThreads) column_count_kernel(const ColumnInfo* __restrict__ infos,
                                                                  uint32_t* __restrict__ counts, int nx, int ny,
                                                                  float3 vs, float hdiag, float extent) {
    const ColumnInfo ci = infos[blockIdx.x];
    const int by = ci.box[4] - ci.box[1], bz = ci.box[5] - ci.box[2];
    const int rows = by * bz;
    const float r0 = hdiag + extent + 2e-3f;
    uint32_t cnt = 0;
    for (int r = threadIdx.x; r < rows; r += kColThreads) {
        const int y = ci.box[1] + r % by, z = ci.box[2] + r / by;
        int xa, xb;
        row_interval(ci, y, z, vs, r0, xa, xb);
        for (int x = xa; x < xb; x++)
            cnt += candidate(ci, make_float3((x + 0.5f) * vs.x, (y + 0.5f) * vs.y, (z + 0.5f) * vs.z), hdiag, extent);
    }
    typedef cub::BlockReduce<uint32_t, kColThreads> Reduce;
    __shared__ typename Reduce::TempStorage tmp;
    uint32_t tot = Reduce(tmp).Sum(cnt);
    if (threadIdx.x == 0) counts[blockIdx.x] = tot;
    (void)nx; (void)ny;
}

// Pass 2: values of the candidates, nonzeros compacted in voxel order into
// the beamlet's temporary segment; writes the row's nnz and max |value|.
// Rows (y, z) of the box are taken kColThreads at a time in voxel order; their
// admissible x intervals are concatenated by a scan, and the concatenation is
// tested kColChunk voxels at a time with an order-preserving compaction.  The
// candidates gather in shared memory across chunks and row groups until at
// least kColChunk wait; then all threads compute their values (a few per
// thread, so the block barrier after them waits on a balanced share) and the
// nonzeros are compacted in order into the segment.
__global__ void __launch_bounds__(kColThreads) column_value_kernel(
    const ColumnInfo* __restrict__ infos, const float* const* __restrict__ dose, const uint64_t* __restrict__ cap_off,
    int32_t* __restrict__ tmp_col, float* __restrict__ tmp_val, uint32_t* __restrict__ row_nnz,
    float* __restrict__ row_max, int nx, int ny, float3 vs, float hdiag, float extent, int ss) {
    const ColumnInfo ci = infos[blockIdx.x];
    const float* __restrict__ bev = dose[blockIdx.x];
    const int by = ci.box[4] - ci.box[1], bz = ci.box[5] - ci.box[2];
    const int rows = by * bz;
    const float r0 = hdiag + extent + 2e-3f;
    const uint64_t base = cap_off[blockIdx.x];
    const uint64_t cap = cap_off[blockIdx.x + 1] - base;
    typedef cub::BlockScan<uint32_t, kColThreads> Scan;
    typedef cub::BlockReduce<float, kColThreads> RMax;
    __shared__ typename Scan::TempStorage scan_tmp;
    __shared__ typename RMax::TempStorage max_tmp;
    __shared__ uint32_t s_roff[kColThreads + 1];  // start of each row's interval in the concatenation
    __shared__ int s_rx[kColThreads];             // first x of the row's interval
    __shared__ int s_cand[2 * kColChunk];         // voxel index of the waiting candidates, in order
    __shared__ float s_val[2 * kColChunk];
    uint32_t written = 0;  // uniform across the block
    uint32_t pend = 0;     // candidates waiting in s_cand (uniform)
    float vmax = 0.0f;
    // values of the waiting candidates, then their nonzeros in order
    auto flush = [&]() {
        for (uint32_t k = threadIdx.x; k < pend; k += kColThreads) {
            const int v = s_cand[k];
            const int x = v % nx, y = (v / nx) % ny, z = v / (nx * ny);
            s_val[k] = ss == 5 ? column_value<5>(ci, bev, x, y, z, vs, hdiag, extent, ss)
                               : column_value<0>(ci, bev, x, y, z, vs, hdiag, extent, ss);
        }
        __syncthreads();
        const uint32_t per = (pend + kColThreads - 1) / kColThreads;  // a contiguous run per thread
        const uint32_t k0 = min(pend, threadIdx.x * per), k1 = min(pend, k0 + per);
        uint32_t nzc = 0;
        for (uint32_t k = k0; k < k1; k++) nzc += s_val[k] != 0.0f;
        uint32_t npos, n_nz;
        Scan(scan_tmp).ExclusiveSum(nzc, npos, n_nz);
        for (uint32_t k = k0; k < k1; k++) {
            if (s_val[k] != 0.0f) {
                if (written + npos < cap) {
                    tmp_col[base + written + npos] = s_cand[k];
                    tmp_val[base + written + npos] = s_val[k];
                }
                vmax = fmaxf(vmax, fabsf(s_val[k]));
                npos++;
            }
        }
        written += n_nz;
        pend = 0;
        __syncthreads();  // s_cand / s_val / scan_tmp reuse
    };
    for (int r0w = 0; r0w < rows; r0w += kColThreads) {
        const int r = r0w + threadIdx.x;
        int xa = 0, xb = 0;
        if (r < rows) row_interval(ci, ci.box[1] + r % by, ci.box[2] + r / by, vs, r0, xa, xb);
        uint32_t off, total;
        Scan(scan_tmp).ExclusiveSum((uint32_t)(xb - xa), off, total);
        s_roff[threadIdx.x] = off;
        s_rx[threadIdx.x] = xa;
        if (threadIdx.x == 0) s_roff[kColThreads] = total;
        __syncthreads();
        for (uint32_t f0 = 0; f0 < total; f0 += kColChunk) {
            // candidate test, kPerThread consecutive voxels per thread
            uint32_t flags = 0, cnt = 0;
            int vox[kPerThread];
#pragma unroll
            for (int q = 0; q < kPerThread; q++) {
                const uint32_t f = f0 + threadIdx.x * kPerThread + q;
                vox[q] = -1;
                if (f < total) {
                    int lo = 0, hi = kColThreads;  // last row whose start is <= f
                    while (hi - lo > 1) {
                        const int mid = (lo + hi) >> 1;
                        if (s_roff[mid] <= f) lo = mid; else hi = mid;
                    }
                    const int rr = r0w + lo;
                    const int x = s_rx[lo] + (int)(f - s_roff[lo]), y = ci.box[1] + rr % by, z = ci.box[2] + rr / by;
                    if (candidate(ci, make_float3((x + 0.5f) * vs.x, (y + 0.5f) * vs.y, (z + 0.5f) * vs.z), hdiag,
                                  extent)) {
                        flags |= 1u << q;
                        cnt++;
                        vox[q] = x + nx * (y + ny * z);
                    }
                }
            }
            uint32_t pos, n_cand;
            Scan(scan_tmp).ExclusiveSum(cnt, pos, n_cand);
#pragma unroll
            for (int q = 0; q < kPerThread; q++)  // pend < kColChunk and n_cand <= kColChunk
                if (flags & (1u << q)) s_cand[pend + pos++] = vox[q];
            pend += n_cand;
            __syncthreads();
            if (pend >= (uint32_t)kColChunk) flush();
        }
        __syncthreads();  // s_roff / s_rx reuse
    }
    if (pend) flush();
    float m = RMax(max_tmp).Reduce(vmax, cub::Max());
    if (threadIdx.x == 0) {
        row_nnz[blockIdx.x] = written;
        row_max[blockIdx.x] = m;
    }
}

template <typename VT>
__device__ __forceinline__ VT encode(float v, float inv_scale);
template <>
__device__ __forceinline__ float encode<float>(float v, float) { return v; }
template <>
__device__ __forceinline__ __half encode<__half>(float v, float s) { return __float2half_rn(v * s); }
template <>
__device__ __forceinline__ __nv_bfloat16 encode<__nv_bfloat16>(float v, float s) { return __float2bfloat16_rn(v * s); }

// Pass 3: copy each row's segment to its final CSR position.
template <typename VT>
__global__ void column_gather_kernel(const uint64_t* __restrict__ cap_off, const int64_t* __restrict__ row_off,
                                     const int32_t* __restrict__ tmp_col, const float* __restrict__ tmp_val,
                                     const float* __restrict__ inv_scale, int32_t* __restrict__ col,
                                     VT* __restrict__ val) {
    const int r = blockIdx.x;
    const uint64_t src = cap_off[r];
    const int64_t dst = row_off[r], n = row_off[r + 1] - row_off[r];
    const float s = inv_scale ? inv_scale[r] : 1.0f;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        col[dst + i] = tmp_col[src + i];
        val[dst + i] = encode<VT>(tmp_val[src + i], s);
    }
}

// Row offsets of a batch from its per-row nonzero counts, on the device:
// row_off[0] holds the batch's first offset; row_off[1..n] = row_off[0] +
// inclusive prefix sums.  For 16-bit values also the row scales (row maximum,
// 1 for an empty row) and their reciprocals.
__global__ void __launch_bounds__(1024) column_rows_kernel(const uint32_t* __restrict__ nnz,
                                                           const float* __restrict__ vmax, int64_t n,
                                                           int64_t* __restrict__ row_off, float* __restrict__ scale,
                                                           float* __restrict__ inv_scale) {
    typedef cub::BlockScan<int64_t, 1024> Scan;
    __shared__ typename Scan::TempStorage tmp;
    __shared__ int64_t s_carry;
    if (threadIdx.x == 0) s_carry = row_off[0];
    __syncthreads();
    for (int64_t i0 = 0; i0 < n; i0 += 1024) {
        const int64_t i = i0 + threadIdx.x;
        int64_t incl, total;
        Scan(tmp).InclusiveSum(i < n ? (int64_t)nnz[i] : 0, incl, total);
        if (i < n) {
            row_off[i + 1] = s_carry + incl;
            if (scale) {
                const float sc = vmax[i] > 0.0f ? vmax[i] : 1.0f;
                scale[i] = sc;
                inv_scale[i] = 1.0f / sc;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) s_carry += total;
        __syncthreads();
    }
}

}  // namespace

int launch_column_rows(size_t n, const uint32_t* d_nnz, const float* d_max, int64_t* d_row_off, float* d_scale,
                       float* d_inv_scale, cudaStream_t stream) {
    if (!n) return FD2_OK;
    column_rows_kernel<<<1, 1024, 0, stream>>>(d_nnz, d_max, (int64_t)n, d_row_off, d_scale, d_inv_scale);
    FD2_CHECK_CUDA(cudaGetLastError());
    return FD2_OK;
}

int launch_bev2pvcs(const ColumnInfo& ci, const fd2_volume_t& v, const float* d_bev, float* d_out, size_t pitch,
                    int ss, float extent, int sm_count, cudaStream_t stream) {
    if (ss <= 0) {
        dim3 block(32, 8), grid((v.dim[0] + 31) / 32, (v.dim[1] + 7) / 8);
        const uint64_t columns = (uint64_t)grid.x * grid.y, want = (uint64_t)sm_count * 8;
        const unsigned planes = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(kDenseZ, columns * v.dim[2] / want));
        grid.z = std::min((v.dim[2] + planes - 1) / planes, 65535u);
        bev2pvcs_kernel<<<grid, block, 0, stream>>>(ci, d_bev, d_out, pitch, v.dim[0], v.dim[1], v.dim[2],
                                                    v.voxel_size[0], v.voxel_size[1], v.voxel_size[2], (int)planes);
    } else {
        const bool small = (uint64_t)ci.fx * ci.fy * ci.L < (1ull << 30);
        const uint64_t voxels = (uint64_t)v.dim[0] * v.dim[1] * v.dim[2];
        const SsFrame f(ci, v, extent);
        if (ss <= 2 || (ss == 3 && voxels < (1u << 19))) {
            dim3 block(8, 8, 4), grid((v.dim[0] + 7) / 8, (v.dim[1] + 7) / 8, (v.dim[2] + 3) / 4);
            (small ? bev2pvcs_ss_thread_kernel<int> : bev2pvcs_ss_thread_kernel<size_t>)<<<grid, block, 0, stream>>>(
                ci, d_bev, d_out, pitch, v.dim[0], v.dim[1], v.dim[2], f, ss);
        } else {
            const uint64_t tiles = (uint64_t)((v.dim[0] + kSsTile - 1) / kSsTile) * ((v.dim[1] + kSsTile - 1) / kSsTile) *
                                   ((v.dim[2] + kSsTile - 1) / kSsTile);
            // a block takes its hit tiles in turn: where the launch is little more than
            // two waves, as many tiles as hold one hit, by the part of the volume that
            // the sampled cylinder and its rim fill
            const double rim = kSsTile * f.hv, ext = std::fabs(extent);
            const double side_x = 2 * (std::min(ext, (double)f.mx / ci.inv_sad) + rim),
                         side_z = 2 * (std::min(ext, (double)f.mz / ci.inv_sad) + rim);
            const double part = 0.8 * side_x * side_z * ((double)ci.L * ci.ls + 2 * rim) /
                                ((double)voxels * f.vx * f.vy * f.vz);
            int per = 32;
            while (per > 2 && tiles <= (uint64_t)per * 7 * sm_count && per * part > 1.0) per /= 2;
            const unsigned blocks = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((tiles + per - 1) / per, 1 << 20));
            (small ? bev2pvcs_ss_kernel<int> : bev2pvcs_ss_kernel<size_t>)<<<blocks, kSsThreads, 0, stream>>>(
                ci, d_bev, d_out, pitch, v.dim[0], v.dim[1], v.dim[2], f, ss, per);
        }
    }
    FD2_CHECK_CUDA(cudaGetLastError());
    return FD2_OK;
}

int launch_column_count(const ColumnInfo* d_infos, size_t n, uint32_t* d_counts, const fd2_volume_t& v, float extent,
                        cudaStream_t stream) {
    if (!n) return FD2_OK;
    float3 vs = make_float3(v.voxel_size[0], v.voxel_size[1], v.voxel_size[2]);
    float hdiag = 0.5f * sqrtf(vs.x * vs.x + vs.y * vs.y + vs.z * vs.z);
    column_count_kernel<<<(unsigned)n, kColThreads, 0, stream>>>(d_infos, d_counts, v.dim[0], v.dim[1], vs, hdiag,
                                                                 extent);
    FD2_CHECK_CUDA(cudaGetLastError());
    return FD2_OK;
}

int launch_column_values(const ColumnInfo* d_infos, size_t n, const float* const* d_dose, const uint64_t* d_cap_off,
                         int32_t* d_tmp_col, float* d_tmp_val, uint32_t* d_row_nnz, float* d_row_max,
                         const fd2_volume_t& v, float extent, int ss, cudaStream_t stream) {
    if (!n) return FD2_OK;
    float3 vs = make_float3(v.voxel_size[0], v.voxel_size[1], v.voxel_size[2]);
    float hdiag = 0.5f * sqrtf(vs.x * vs.x + vs.y * vs.y + vs.z * vs.z);
    column_value_kernel<<<(unsigned)n, kColThreads, 0, stream>>>(d_infos, d_dose, d_cap_off, d_tmp_col, d_tmp_val,
                                                                 d_row_nnz, d_row_max, v.dim[0], v.dim[1], vs, hdiag,
                                                                 extent, ss);
    FD2_CHECK_CUDA(cudaGetLastError());
    return FD2_OK;
}

int launch_column_gather(size_t n, const uint64_t* d_cap_off, const int64_t* d_row_off, const int32_t* d_tmp_col,
                         const float* d_tmp_val, const float* d_inv_scale, int32_t* d_col, void* d_val,
                         int value_type, cudaStream_t stream) {
    if (!n) return FD2_OK;
    if (value_type == FD2_VALUES_F16)
        column_gather_kernel<__half><<<(unsigned)n, 256, 0, stream>>>(d_cap_off, d_row_off, d_tmp_col, d_tmp_val,
                                                                      d_inv_scale, d_col, (__half*)d_val);
    else if (value_type == FD2_VALUES_BF16)
        column_gather_kernel<__nv_bfloat16><<<(unsigned)n, 256, 0, stream>>>(
            d_cap_off, d_row_off, d_tmp_col, d_tmp_val, d_inv_scale, d_col, (__nv_bfloat16*)d_val);
    else
        column_gather_kernel<float><<<(unsigned)n, 256, 0, stream>>>(d_cap_off, d_row_off, d_tmp_col, d_tmp_val,
                                                                     nullptr, d_col, (float*)d_val);
    FD2_CHECK_CUDA(cudaGetLastError());
    return FD2_OK;
}

}  // namespace fd2
