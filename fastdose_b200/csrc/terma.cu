// terma.cu -- polyenergetic Terma ray trace into beam's-eye-view (BEV) slabs.
//
// Restates d_TermaComputeCollective (FastDoseLib/src/TermaComp.cu:179-253): for
// every BEV pixel, a ray from the source through the pixel centre at the SAD
// plane is stepped long_spacing/4 along the central-axis projection; each
// sub-step samples the density trilinearly (texel centres at i+0.5, zero outside
// the volume), accumulates radiological path length, and adds
// sum_e fluence_e*E_e*mu_e*exp(-mu_e*rpl) / SXD^2.  Outputs are the slice means
// of Terma and density, [long_dim][pitch/4] per beam.
//
// B200 layout: one thread per (beam, pixel); the 256 pixels of a 16x16 beamlet
// map form one block, so every slice store is a fully coalesced 1 KB row.  The
// density volume is read through the read-only path (L1/L2); neighbouring rays
// touch neighbouring voxels.  Pixels with zero fluence skip the spectrum sum
// (their Terma is exactly zero in the reference too).
#include "fd2_internal.cuh"

namespace fd2 {

namespace {

constexpr int kSubSteps = 4;  // SUPER_SAMPLING, TermaComp.cu:65

__device__ __forceinline__ float fetch(const float* __restrict__ vol, int nx, int ny, int nz, int i, int j, int k) {
    if ((unsigned)i >= (unsigned)nx || (unsigned)j >= (unsigned)ny || (unsigned)k >= (unsigned)nz) return 0.0f;
    return __ldg(vol + (size_t)i + (size_t)nx * ((size_t)j + (size_t)ny * (size_t)k));
}

// a (1 - w) + b w with its one fused multiply-add spelled out, so that every
// instance of the kernel rounds alike: a beam's Terma does not depend on the batch.
__device__ __forceinline__ float mix(float a, float b, float w) {
    return __fmaf_rn(a, __fsub_rn(1.0f, w), __fmul_rn(b, w));
}

// Trilinear sample at unnormalised coordinates (u, v, w) in voxel units.  kAtOnce:
// all eight texels are read before the first is used, else the upper four follow
// the blend of the lower four.
template <bool kAtOnce>
__device__ __forceinline__ float trilinear(const float* __restrict__ vol, int nx, int ny, int nz, float u, float v,
                                           float w) {
    float xb = u - 0.5f, yb = v - 0.5f, zb = w - 0.5f;
    float fi = floorf(xb), fj = floorf(yb), fk = floorf(zb);
    float ax = xb - fi, ay = yb - fj, az = zb - fk;
    int i = (int)fi, j = (int)fj, k = (int)fk;
    const bool inside = (unsigned)i < (unsigned)(nx - 1) && (unsigned)j < (unsigned)(ny - 1) && (unsigned)k < (unsigned)(nz - 1);
    const float* p = vol + ((size_t)i + (size_t)nx * ((size_t)j + (size_t)ny * (size_t)k));  // read inside only
    const size_t plane = (size_t)nx * ny;
    float t[8];  // corner (q & 1, q >> 1 & 1, q >> 2)
    float c00, c10, c01, c11;
    auto read = [&](int q, const float* r) {  // inside: no test between the reads
        t[q] = __ldg(r);
        t[q + 1] = __ldg(r + 1);
        t[q + 2] = __ldg(r + nx);
        t[q + 3] = __ldg(r + nx + 1);
    };
    auto blend = [&](int q, float& low, float& high) {
        low = mix(t[q], t[q + 1], ax);
        high = mix(t[q + 2], t[q + 3], ax);
    };
    auto read_tested = [&]() {
#pragma unroll
        for (int q = 0; q < 8; q++) t[q] = fetch(vol, nx, ny, nz, i + (q & 1), j + (q >> 1 & 1), k + (q >> 2));
    };
    if constexpr (kAtOnce) {
        if (inside) {
            read(0, p);
            read(4, p + plane);
        } else {
            read_tested();
        }
        blend(0, c00, c10);
        blend(4, c01, c11);
    } else if (inside) {
        read(0, p);
        blend(0, c00, c10);
        read(4, p + plane);
        blend(4, c01, c11);
    } else {
        read_tested();
        blend(0, c00, c10);
        blend(4, c01, c11);
    }
    return mix(mix(c00, c10, ay), mix(c01, c11, ay), az);
}

// BEV -> PVCS rotation of v (inverse of the couch/gantry/collimator rotation).
__device__ __forceinline__ float3 bev_to_pvcs(float3 v, float th, float ph, float co) {
    float s, c;
    sincosf(-(ph + co), &s, &c);
    // about y by -(phi+coll)
    float3 t = make_float3(c * v.x + s * v.z, v.y, -s * v.x + c * v.z);
    // about the couch axis r = (sin(-phi), 0, cos(-phi)) by theta (Rodrigues)
    float sr, cr;
    sincosf(-ph, &sr, &cr);
    float st, ct;
    sincosf(th, &st, &ct);
    float k = (1.0f - ct) * (t.x * sr + t.z * cr);
    return make_float3(k * sr + ct * t.x + st * (-cr * t.y), k * 0.0f + ct * t.y + st * (cr * t.x - sr * t.z),
                       k * cr + ct * t.z + st * (sr * t.y));
}

// The ray trace waits on density reads.  kThreads 256, 40 registers, 6 blocks per
// SM: the extra warps hide more of that latency (32 registers spilled and was
// slower).  There the texels are read four at a time: eight at once spill at 40
// registers, and with 48 registers and 5 blocks they are slower on 16 x 16 maps.
// The stage, with the texels tested one by one / eight at once at 40 / at 48
// registers / four at a time at 40: 100 beams of 16 x 16 maps 16.9 / 14.2 / 12.9 /
// 12.4 ms; 24 beams of 20 x 20 (two blocks a map, the second half empty) 4.41 /
// 4.81 / 4.15 / 4.13 ms; 8 beams of 24 x 24 2.23 / 2.47 / 2.22 / 2.14 ms; 12 beams
// of 17 x 17 1.93 / 2.07 / 1.76 / 1.82 ms.
// kThreads 64, for launches of up to 24 blocks of 256 an SM: the rays spread over
// four times the blocks, which fill the SMs to the end, and without a register
// limit a slice's reads are in flight together.  One slab beam 140 -> 113 us, four
// 32 x 32 fields 408 -> 307 us (324 with four texels at a time); 1000 beams of 8 x 8
// maps 1.4 times as fast as with 256, 600 of 16 x 16 1.3 times, 2500 1.05.  Above
// that line the two are within 5 % of each other on repeated beams (3600 blocks of
// 20 x 20: 256 by 2 %, 4000 of 8 x 8: 64 by 5 %), but the 100-beam plan of 16 x 16
// maps takes 12.4 ms with 256 and 15.2 with 64.
template <bool kSkipDark, int kThreads>
__global__ void __launch_bounds__(kThreads, kThreads == 256 ? 6 : 4) terma_kernel(const fd2_beam_t* __restrict__ beams,
                                                    const float* const* __restrict__ fluence,
                                                    float* const* __restrict__ terma, float* const* __restrict__ dens,
                                                    const float* __restrict__ density, int nx, int ny, int nz,
                                                    float vx, float vy, float vz, SpectrumParams spec) {
    const int bi = blockIdx.x;
    const fd2_beam_t& b = beams[bi];
    const int fx = b.fmap_size[0], fy = b.fmap_size[1];
    const int p = blockIdx.y * blockDim.x + threadIdx.x;
    if (p >= fx * fy) return;
    const int ix = p % fx, iy = p / fx;
    const float fl = fluence[bi][p];
    const float sad = b.sad, ls = b.long_spacing;
    float3 pc = bev_to_pvcs(make_float3((ix + 0.5f - fx * 0.5f) * b.beamlet_size[0], sad,
                                        (iy + 0.5f - fy * 0.5f) * b.beamlet_size[1]),
                            b.angles[0], b.angles[1], b.angles[2]);
    const float k = ls / (sad * kSubSteps);
    const float3 st = make_float3(pc.x * k, pc.y * k, pc.z * k);
    const float stn = sqrtf(st.x * st.x + st.y * st.y + st.z * st.z);
    float sxd = b.lim_min / sad;
    float3 cn = make_float3((b.source[0] + pc.x * sxd) / vx, (b.source[1] + pc.y * sxd) / vy,
                            (b.source[2] + pc.z * sxd) / vz);
    const float3 sn = make_float3(st.x / vx, st.y / vy, st.z / vz);
    const size_t pitch = b.TermaBEV_pitch / sizeof(float);
    float* __restrict__ to = terma[bi];
    float* __restrict__ ro = dens[bi];
    const bool dark = kSkipDark && fl == 0.0f;
    float rpl = 0.0f;
    const uint32_t L = b.long_dim;
    for (uint32_t i = 0; i < L; i++) {
        float tavg = 0.0f, davg = 0.0f;
#pragma unroll
        for (int j = 0; j < kSubSteps; j++) {
            cn.x += sn.x;
            cn.y += sn.y;
            cn.z += sn.z;
            float d = trilinear<kThreads != 256>(density, nx, ny, nz, cn.x, cn.y, cn.z);
            rpl += d * stn;
            davg += d;
            sxd += k;
            if (!dark) {
                float tl = 0.0f;
                for (int e = 0; e < spec.n; e++) tl += spec.fluence_energy_mu[e] * fl * __expf(-spec.mu[e] * rpl);
                tavg += __fdividef(tl, sxd * sxd);
            }
        }
        to[p + pitch * i] = tavg * (1.0f / kSubSteps);
        ro[p + pitch * i] = davg * (1.0f / kSubSteps);
    }
}

}  // namespace

int launch_terma(fd2_context* ctx, size_t fmap_npixels, size_t n_beams, const fd2_beam_t* d_beams, const float* const* d_fluence,
                 float* const* d_terma, float* const* d_dens, const fd2_density* density,
                 const fd2_spectrum* spectrum, int fluence_skip, cudaStream_t stream) {
    (void)ctx;
    if (n_beams == 0) return FD2_OK;
    SpectrumParams sp;
    sp.n = spectrum->n;
    for (int e = 0; e < sp.n; e++) {
        sp.fluence_energy_mu[e] = spectrum->fluence[e] * spectrum->energy[e] * spectrum->mu[e];
        sp.mu[e] = spectrum->mu[e];
    }
    const fd2_volume_t& v = density->vol;
    // blocks per beam cover up to 1024 pixels (the reference's bound: one block per beam)
    const size_t blocks256 = n_beams * ((fmap_npixels + 255) / 256);
    const unsigned threads = blocks256 < 24 * (size_t)ctx->sm_count ? 64 : 256;
    dim3 grid((unsigned)n_beams, (unsigned)((fmap_npixels + threads - 1) / threads)), block(threads);
    auto kernel = threads == 64 ? (fluence_skip ? terma_kernel<true, 64> : terma_kernel<false, 64>)
                                : (fluence_skip ? terma_kernel<true, 256> : terma_kernel<false, 256>);
    kernel<<<grid, block, 0, stream>>>(d_beams, d_fluence, d_terma, d_dens, density->d_density, v.dim[0], v.dim[1],
                                       v.dim[2], v.voxel_size[0], v.voxel_size[1], v.voxel_size[2], sp);
    FD2_CHECK_CUDA(cudaGetLastError());
    if (ctx) ctx->launches += 1;
    return FD2_OK;
}

}  // namespace fd2

extern "C" int fd2_terma_compute(fd2_context* ctx, size_t fmap_npixels, size_t n_beams, const fd2_beam_t* d_beams,
                                 float* const* d_fluence, float* const* d_terma, float* const* d_density_bev,
                                 const fd2_density* density, const fd2_spectrum* spectrum, void* stream) {
    FD2_REQUIRE(ctx && d_beams && d_fluence && d_terma && d_density_bev && density && spectrum,
                FD2_ERR_INVALID_ARGUMENT, "terma_compute: null argument");
    FD2_REQUIRE(fmap_npixels > 0 && fmap_npixels <= 1024, FD2_ERR_INVALID_ARGUMENT,
                "terma_compute: fmap_npixels %zu outside 1..1024", fmap_npixels);
    return fd2::launch_terma(ctx, fmap_npixels, n_beams, d_beams, (const float* const*)d_fluence, d_terma, d_density_bev,
                             density, spectrum, 1, (cudaStream_t)stream);
}
