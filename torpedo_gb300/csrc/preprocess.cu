// preprocess.cu — kernel (a): per-Gaussian projection to a 48-byte Splat, the
// depth-sort input, and the tile-count exclusive scan (b, first half).
//
// Reference: project.slang:33-107 with splat/common.slang (SH, frustum test,
// camera position) and splat/volume.slang (ndc2pix, bounding rect, 3D
// covariance, EWA projection, Jacobian); prefix.slang:40-158 for the scan.
//
// GB300 layout: a CTA of 128 threads owns 128 consecutive records (30,720 B).
// The CTA stages them into shared memory with coalesced 16-byte asynchronous
// copies (cp.async, 15 per thread) while other CTAs of the SM project theirs;
// threads then read their record with conflict-free 16-byte loads (record
// stride 60 words). The copies complete
// by a hardware wait (cp.async.wait_group), not a software spin, so no wait
// can give up with a copy in flight, and the CTA drains every copy it issued
// before it exits. Besides the splat, each (view, Gaussian) gets a
// depth-sort key (view << 32 | bits(viewZ)) whose digit histograms are
// accumulated here. The tile counts are scanned afterwards in depth order
// (keygen.cu; scan_tiles_kernel is the standalone scan). Arithmetic
// follows the shader source left to right with matrix products accumulated
// k = 0..n-1; this file is compiled with --fmad=false so no product is fused
// into an add.
#include <algorithm>
#include <cstddef>

#include "tpd_common.cuh"
#include "tpd_kernels.h"
#include "tpd_scan.cuh"

namespace tpd {
namespace {

constexpr uint32_t kPreThreads = 128;

// SH constants (splat/common.slang:3-20).
__constant__ float cSH_C0 = 0.28209479177387814f;
__constant__ float cSH_C1 = 0.4886025119029199f;
__constant__ float cSH_C2[5] = {1.0925484305920792f, -1.0925484305920792f, 0.31539156525252005f,
                                -1.0925484305920792f, 0.5462742152960396f};
__constant__ float cSH_C3[7] = {-0.5900435899266435f, 2.890611442640554f, -0.4570457994644658f,
                                0.3731763325901154f, -0.4570457994644658f, 1.445305721320277f,
                                -0.5900435899266435f};

__device__ __forceinline__ void mat4mul(const float* A, const float* B, float* C) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            C[i * 4 + j] = A[i * 4 + 0] * B[0 * 4 + j] + A[i * 4 + 1] * B[1 * 4 + j] +
                           A[i * 4 + 2] * B[2 * 4 + j] + A[i * 4 + 3] * B[3 * 4 + j];
}

__device__ __forceinline__ void mat3mul(const float* A, const float* B, float* C) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            C[i * 3 + j] = A[i * 3 + 0] * B[0 * 3 + j] + A[i * 3 + 1] * B[1 * 3 + j] + A[i * 3 + 2] * B[2 * 3 + j];
}

__device__ __forceinline__ void mat3T(const float* A, float* B) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) B[j * 3 + i] = A[i * 3 + j];
}

// frame_begin: one CTA. Clears tickets / sort histograms, advances the tag and
// computes per-entity view*model and projview*model (the products of
// passFrustumClipping, common.slang:102,106, hoisted out of the per-Gaussian loop;
// identical values since they do not depend on the Gaussian).
__global__ void frame_begin_kernel(FrameCtl* ctl, const float* transforms, uint32_t n_ent, const ViewConst* views,
                                   uint32_t n_views, float* ent_mats) {
    pdl_trigger();  // the preprocess may be scheduled; it waits for this kernel
    const uint32_t t = threadIdx.x;
    for (uint32_t i = t; i < 32; i += blockDim.x) ctl->ticket[i] = 0;
    for (uint32_t i = t; i < 128; i += blockDim.x) ctl->tile_hist[i] = 0;
    for (uint32_t i = t; i < 32; i += blockDim.x) ctl->list_class[i] = 0;
    for (uint32_t i = t; i < 8 * 256; i += blockDim.x) {
        (&ctl->sort_hist[0][0])[i] = 0;
        (&ctl->depth_hist[0][0])[i] = 0;
    }
    if (t == 0) {
        ctl->tag = ctl->tag + 1;
        ctl->status = 0;
        ctl->total_keys = 0;
        ctl->total_strips = 0;
        ctl->visible = 0;
        ctl->depth_count = 0;
        ctl->depth_skips = 0;
    }
    if (!views || !ent_mats) return;
    for (uint32_t ve = t; ve < n_views * n_ent; ve += blockDim.x) {
        const uint32_t v = ve / n_ent, e = ve % n_ent;
        float M[16];
        if (transforms) {
            for (int k = 0; k < 16; ++k) M[k] = transforms[size_t(e) * 16 + k];
        } else {
            for (int k = 0; k < 16; ++k) M[k] = (k % 5) == 0 ? 1.0f : 0.0f;
        }
        float V[16], P[16], VM[16], PM[16];
        for (int k = 0; k < 16; ++k) { V[k] = views[v].view[k]; P[k] = views[v].projview[k]; }
        mat4mul(V, M, VM);
        mat4mul(P, M, PM);
        float* o = ent_mats + size_t(ve) * kEntityMatFloats;
        for (int k = 0; k < 12; ++k) o[k] = VM[k];
        for (int k = 0; k < 16; ++k) o[12 + k] = PM[k];
    }
}

// A record staged in shared memory, read 16 bytes at a time: at a stride of
// 60 words that is free of bank conflicts, a single word is not (lanes meet on
// eight banks, four each).
struct Rec {
    const float* p;
    __device__ __forceinline__ float4 f4(int q) const { return reinterpret_cast<const float4*>(p)[q]; }
};

__device__ __forceinline__ void unpack4(float4 f, float* to) {
    to[0] = f.x;
    to[1] = f.y;
    to[2] = f.z;
    to[3] = f.w;
}

// The constants of a view that project_one uses, in registers (four 16-byte loads).
struct ViewRegs {
    float view[12];  // rows 0..2 of the view matrix
    float focal[2];
    uint32_t width, height;
    __device__ __forceinline__ explicit ViewRegs(const ViewConst* v) {
        const float4* p = reinterpret_cast<const float4*>(v);
#pragma unroll
        for (int r = 0; r < 3; ++r) unpack4(__ldg(p + r), view + 4 * r);
        const float4 f = __ldg(p + 8);
        focal[0] = f.x;
        focal[1] = f.y;
        width = __float_as_uint(f.z);
        height = __float_as_uint(f.w);
    }
};
static_assert(offsetof(ViewConst, focal) == 128 && offsetof(ViewConst, width) == 136 && sizeof(ViewConst) % 16 == 0,
              "ViewRegs reads focal, width and height as 16 bytes");

// The 3D covariance of a Gaussian, which no view changes: computed at the
// first view that keeps the Gaussian. (It is symmetric to the bit: element
// (i, j) multiplies and adds the same factors in the same order as (j, i).)
struct Covariance {
    float c[6];
    bool known;
};

// project() for one Gaussian. Returns the tile count (0 when culled) and fills
// s.
__device__ __forceinline__ uint32_t project_one(const Rec& rec, const float* em, const ViewRegs& v,
                                                uint32_t deg, bool compat, Covariance& cov, Splat& s) {
    s = Splat{0.f, 0.f, 0.f, 0u, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const float4 pos_op = rec.f4(0);
    const float mean[3] = {pos_op.x, pos_op.y, pos_op.z};

    // passFrustumClipping (common.slang:98-119)
    float vp[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        vp[i] = em[i * 4 + 0] * mean[0] + em[i * 4 + 1] * mean[1] + em[i * 4 + 2] * mean[2] + em[i * 4 + 3] * 1.0f;
    if (vp[2] <= 0.0f) return 0;
    float cp[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        cp[i] = em[12 + i * 4 + 0] * mean[0] + em[12 + i * 4 + 1] * mean[1] + em[12 + i * 4 + 2] * mean[2] +
                em[12 + i * 4 + 3] * 1.0f;
    const float k13 = 1.3f;
    if (cp[0] < -k13 * cp[3] || cp[0] > k13 * cp[3]) return 0;
    if (cp[1] < -k13 * cp[3] || cp[1] > k13 * cp[3]) return 0;
    if (cp[2] < 0.0f || cp[2] > cp[3]) return 0;
    const float inv_w = 1.0f / cp[3];
    const float ndc_x = cp[0] * inv_w, ndc_y = cp[1] * inv_w;

    // focal = 0.5 * imageSize * focalNDC (project.slang:55)
    const float fx = (0.5f * float(v.width)) * v.focal[0];
    const float fy = (0.5f * float(v.height)) * v.focal[1];

    // computeCovariance (volume.slang:20-41)
    if (!cov.known) {
        const float4 q = rec.f4(1), sc = rec.f4(2);
        const float S[9] = {sc.x * sc.w, 0.f, 0.f, 0.f, sc.y * sc.w, 0.f, 0.f, 0.f, sc.z * sc.w};
        const float x = q.x, y = q.y, z = q.z, w = q.w;
        const float R[9] = {1.0f - 2.0f * (y * y + z * z), 2.0f * (x * y - w * z), 2.0f * (x * z + w * y),
                            2.0f * (x * y + w * z), 1.0f - 2.0f * (x * x + z * z), 2.0f * (y * z - w * x),
                            2.0f * (x * z - w * y), 2.0f * (y * z + w * x), 1.0f - 2.0f * (x * x + y * y)};
        float sigma[9], sigmaT[9], full[9];
        mat3mul(R, S, sigma);
        mat3T(sigma, sigmaT);
        mat3mul(sigma, sigmaT, full);
        cov.c[0] = full[0];
        cov.c[1] = full[1];
        cov.c[2] = full[2];
        cov.c[3] = full[4];
        cov.c[4] = full[5];
        cov.c[5] = full[8];
        cov.known = true;
    }
    const float cov3[9] = {cov.c[0], cov.c[1], cov.c[2], cov.c[1], cov.c[3], cov.c[4], cov.c[2], cov.c[4], cov.c[5]};

    // projectCovariance + computeJacobian (volume.slang:44-63)
    const float W3[9] = {v.view[0], v.view[1], v.view[2], v.view[4], v.view[5],
                         v.view[6], v.view[8], v.view[9], v.view[10]};
    const float f0 = fx / vp[2], f1 = fy / vp[2];
    const float t0 = vp[0] / vp[2], t1 = vp[1] / vp[2];
    const float J[9] = {f0, 0.f, -f0 * t0, 0.f, f1, -f1 * t1, 0.f, 0.f, 0.f};
    float Tm[9], TmT[9], inner[9], cov2[9];
    mat3mul(J, W3, Tm);
    mat3T(Tm, TmT);
    mat3mul(cov3, TmT, inner);
    mat3mul(Tm, inner, cov2);

    // low-pass filter and inverse (project.slang:60-66)
    const float ca = cov2[0] + 0.3f, cb = cov2[3], cc = cov2[4] + 0.3f;
    const float det = ca * cc - cb * cb;
    if (det == 0.0f) return 0;
    const float det_inv = 1.0f / det;
    const float conic0 = cc * det_inv, conic1 = -cb * det_inv, conic2 = ca * det_inv;

    // screen-space extent (project.slang:69-72)
    const float mid = 0.5f * (ca + cc);
    const float l1 = mid + sqrtf(fmaxf(0.1f, mid * mid - det));
    const float l2 = mid - sqrtf(fmaxf(0.1f, mid * mid - det));
    const float radius = ceilf(3.0f * sqrtf(fmaxf(l1, l2)));

    // ndc2pix (volume.slang:3-8) and getBoundingRect
    const float px = ((ndc_x + 1.0f) * float(v.width) - 1.0f) * 0.5f;
    const float py = ((ndc_y + 1.0f) * float(v.height) - 1.0f) * 0.5f;
    uint32_t x0, y0, x1, y1;
    bounding_rect(px, py, radius, grid_x(v.width), grid_y(v.height), x0, y0, x1, y1);
    const uint32_t touched = (x1 - x0) * (y1 - y0);
    if (touched == 0) return 0;

    // camera position (common.slang:88-92) and view direction from the pre-model mean
    float campos[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        campos[i] = -(v.view[0 * 4 + i] * v.view[0 * 4 + 3] + v.view[1 * 4 + i] * v.view[1 * 4 + 3] +
                      v.view[2 * 4 + i] * v.view[2 * 4 + 3]);
    const float d0 = mean[0] - campos[0], d1 = mean[1] - campos[1], d2 = mean[2] - campos[2];
    const float len = sqrtf(d0 * d0 + d1 * d1 + d2 * d2);
    const float dx = d0 / len, dy = d1 / len, dz = d2 / len;

    // evaluateSphericalHarmonics (common.slang:35-80)
    // the basis first, then a channel at a time, so that one channel's
    // coefficients are in registers
    float B[16], s12 = 0.f;
    if (deg > 0) {
        B[1] = cSH_C1 * dy;
        B[2] = cSH_C1 * dz;
        B[3] = cSH_C1 * dx;
        if (deg > 1) {
            const float xx = dx * dx, yy = dy * dy, zz = dz * dz, xy = dx * dy, yz = dy * dz, zx = dz * dx;
            B[4] = cSH_C2[0] * xy;
            B[5] = cSH_C2[1] * yz;
            B[6] = cSH_C2[2] * (2.0f * zz - xx - yy);
            B[7] = cSH_C2[3] * zx;
            B[8] = cSH_C2[4] * (xx - yy);
            if (deg > 2) {
                B[9] = (cSH_C3[0] * dy) * (3.0f * xx - yy);
                B[10] = (cSH_C3[1] * xy) * dz;
                B[11] = (cSH_C3[2] * dy) * (4.0f * zz - xx - yy);
                s12 = (cSH_C3[3] * dz) * (2.0f * zz - 3.0f * xx - 3.0f * yy);
                B[13] = (cSH_C3[4] * dx) * (4.0f * zz - xx - yy);
                B[14] = (cSH_C3[5] * dz) * (xx - yy);
                B[15] = (cSH_C3[6] * dx) * (xx - 3.0f * yy);
            }
        }
    }
    float res[3], dc[4];
    unpack4(rec.f4(3), dc);  // words 12..15: the three DC terms, the first channel's first coefficient
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        // the channel's 15 coefficients: words 15 + 15 c .. 29 + 15 c
        constexpr int kFirst[3] = {3, 7, 11};  // the 16-byte piece holding the first of them
        const int skip = 15 + 15 * c - 4 * kFirst[c];
        float f[20] = {};
        auto F = [&](int idx) { return f[skip + idx - 1]; };
        float r = cSH_C0 * dc[c];
        if (deg > 0) {
            unpack4(rec.f4(kFirst[c]), f);
            unpack4(rec.f4(kFirst[c] + 1), f + 4);
            r = r - B[1] * F(1) + B[2] * F(2) - B[3] * F(3);
            if (deg > 1) {
                unpack4(rec.f4(kFirst[c] + 2), f + 8);
                unpack4(rec.f4(kFirst[c] + 3), f + 12);
                r = r + B[4] * F(4) + B[5] * F(5) + B[6] * F(6) + B[7] * F(7) + B[8] * F(8);
                if (deg > 2) {
                    if (c < 2) unpack4(rec.f4(kFirst[c] + 4), f + 16);
                    r = r + B[9] * F(9) + B[10] * F(10) + B[11] * F(11);
                    if (compat) r = r + s12 + F(12);  // common.slang:69 as written
                    else r = r + s12 * F(12);
                    r = r + B[13] * F(13) + B[14] * F(14) + B[15] * F(15);
                }
            }
        }
        res[c] = r;
    }

    s.r = fmaxf(res[0] + 0.5f, 0.0f);
    s.g = fmaxf(res[1] + 0.5f, 0.0f);
    s.b = fmaxf(res[2] + 0.5f, 0.0f);
    s.tiles = touched;
    s.px = px;
    s.py = py;
    s.depth = vp[2];
    s.radius = radius;
    s.cx = conic0;
    s.cy = conic1;
    s.cz = conic2;
    s.opacity = pos_op.w;
    return touched;
}

// Persistent CTAs over chunks of kPreThreads records, kCtas of them per SM:
// while some project, the records of others stream in (asynchronous 16-byte
// copies; one stage per CTA, since two stages at three CTAs hold no more bytes
// in flight but fewer warps). One view is bound by the record stream and the
// splat stores, and four CTAs are enough (1M Gaussians 69 us, six 76); with
// several views per record the projection's latency counts and six, the most
// that shared memory holds, are faster (500,000 x 8 views 137 us, four 156;
// 1.5M x 8 views of which few see a Gaussian 350 against 392).
constexpr uint32_t kDepthPassesMax = 5;  // depth keys: 32 bits + log2(256 views)

struct PreSmem {
    float rec[kPreThreads * kRecordFloats];              // 30,720 B
    uint32_t hist[kDepthPassesMax][256];                  // depth-key digit counts of this CTA
    uint32_t kept;                                        // depth keys of visible items in this CTA
};

template <int kCtas>
__global__ void __launch_bounds__(kPreThreads, kCtas) preprocess_kernel(PreprocessArgs a) {
    extern __shared__ __align__(128) unsigned char pre_smem[];
    PreSmem& S = *reinterpret_cast<PreSmem*>(pre_smem);

    const uint32_t tid = threadIdx.x;
    for (uint32_t k = tid; k < kDepthPassesMax * 256; k += kPreThreads) (&S.hist[0][0])[k] = 0;
    // launched as a dependent of frame_begin_kernel (the frame's control block).
    // No early trigger: the depth sort's first pass is one wave of CTAs, which
    // must be placed on empty SMs, not onto the first ones this grid frees
    pdl_wait();
    if (tid == 0) S.kept = 0;
    uint32_t kept = 0;  // this thread's visible items (the depth sort drops the others)
    const uint32_t nchunks = (a.n + kPreThreads - 1) / kPreThreads;
    const uint32_t npass = min(kDepthPassesMax, (a.depth_key_bits + 7) / 8);
    // chunk's records into shared memory: piece q (16 bytes) by thread q % 128, so a
    // warp's copies are 512 consecutive bytes; a record is 15 whole pieces
    auto issue = [&](uint32_t chunk) {
        const uint32_t base = chunk * kPreThreads;
        const uint32_t pieces = min(kPreThreads, a.n - base) * (kRecordBytes / 16u);
        const char* src = reinterpret_cast<const char*>(a.recs + size_t(base) * kRecordFloats);
        char* dst = reinterpret_cast<char*>(S.rec);
        for (uint32_t q = tid; q < pieces; q += kPreThreads) cp_async16(dst + 16u * q, src + 16u * q);
    };
    for (uint32_t chunk = blockIdx.x; chunk < nchunks; chunk += gridDim.x) {
        issue(chunk);
        cp_async_commit();
        cp_async_wait_all();  // this thread's pieces of the chunk have landed
        __syncthreads();      // and every other thread's

        const uint32_t base = chunk * kPreThreads;
        const uint32_t cnt = min(kPreThreads, a.n - base);
        const uint32_t i = base + tid;
        const uint32_t e = (tid < cnt && a.ent_idx) ? a.ent_idx[i] : 0u;
        Covariance cov;
        cov.known = false;
        for (uint32_t v = 0; v < a.n_views; ++v) {
            Splat sp;
            uint32_t tiles = 0;
            if (tid < cnt) {
                const float* em = a.ent_mats + (size_t(v) * a.n_ent + e) * kEntityMatFloats;
                float emr[kEntityMatFloats];
#pragma unroll
                for (int k = 0; k < kEntityMatFloats / 4; ++k)
                    unpack4(__ldg(reinterpret_cast<const float4*>(em) + k), emr + 4 * k);
                tiles = project_one(Rec{S.rec + tid * kRecordFloats}, emr, ViewRegs(a.views + v), a.sh_degree,
                                    a.band3_compat != 0, cov, sp);
            } else {
                sp = Splat{0.f, 0.f, 0.f, 0u, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            }
            if (tid < cnt) {
                const size_t item = size_t(v) * a.n + i;
                float4* dst = reinterpret_cast<float4*>(a.splats + item);
                const float4* src = reinterpret_cast<const float4*>(&sp);
                dst[0] = src[0];
                dst[1] = src[1];
                dst[2] = src[2];
                if (a.depth_keys) {
                    // culled: low 32 bits 0xFFFFFFFF, dropped by the depth sort's first pass
                    const uint64_t key = (uint64_t(v) << 32) | (tiles ? __float_as_uint(sp.depth) : 0xFFFFFFFFu);
                    a.depth_keys[item] = key;
                    a.depth_items[item] = uint32_t(item);
                    if (tiles) {
                        ++kept;
                        for (uint32_t p = 0; p < npass; ++p) {
                            const uint32_t bits = min(8u, a.depth_key_bits - 8 * p);
                            atomicAdd(&S.hist[p][uint32_t(key >> (8 * p)) & ((1u << bits) - 1u)], 1u);
                        }
                    }
                }
            }
        }
        __syncthreads();  // every thread is done with the records before they are replaced
    }
    if (!a.depth_keys) return;
    kept = warp_sum(kept);
    if ((tid & 31u) == 0 && kept) atomicAdd(&S.kept, kept);
    __syncthreads();
    if (tid == 0 && S.kept) atomicAdd(&a.ctl->depth_count, S.kept);
    for (uint32_t p = 0; p < npass; ++p)
        for (uint32_t d = tid; d < 256; d += kPreThreads)
            if (S.hist[p][d]) atomicAdd(&a.ctl->depth_hist[p][d], S.hist[p][d]);
}

// Exclusive scan of Splat.tiles (prefix.slang:40-158) over partitions of 256
// threads x kScanItems items taken by atomic ticket, a warp's items in chunks
// of 32, one per lane (a splat is 48 bytes, so a chunk's counts lie in 12 lines;
// four consecutive items per lane touched four times as many, 18 us for 1M
// splats). 16 items per lane take 8 us (36 MB of sectors and offsets, 5 at copy
// speed), 8 items 11, 4 items 13: fewer partitions shorten the look-back's
// chain. Total -> *total. (The frame scans its counts in depth order,
// scan_items_kernel.)
constexpr uint32_t kScanThreads = 256;
constexpr uint32_t kScanItems = 16;
static_assert(kScanThreads * kScanItems == kScanTilesPart, "the descriptors are counted for these partitions");

// Clears what the scan starts from: the look-back descriptors, the ticket,
// the status and the total (of no splats).
__global__ void scan_begin_kernel(uint64_t* desc, uint32_t entries, FrameCtl* ctl, uint32_t* status, uint32_t* total) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < entries) desc[i] = 0;
    if (i == 0) {
        ctl->ticket[kTicketScan] = 0;
        ctl->tag = 0;
        *status = 0;
        *total = 0;
    }
}

__global__ void __launch_bounds__(kScanThreads)
    scan_tiles_kernel(const Splat* splats, uint32_t n, uint32_t* offsets, uint64_t* desc, FrameCtl* ctl,
                      uint32_t* status, uint32_t* total_out, uint32_t spin_limit, uint32_t never_publish) {
    constexpr uint32_t kScanTile = kScanTilesPart;
    constexpr uint32_t kTag = 1;  // (a cleared descriptor has tag 0)
    __shared__ uint32_t s_part, s_excl;
    __shared__ uint32_t s_warp[kScanThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    pdl_wait();  // launched as a dependent of scan_begin_kernel
    if (tid == 0) s_part = atomicAdd(&ctl->ticket[kTicketScan], 1u);
    __syncthreads();
    const uint32_t part = s_part;
    const uint64_t base = uint64_t(part) * kScanTile + warp * (32u * kScanItems) + lane;
    if (uint64_t(part) * kScanTile >= n) return;  // (uniform) past the items; nothing waits on it
    uint32_t v[kScanItems], incl[kScanItems], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < kScanItems; ++k) v[k] = base + 32u * k < n ? splats[base + 32u * k].tiles : 0u;
#pragma unroll
    for (uint32_t k = 0; k < kScanItems; ++k) {
        incl[k] = sum + warp_inclusive_scan(v[k]);
        sum = __shfl_sync(0xFFFFFFFFu, incl[k], 31);
    }
    if (lane == 0) s_warp[warp] = sum;
    __syncthreads();
    uint32_t wbase = 0, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < kScanThreads / 32; ++w) {
        const uint32_t sw = s_warp[w];
        if (w < warp) wbase += sw;
        total += sw;
    }
    if (warp == 0) {
        const uint32_t ex = warp_lookback(desc, part, total, kTag, status, spin_limit, never_publish != 0);
        if (lane == 0) {
            s_excl = ex;
            if (part == (n - 1u) / kScanTile) *total_out = ex + total;
        }
    }
    __syncthreads();
    const uint32_t first = s_excl + wbase;
#pragma unroll
    for (uint32_t k = 0; k < kScanItems; ++k)
        if (base + 32u * k < n) offsets[base + 32u * k] = first + incl[k] - v[k];
}

// Raw parameters -> records (activation as in GaussianGeometry.cpp:112-115:
// sigmoid opacity, exp scale, modifier 1; the quaternion is copied as given).
// One thread per 16 bytes of a record (15 of them), so the records are written
// and the 192 bytes of SH read coalesced; a thread per record took 106 us for
// 200,000 records, this 23 (96 MB in and out, 14 us at copy speed). kVec: quats and sh are 16-byte aligned.
template <bool kVec>
__global__ void __launch_bounds__(256)
    pack_records_kernel(const float* __restrict__ means, const float* __restrict__ log_scales,
                        const float* __restrict__ quats, const float* __restrict__ logits,
                        const float* __restrict__ sh, uint32_t n, float* __restrict__ recs) {
    constexpr uint32_t kPieces = kRecordFloats / 4;
    const uint64_t t = uint64_t(blockIdx.x) * 256u + threadIdx.x;
    if (t >= uint64_t(n) * kPieces) return;
    const size_t i = t / kPieces;
    const uint32_t q = uint32_t(t - uint64_t(i) * kPieces);
    auto four = [](const float* p) {
        return kVec ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(p[0], p[1], p[2], p[3]);
    };
    float4 v;
    if (q == 0)
        v = make_float4(means[i * 3 + 0], means[i * 3 + 1], means[i * 3 + 2], 1.0f / (1.0f + expf(-logits[i])));
    else if (q == 1)
        v = four(quats + i * 4);
    else if (q == 2)
        v = make_float4(expf(log_scales[i * 3 + 0]), expf(log_scales[i * 3 + 1]), expf(log_scales[i * 3 + 2]), 1.0f);
    else
        v = four(sh + i * 48 + (q - 3u) * 4u);
    reinterpret_cast<float4*>(recs)[t] = v;
}

}  // namespace

void launch_frame_begin(FrameCtl* ctl, const float* transforms, uint32_t n_ent, const ViewConst* views,
                        uint32_t n_views, float* ent_mats, cudaStream_t s) {
    frame_begin_kernel<<<1, 256, 0, s>>>(ctl, transforms, n_ent, views, n_views, ent_mats);
}

namespace {
// The resident CTAs per SM, for the current device.
template <int kCtas>
int preprocess_setup() {
    int r = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, preprocess_kernel<kCtas>, kPreThreads, sizeof(PreSmem));
    return r > 0 ? r : 1;
}

template <int kCtas>
void launch_preprocess_t(const PreprocessArgs& a, int num_sms, cudaStream_t s) {
    static_assert(sizeof(PreSmem) <= 48 * 1024, "no shared-memory opt-in");
    const int per_sm = device_once(preprocess_setup<kCtas>);
    const uint32_t chunks = (a.n + kPreThreads - 1) / kPreThreads;
    const uint32_t blocks = std::min<uint32_t>(chunks, uint32_t((num_sms > 0 ? num_sms : 148) * per_sm));
    launch_dependent(preprocess_kernel<kCtas>, dim3(blocks), dim3(kPreThreads), sizeof(PreSmem), s, a);
}
}  // namespace

void launch_preprocess(const PreprocessArgs& a, int num_sms, cudaStream_t s) {
    if (a.n == 0 || a.n_views == 0) return;
    if (a.n_views > 1)
        launch_preprocess_t<6>(a, num_sms, s);
    else
        launch_preprocess_t<4>(a, num_sms, s);
}

void launch_scan_tiles(const Splat* splats, uint32_t n, uint32_t* offsets, uint32_t* total, uint64_t* desc,
                       FrameCtl* ctl, uint32_t* status, uint32_t spin_limit, uint32_t never_publish, cudaStream_t s) {
    const uint32_t parts = uint32_t(scan_tiles_desc_entries(n));
    scan_begin_kernel<<<parts / 256 + 1, 256, 0, s>>>(desc, parts, ctl, status, total);
    if (n == 0) return;
    launch_dependent(scan_tiles_kernel, dim3(parts), dim3(kScanThreads), 0, s, splats, n, offsets, desc, ctl, status,
                     total, spin_limit, never_publish);
}

void launch_pack_records(const float* means, const float* log_scales, const float* quats, const float* logits,
                         const float* sh, uint32_t n, float* recs, cudaStream_t s) {
    if (n == 0) return;
    const uint64_t blocks = (uint64_t(n) * (kRecordFloats / 4) + 255) / 256;
    const bool vec = ((reinterpret_cast<uintptr_t>(quats) | reinterpret_cast<uintptr_t>(sh)) & 15u) == 0;
    if (vec)
        pack_records_kernel<true><<<unsigned(blocks), 256, 0, s>>>(means, log_scales, quats, logits, sh, n, recs);
    else
        pack_records_kernel<false><<<unsigned(blocks), 256, 0, s>>>(means, log_scales, quats, logits, sh, n, recs);
}

}  // namespace tpd
