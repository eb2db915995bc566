// backward.cu — preprocess adjoint: dL/d(px, py, conic, opacity, colour) of each
// (view, Gaussian) -> dL/d(mean, log-scale, quaternion, opacity logit, SH).
//
// The reference has no backward pass (differential/ is an empty placeholder);
// this is the adjoint of its forward maths, project.slang:33-90 with
// splat/volume.slang:20-63 and splat/common.slang:35-92:
//   colour  = max(SH(dir) + 0.5, 0), dir = normalize(mean - campos) (pre-model mean)
//   (px,py) = ndc2pix(clip.xy / clip.w), clip = projview*model*(mean, 1)
//   conic   = inverse(T Sigma T^T + 0.3 I), T = J(view*model*(mean,1)) * W(view)
//   Sigma   = (R S)(R S)^T, R from the quaternion as stored (not normalised),
//             S = diag(exp(log_scale) * modifier)
//   opacity = sigmoid(logit)
// Two threads per Gaussian, one for the colour's adjoint and one for the
// others', loop over the views, so gradients of the batched form accumulate in
// registers and are written once (no atomics).
#include "tpd_common.cuh"
#include "tpd_kernels.h"

namespace tpd {
namespace {

constexpr float SH_C0 = 0.28209479177387814f;
constexpr float SH_C1 = 0.4886025119029199f;
constexpr float C2_0 = 1.0925484305920792f, C2_1 = -1.0925484305920792f, C2_2 = 0.31539156525252005f,
                C2_3 = -1.0925484305920792f, C2_4 = 0.5462742152960396f;
constexpr float C3_0 = -0.5900435899266435f, C3_1 = 2.890611442640554f, C3_2 = -0.4570457994644658f,
                C3_3 = 0.3731763325901154f, C3_4 = -0.4570457994644658f, C3_5 = 1.445305721320277f,
                C3_6 = -0.5900435899266435f;

// SH basis value b and its direction gradient g for feature k = 1..15.
__device__ __forceinline__ void sh_basis(int k, float x, float y, float z, float& b, float& g0, float& g1, float& g2) {
    const float xx = x * x, yy = y * y, zz = z * z;
    g0 = g1 = g2 = 0.f;
    switch (k) {
        case 1: b = -SH_C1 * y; g1 = -SH_C1; break;
        case 2: b = SH_C1 * z; g2 = SH_C1; break;
        case 3: b = -SH_C1 * x; g0 = -SH_C1; break;
        case 4: b = C2_0 * x * y; g0 = C2_0 * y; g1 = C2_0 * x; break;
        case 5: b = C2_1 * y * z; g1 = C2_1 * z; g2 = C2_1 * y; break;
        case 6: b = C2_2 * (2.f * zz - xx - yy); g0 = -2.f * C2_2 * x; g1 = -2.f * C2_2 * y; g2 = 4.f * C2_2 * z; break;
        case 7: b = C2_3 * z * x; g0 = C2_3 * z; g2 = C2_3 * x; break;
        case 8: b = C2_4 * (xx - yy); g0 = 2.f * C2_4 * x; g1 = -2.f * C2_4 * y; break;
        case 9: b = C3_0 * y * (3.f * xx - yy); g0 = C3_0 * 6.f * x * y; g1 = C3_0 * (3.f * xx - 3.f * yy); break;
        case 10: b = C3_1 * x * y * z; g0 = C3_1 * y * z; g1 = C3_1 * x * z; g2 = C3_1 * x * y; break;
        case 11: b = C3_2 * y * (4.f * zz - xx - yy); g0 = C3_2 * (-2.f * x * y); g1 = C3_2 * (4.f * zz - xx - 3.f * yy); g2 = C3_2 * 8.f * y * z; break;
        case 12: b = C3_3 * z * (2.f * zz - 3.f * xx - 3.f * yy); g0 = C3_3 * (-6.f * x * z); g1 = C3_3 * (-6.f * y * z); g2 = C3_3 * (6.f * zz - 3.f * xx - 3.f * yy); break;
        case 13: b = C3_4 * x * (4.f * zz - xx - yy); g0 = C3_4 * (4.f * zz - 3.f * xx - yy); g1 = C3_4 * (-2.f * x * y); g2 = C3_4 * 8.f * x * z; break;
        case 14: b = C3_5 * z * (xx - yy); g0 = C3_5 * 2.f * x * z; g1 = -C3_5 * 2.f * y * z; g2 = C3_5 * (xx - yy); break;
        case 15: b = C3_6 * x * (xx - 3.f * yy); g0 = C3_6 * (3.f * xx - 3.f * yy); g1 = C3_6 * (-6.f * x * y); break;
        default: b = 0.f;
    }
}

constexpr uint32_t kBwdThreads = 128;  // Gaussians per CTA

__device__ __forceinline__ void unpack4(float4 f, float* to) {
    to[0] = f.x;
    to[1] = f.y;
    to[2] = f.z;
    to[3] = f.w;
}

// The Gaussian of a thread and its views' data.
struct Item {
    const PreprocessBackwardArgs& a;
    uint32_t i, e;      // Gaussian, entity
    bool active;
    const float* rec;   // its record in shared memory, 16-byte aligned
    __device__ __forceinline__ float radius(uint32_t v) const {
        return active && v < a.n_views ? a.splats[size_t(v) * a.n + i].radius : 0.0f;
    }
    __device__ __forceinline__ const float4* splat(uint32_t v) const {
        return reinterpret_cast<const float4*>(a.splats + size_t(v) * a.n + i);
    }
    __device__ __forceinline__ const float4* g2d(uint32_t v) const {
        return reinterpret_cast<const float4*>(a.g2d + (size_t(v) * a.n + i) * kG2DStride);
    }
    __device__ __forceinline__ float4 f4(int q) const { return reinterpret_cast<const float4*>(rec)[q]; }
};

// Walks the views that the item is in. A view's radius (0: not in it) is
// loaded two views ahead and, where it is not 0, load(v) one view ahead, so a
// view without the Gaussian costs four bytes and the loads of one with it
// overlap the work on the view before. take() moves what was loaded to the
// work's registers. (Each lane walking only its own views measured slower: the
// views' constants are then loaded per lane.)
template <typename Load, typename Take, typename Work>
__device__ __forceinline__ void for_each_view(const Item& it, Load load, Take take, Work work) {
    float next = it.radius(0), next2 = it.radius(1);
    if (next > 0.0f) load(0u);
    for (uint32_t v = 0; v < it.a.n_views; ++v) {
        const float radius = next;
        take();
        next = next2;
        if (next > 0.0f) load(v + 1u);
        next2 = it.radius(v + 2u);
        if (radius > 0.0f) work(v);
    }
}

// The colour half: dL/dcolour -> SH coefficients gsh and, through the view
// direction, the mean (gm).
__device__ __forceinline__ void colour_adjoint(const Item& it, float (&gsh)[48], float (&gm)[3]) {
    const int nf = it.a.sh_degree >= 3 ? 15 : it.a.sh_degree == 2 ? 8 : it.a.sh_degree == 1 ? 3 : 0;
    const bool compat = it.a.band3_compat != 0;
    const float4 mo = it.f4(0);
    float4 n_c = make_float4(0.f, 0.f, 0.f, 0.f), n_g1 = n_c, col = n_c, g1 = n_c;
    float n_g8 = 0.f, g8 = 0.f;
    auto load = [&](uint32_t v) {
        n_c = it.splat(v)[0];
        n_g1 = it.g2d(v)[1];
        n_g8 = it.g2d(v)[2].x;
    };
    auto take = [&]() {
        col = n_c;
        g1 = n_g1;
        g8 = n_g8;
    };
    for_each_view(it, load, take, [&](uint32_t v) {
        const float graw[3] = {col.x > 0.f ? g1.z : 0.f, col.y > 0.f ? g1.w : 0.f, col.z > 0.f ? g8 : 0.f};
        float V[12];
        const float4* p = reinterpret_cast<const float4*>(it.a.views + v);
#pragma unroll
        for (int r = 0; r < 3; ++r) unpack4(__ldg(p + r), V + 4 * r);
        const float d0 = mo.x + (V[0] * V[3] + V[4] * V[7] + V[8] * V[11]);  // mean - camera position
        const float d1 = mo.y + (V[1] * V[3] + V[5] * V[7] + V[9] * V[11]);
        const float d2 = mo.z + (V[2] * V[3] + V[6] * V[7] + V[10] * V[11]);
        const float inv_len = 1.0f / sqrtf(d0 * d0 + d1 * d1 + d2 * d2);
        const float x = d0 * inv_len, y = d1 * inv_len, z = d2 * inv_len;
#pragma unroll
        for (int c = 0; c < 3; ++c) gsh[c] += graw[c] * SH_C0;
        // dL/ddir through feature k: its three coefficients weighted by the
        // colour gradient, times the basis function's gradient
        float wk[16], gd0 = 0.f, gd1 = 0.f, gd2 = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            // the channel's coefficients: words 15 + 15 c .. 29 + 15 c of the record
            constexpr int kFirst[3] = {3, 7, 11};  // the 16-byte piece holding the first of them
            float f[20];
#pragma unroll
            for (int q = 0; q < (c < 2 ? 5 : 4); ++q) unpack4(it.f4(kFirst[c] + q), f + 4 * q);
#pragma unroll
            for (int k = 1; k <= 15; ++k) {
                const float t = f[15 + 15 * c - 4 * kFirst[c] + k - 1];
                wk[k] = c == 0 ? graw[0] * t : wk[k] + graw[c] * t;
            }
        }
        if (compat) wk[12] = graw[0] + graw[1] + graw[2];  // added, not multiplied, in the forward
#pragma unroll
        for (int k = 1; k <= 15; ++k) {
            if (k > nf) break;
            float b, b0, b1, b2;
            sh_basis(k, x, y, z, b, b0, b1, b2);
            if (k == 12 && compat) b = 1.0f;
#pragma unroll
            for (int c = 0; c < 3; ++c) gsh[3 + c * 15 + (k - 1)] += graw[c] * b;
            gd0 += wk[k] * b0;
            gd1 += wk[k] * b1;
            gd2 += wk[k] * b2;
        }
        const float dd = x * gd0 + y * gd1 + z * gd2;
        gm[0] += (gd0 - x * dd) * inv_len;
        gm[1] += (gd1 - y * dd) * inv_len;
        gm[2] += (gd2 - z * dd) * inv_len;
    });
}

// R from the quaternion as stored, M = R S.
__device__ __forceinline__ void rotation_scale(const float4 q, const float4 sc, float (&R)[9], float (&s)[3], float (&M)[9]) {
    const float qx = q.x, qy = q.y, qz = q.z, qw = q.w;
    R[0] = 1.f - 2.f * (qy * qy + qz * qz);
    R[1] = 2.f * (qx * qy - qw * qz);
    R[2] = 2.f * (qx * qz + qw * qy);
    R[3] = 2.f * (qx * qy + qw * qz);
    R[4] = 1.f - 2.f * (qx * qx + qz * qz);
    R[5] = 2.f * (qy * qz - qw * qx);
    R[6] = 2.f * (qx * qz - qw * qy);
    R[7] = 2.f * (qy * qz + qw * qx);
    R[8] = 1.f - 2.f * (qx * qx + qy * qy);
    s[0] = sc.x * sc.w;
    s[1] = sc.y * sc.w;
    s[2] = sc.z * sc.w;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) M[r * 3 + c] = R[r * 3 + c] * s[c];
}

// The shape half: dL/d(px, py, conic, opacity) -> opacity logit, mean (gm),
// and dL/dSigma + its transpose (gsig: elements (0,0), (0,1), (0,2), (1,1),
// (1,2), (2,2)), which is all that is used of it.
__device__ __forceinline__ void shape_adjoint(const Item& it, float& glogit, float (&gm)[3], float (&gsig)[6]) {
    const float4 mo = it.f4(0);
    const float m[3] = {mo.x, mo.y, mo.z}, op = mo.w;
    float Sig[9];
    {
        float R[9], s[3], M[9];
        rotation_scale(it.f4(1), it.f4(2), R, s, M);
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                Sig[r * 3 + c] = M[r * 3 + 0] * M[c * 3 + 0] + M[r * 3 + 1] * M[c * 3 + 1] + M[r * 3 + 2] * M[c * 3 + 2];
    }
    float4 n_g0 = make_float4(0.f, 0.f, 0.f, 0.f), n_g1 = n_g0, g0 = n_g0, g1 = n_g0;
    auto load = [&](uint32_t v) {
        n_g0 = it.g2d(v)[0];
        n_g1 = it.g2d(v)[1];
    };
    auto take = [&]() {
        g0 = n_g0;
        g1 = n_g1;
    };
    for_each_view(it, load, take, [&](uint32_t v) {
        const float gpx = g0.x, gpy = g0.y, gA = g0.z, gB = g0.w, gC = g1.x, gop = g1.y;
        // the view's constants and the entity's matrices, 16 bytes at a time
        float V[12], em[kEntityMatFloats];
        const float4* p = reinterpret_cast<const float4*>(it.a.views + v);
#pragma unroll
        for (int r = 0; r < 3; ++r) unpack4(__ldg(p + r), V + 4 * r);
        const float4 f = __ldg(p + 8);  // focal, width, height
        const float Wd = float(__float_as_uint(f.z)), Hd = float(__float_as_uint(f.w));
        const float fxp = 0.5f * Wd * f.x, fyp = 0.5f * Hd * f.y;
        const float4* m4 =
            reinterpret_cast<const float4*>(it.a.ent_mats + (size_t(v) * it.a.n_ent + it.e) * kEntityMatFloats);
#pragma unroll
        for (int k = 0; k < kEntityMatFloats / 4; ++k) unpack4(__ldg(m4 + k), em + 4 * k);
        float vp[3], cp[4];
#pragma unroll
        for (int r = 0; r < 3; ++r) vp[r] = em[r * 4] * m[0] + em[r * 4 + 1] * m[1] + em[r * 4 + 2] * m[2] + em[r * 4 + 3];
#pragma unroll
        for (int r = 0; r < 4; ++r)
            cp[r] = em[12 + r * 4] * m[0] + em[12 + r * 4 + 1] * m[1] + em[12 + r * 4 + 2] * m[2] + em[12 + r * 4 + 3];

        glogit += gop * op * (1.f - op);

        // pixel position -> clip -> mean
        const float iw = 1.0f / cp[3];
        const float gc0 = gpx * Wd * (0.5f * iw), gc1 = gpy * Hd * (0.5f * iw);
        const float gc3 = -(gc0 * cp[0] + gc1 * cp[1]) * iw;
#pragma unroll
        for (int d = 0; d < 3; ++d) gm[d] += em[12 + 0 * 4 + d] * gc0 + em[12 + 1 * 4 + d] * gc1 + em[12 + 3 * 4 + d] * gc3;

        // 2D covariance. J by divisions, each rounded once as in the forward: the
        // conic's gradient amplifies J's error for thin splats (with one reciprocal
        // and multiplications single gradients moved by up to 2e-3; 183 us instead
        // of 187 for 8 views of 500,000)
        const float vz = vp[2], ivz = 1.0f / vz;
        const float J0 = fxp / vz, J2 = -fxp * vp[0] / (vz * vz), J4 = fyp / vz, J5 = -fyp * vp[1] / (vz * vz);
        float Tm[6];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            Tm[c] = J0 * V[0 * 4 + c] + J2 * V[2 * 4 + c];
            Tm[3 + c] = J4 * V[1 * 4 + c] + J5 * V[2 * 4 + c];
        }
        float TS[6];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                TS[r * 3 + c] = Tm[r * 3 + 0] * Sig[0 * 3 + c] + Tm[r * 3 + 1] * Sig[1 * 3 + c] + Tm[r * 3 + 2] * Sig[2 * 3 + c];
        const float ca = TS[0] * Tm[0] + TS[1] * Tm[1] + TS[2] * Tm[2] + 0.3f;
        const float cb = TS[3] * Tm[0] + TS[4] * Tm[1] + TS[5] * Tm[2];
        const float cc = TS[3] * Tm[3] + TS[4] * Tm[4] + TS[5] * Tm[5] + 0.3f;
        const float det = ca * cc - cb * cb;
        const float idet2 = 1.f / (det * det);
        const float ga = (-gA * cc * cc + gB * cb * cc - gC * cb * cb) * idet2;
        const float gb = (2.f * gA * cb * cc - gB * (ca * cc + cb * cb) + 2.f * gC * ca * cb) * idet2;
        const float gc = (-gA * cb * cb + gB * ca * cb - gC * ca * ca) * idet2;
        // G = [[ga, 0], [gb, gc]]: dL/dSig = T^T G T, dL/dT = (G + G^T) T Sig
        {
            int k = 0;
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int c = r; c < 3; ++c, ++k)
                    gsig[k] += 2.f * ga * Tm[r] * Tm[c] + 2.f * gc * Tm[3 + r] * Tm[3 + c] +
                               gb * (Tm[3 + r] * Tm[c] + Tm[3 + c] * Tm[r]);
        }
        float gT[6];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            gT[c] = 2.f * ga * TS[c] + gb * TS[3 + c];
            gT[3 + c] = gb * TS[c] + 2.f * gc * TS[3 + c];
        }
        // T = J W: dL/dJ = dL/dT W^T (only J0, J2, J4, J5 are non-zero functions of vp)
        const float gJ0 = gT[0] * V[0] + gT[1] * V[1] + gT[2] * V[2];
        const float gJ2 = gT[0] * V[8] + gT[1] * V[9] + gT[2] * V[10];
        const float gJ4 = gT[3] * V[4] + gT[4] * V[5] + gT[5] * V[6];
        const float gJ5 = gT[3] * V[8] + gT[4] * V[9] + gT[5] * V[10];
        // J0 = fx / z, J2 = -fx x / z^2, J4 = fy / z, J5 = -fy y / z^2
        const float gvp0 = -gJ2 * J0 * ivz;
        const float gvp1 = -gJ5 * J4 * ivz;
        const float gvp2 = -(gJ0 * J0 + 2.f * gJ2 * J2 + gJ4 * J4 + 2.f * gJ5 * J5) * ivz;
#pragma unroll
        for (int d = 0; d < 3; ++d) gm[d] += em[0 * 4 + d] * gvp0 + em[1 * 4 + d] * gvp1 + em[2 * 4 + d] * gvp2;
    });
}

// A barrier of the whole CTA that its two halves reach in their own code (a
// barrier resource of its own: bar.sync counts arrivals, wherever they come from).
__device__ __forceinline__ void records_done() {
    asm volatile("bar.sync 1, %0;" ::"n"(2 * kBwdThreads) : "memory");
}

// A CTA of 256 threads for 128 Gaussians: the first four warps take the colour
// half of each, the other four the shape half. One thread for both held 168
// registers, three CTAs of four warps per SM, and waited on its own chains
// (issue on 40% of the cycles). 8 views of 500,000: 276 -> 187 us, of 1.5M of
// which few are in a view 655 -> 540. Three CTAs per SM spill (222 us).
// Its records are staged into shared memory with coalesced 16-byte loads (a
// record is 240 B, so thread-per-record loads would stride), and its SH
// gradients leave through the same buffer as coalesced 16-byte stores.
__global__ void __launch_bounds__(2 * kBwdThreads, 2) preprocess_backward_kernel(PreprocessBackwardArgs a) {
    __shared__ __align__(16) float srec[kBwdThreads * kRecordFloats];  // 30 KB; reused for the SH gradients
    __shared__ float sgm[3][kBwdThreads];                              // the colour half's mean gradients
    pdl_wait();  // launched as a dependent of the stream's previous kernel: its output is read below
    pdl_trigger();
    const uint32_t base = blockIdx.x * kBwdThreads;
    const uint32_t cnt = min(kBwdThreads, a.n - base);
    {
        const float4* src = reinterpret_cast<const float4*>(a.recs + size_t(base) * kRecordFloats);
        float4* dst = reinterpret_cast<float4*>(srec);
        for (uint32_t k = threadIdx.x; k < cnt * (kRecordFloats / 4); k += 2 * kBwdThreads) dst[k] = src[k];
    }
    __syncthreads();
    const uint32_t t = threadIdx.x % kBwdThreads, i = base + t;
    const bool active = t < cnt;
    const Item it{a, i, (a.ent_idx && active) ? a.ent_idx[i] : 0u, active, srec + (active ? t : 0u) * kRecordFloats};
    if (threadIdx.x < kBwdThreads) {
        float gsh[48], gm[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 48; ++k) gsh[k] = 0.f;
        colour_adjoint(it, gsh, gm);
        sgm[0][t] = gm[0];
        sgm[1][t] = gm[1];
        sgm[2][t] = gm[2];
        records_done();
        if (active) {
            float4* mine = reinterpret_cast<float4*>(srec + t * 48);
#pragma unroll
            for (int k = 0; k < 12; ++k) mine[k] = make_float4(gsh[4 * k], gsh[4 * k + 1], gsh[4 * k + 2], gsh[4 * k + 3]);
        }
    } else {
        float glogit = 0.f, gm[3] = {0.f, 0.f, 0.f}, gsig[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        shape_adjoint(it, glogit, gm, gsig);
        // Sigma = M M^T, M = R S
        const float4 q = it.f4(1);
        float R[9], s[3], M[9], gM[9], gR[9];
        rotation_scale(q, it.f4(2), R, s, M);
        const float gS[9] = {gsig[0], gsig[1], gsig[2], gsig[1], gsig[3], gsig[4], gsig[2], gsig[4], gsig[5]};
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                gM[r * 3 + c] = gS[r * 3 + 0] * M[0 * 3 + c] + gS[r * 3 + 1] * M[1 * 3 + c] + gS[r * 3 + 2] * M[2 * 3 + c];
                gR[r * 3 + c] = gM[r * 3 + c] * s[c];
            }
        const float qx = q.x, qy = q.y, qz = q.z, qw = q.w;
        float gq[4], gls[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) gls[c] = (gM[0 * 3 + c] * R[0 * 3 + c] + gM[1 * 3 + c] * R[1 * 3 + c] + gM[2 * 3 + c] * R[2 * 3 + c]) * s[c];
        gq[0] = gR[1] * 2.f * qy + gR[2] * 2.f * qz + gR[3] * 2.f * qy + gR[4] * (-4.f * qx) + gR[5] * (-2.f * qw) +
                gR[6] * 2.f * qz + gR[7] * 2.f * qw + gR[8] * (-4.f * qx);
        gq[1] = gR[0] * (-4.f * qy) + gR[1] * 2.f * qx + gR[2] * 2.f * qw + gR[3] * 2.f * qx + gR[5] * 2.f * qz +
                gR[6] * (-2.f * qw) + gR[7] * 2.f * qz + gR[8] * (-4.f * qy);
        gq[2] = gR[0] * (-4.f * qz) + gR[1] * (-2.f * qw) + gR[2] * 2.f * qx + gR[3] * 2.f * qw + gR[4] * (-4.f * qz) +
                gR[5] * 2.f * qy + gR[6] * 2.f * qx + gR[7] * 2.f * qy;
        gq[3] = gR[1] * (-2.f * qz) + gR[2] * 2.f * qy + gR[3] * 2.f * qz + gR[5] * (-2.f * qx) + gR[6] * (-2.f * qy) +
                gR[7] * 2.f * qx;
        records_done();
        if (active) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                a.g_means[size_t(i) * 3 + c] = gm[c] + sgm[c][t];
                a.g_log_scales[size_t(i) * 3 + c] = gls[c];
            }
            if ((reinterpret_cast<uintptr_t>(a.g_quats) & 15u) == 0) {
                reinterpret_cast<float4*>(a.g_quats)[i] = make_float4(gq[0], gq[1], gq[2], gq[3]);
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) a.g_quats[size_t(i) * 4 + c] = gq[c];
            }
            a.g_logits[i] = glogit;
        }
    }
    __syncthreads();
    if ((reinterpret_cast<uintptr_t>(a.g_sh) & 15u) == 0) {
        float4* gs = reinterpret_cast<float4*>(a.g_sh + size_t(base) * 48);
        const float4* from = reinterpret_cast<const float4*>(srec);
        for (uint32_t k = threadIdx.x; k < cnt * 12; k += 2 * kBwdThreads) gs[k] = from[k];
    } else {  // a caller's buffer that is not 16-byte aligned
        float* gs = a.g_sh + size_t(base) * 48;
        for (uint32_t k = threadIdx.x; k < cnt * 48; k += 2 * kBwdThreads) gs[k] = srec[k];
    }
}

}  // namespace

void launch_preprocess_backward(const PreprocessBackwardArgs& a, cudaStream_t s) {
    if (a.n == 0) return;
    launch_dependent(preprocess_backward_kernel, dim3((a.n + kBwdThreads - 1) / kBwdThreads), dim3(2 * kBwdThreads),
                     0, s, a);
}

}  // namespace tpd
