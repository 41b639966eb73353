// scene.cu -- per-Gaussian kernels: instance snapshot, per-forward preparation (live opacity,
// scaling factor, SH colour) and the post-backward gradient fold with the SH backward.
#include "gray_bulk.cuh"
#include "gray_device.cuh"
#include "gray_internal.h"

namespace gray {

// Real SH basis without the DC term, degrees 1..3 (15 functions) in the reference's order
// (cuda/utils/sh.cu:54-67: per degree l, m = l..1 -> sqrt2 Im, m = 0, m = 1..l -> sqrt2 Re).
#define SH_C0 0.28209479177387814f
#define SH_C1 0.48860251190291992f
#define SH_C2_0 1.0925484305920792f
#define SH_C2_2 0.31539156525252005f
#define SH_C2_4 0.54627421529603959f
#define SH_C3_0 0.59004358992664352f
#define SH_C3_1 2.8906114426405538f
#define SH_C3_2 0.45704579946446572f
#define SH_C3_3 0.3731763325901154f
#define SH_C3_5 1.4453057213202769f

__device__ __forceinline__ void sh_basis(float x, float y, float z, float b[15]) {
    float xx = x * x, yy = y * y, zz = z * z;
    b[0] = -SH_C1 * y;
    b[1] = SH_C1 * z;
    b[2] = -SH_C1 * x;
    b[3] = SH_C2_0 * (x * y);
    b[4] = -SH_C2_0 * (y * z);
    b[5] = SH_C2_2 * (2.0f * zz - xx - yy);
    b[6] = -SH_C2_0 * (x * z);
    b[7] = SH_C2_4 * (xx - yy);
    b[8] = -SH_C3_0 * (y * (3.0f * xx - yy));
    b[9] = SH_C3_1 * (x * y * z);
    b[10] = -SH_C3_2 * (y * (4.0f * zz - xx - yy));
    b[11] = SH_C3_3 * (z * (2.0f * zz - 3.0f * xx - 3.0f * yy));
    b[12] = -SH_C3_2 * (x * (4.0f * zz - xx - yy));
    b[13] = SH_C3_5 * (z * (xx - yy));
    b[14] = -SH_C3_0 * (x * (xx - 3.0f * yy));
}

__device__ __forceinline__ void sh_basis_grad(float x, float y, float z, float dx[15], float dy[15], float dz[15]) {
    float xx = x * x, yy = y * y, zz = z * z;
    dx[0] = 0.0f;          dy[0] = -SH_C1;          dz[0] = 0.0f;
    dx[1] = 0.0f;          dy[1] = 0.0f;            dz[1] = SH_C1;
    dx[2] = -SH_C1;        dy[2] = 0.0f;            dz[2] = 0.0f;
    dx[3] = SH_C2_0 * y;   dy[3] = SH_C2_0 * x;     dz[3] = 0.0f;
    dx[4] = 0.0f;          dy[4] = -SH_C2_0 * z;    dz[4] = -SH_C2_0 * y;
    dx[5] = SH_C2_2 * (-2.0f * x); dy[5] = SH_C2_2 * (-2.0f * y); dz[5] = SH_C2_2 * (4.0f * z);
    dx[6] = -SH_C2_0 * z;  dy[6] = 0.0f;            dz[6] = -SH_C2_0 * x;
    dx[7] = SH_C2_4 * (2.0f * x); dy[7] = SH_C2_4 * (-2.0f * y); dz[7] = 0.0f;
    dx[8] = -SH_C3_0 * (6.0f * x * y);
    dy[8] = -SH_C3_0 * (3.0f * xx - 3.0f * yy);
    dz[8] = 0.0f;
    dx[9] = SH_C3_1 * (y * z);
    dy[9] = SH_C3_1 * (x * z);
    dz[9] = SH_C3_1 * (x * y);
    dx[10] = -SH_C3_2 * (-2.0f * x * y);
    dy[10] = -SH_C3_2 * (4.0f * zz - xx - 3.0f * yy);
    dz[10] = -SH_C3_2 * (8.0f * y * z);
    dx[11] = SH_C3_3 * (-6.0f * x * z);
    dy[11] = SH_C3_3 * (-6.0f * y * z);
    dz[11] = SH_C3_3 * (6.0f * zz - 3.0f * xx - 3.0f * yy);
    dx[12] = -SH_C3_2 * (4.0f * zz - 3.0f * xx - yy);
    dy[12] = -SH_C3_2 * (-2.0f * x * y);
    dz[12] = -SH_C3_2 * (8.0f * x * z);
    dx[13] = SH_C3_5 * (2.0f * x * z);
    dy[13] = SH_C3_5 * (-2.0f * y * z);
    dz[13] = SH_C3_5 * (xx - yy);
    dx[14] = -SH_C3_0 * (3.0f * xx - 3.0f * yy);
    dy[14] = -SH_C3_0 * (-6.0f * x * y);
    dz[14] = 0.0f;
}

__device__ __forceinline__ int sh_count(int degree) {
    return degree <= 0 ? 0 : degree == 1 ? 3 : degree == 2 ? 8 : 15;
}

// ---------------------------------------------------------------------------------------------
// Instance snapshot (reference: populate_bvh_kernel + create_transform_matrix,
// cuda/optix/bvh_wrapper.cu:8-59).  Writes the world->unit-sphere rows (M | mu), the
// unit-sphere->world rows R diag(s), the leaf box and the visibility of each Gaussian.
// ---------------------------------------------------------------------------------------------
// The snapshot of one Gaussian from its parameters (mean, rotation quaternion (r, x, y, z), log
// scales, logit opacity): rows g of (M | mu), rows w of (L | mu), its leaf box and visibility.
struct SnapRecord {
    float4 g[3], w[3], bmin, bmax;
    bool vis;
};

__device__ __forceinline__ void snapshot_one(const float mu_in[3], float4 q, const float log_s[3], float logit_o,
                                             float athr, float p, float gsf, SnapRecord &out) {
    float o = sigmoid_act(logit_o);
    float sf = scaling_factor(o, athr, p);
    float s[3];
#pragma unroll
    for (int k = 0; k < 3; k++) s[k] = gexp(log_s[k]) * sf * gsf;
    float r = q.x, x = q.y, y = q.z, z = q.w;
    float norm = sqrtf(r * r + x * x + y * y + z * z);
    r = r / norm;
    x = x / norm;
    y = y / norm;
    z = z / norm;
    float R[9];
    R[0] = 1.0f - 2.0f * (y * y + z * z);
    R[1] = 2.0f * (x * y - r * z);
    R[2] = 2.0f * (x * z + r * y);
    R[3] = 2.0f * (x * y + r * z);
    R[4] = 1.0f - 2.0f * (x * x + z * z);
    R[5] = 2.0f * (y * z - r * x);
    R[6] = 2.0f * (x * z - r * y);
    R[7] = 2.0f * (y * z + r * x);
    R[8] = 1.0f - 2.0f * (x * x + y * y);
    const float mu[3] = {mu_in[0], mu_in[1], mu_in[2]};
    bool vis = sf > 0.0f && s[0] > 0.0f && s[1] > 0.0f && s[2] > 0.0f && isfinite(s[0]) && isfinite(s[1]) &&
               isfinite(s[2]) && isfinite(mu[0]) && isfinite(mu[1]) && isfinite(mu[2]);
    float L[9];
#pragma unroll
    for (int rr = 0; rr < 3; rr++) {
#pragma unroll
        for (int c = 0; c < 3; c++) L[3 * rr + c] = R[3 * rr + c] * s[c];
    }
#pragma unroll
    for (int rr = 0; rr < 3; rr++) {
        float4 gr;
        gr.x = vis ? R[rr] / s[rr] : 0.0f;
        gr.y = vis ? R[3 + rr] / s[rr] : 0.0f;
        gr.z = vis ? R[6 + rr] / s[rr] : 0.0f;
        gr.w = mu[rr];
        out.g[rr] = gr;
        out.w[rr] = make_float4(L[3 * rr], L[3 * rr + 1], L[3 * rr + 2], mu[rr]);
    }
    if (vis) {
        float pad_mu = 2.0e-6f * (fabsf(mu[0]) + fabsf(mu[1]) + fabsf(mu[2]));
        float h[3];
#pragma unroll
        for (int rr = 0; rr < 3; rr++) {
            float a0 = L[3 * rr], a1 = L[3 * rr + 1], a2 = L[3 * rr + 2];
            float hh = sqrtf(a0 * a0 + a1 * a1 + a2 * a2);
            h[rr] = hh + hh * 1.0e-4f + pad_mu + 1.0e-30f;
        }
        out.bmin = make_float4(mu[0] - h[0], mu[1] - h[1], mu[2] - h[2], 0.0f);
        out.bmax = make_float4(mu[0] + h[0], mu[1] + h[1], mu[2] + h[2], 0.0f);
    } else {
        bool fin = isfinite(mu[0]) && isfinite(mu[1]) && isfinite(mu[2]);
        out.bmin = fin ? make_float4(mu[0], mu[1], mu[2], 0.0f) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        out.bmax = out.bmin;
    }
    out.vis = vis;
}

// Gaussian i's snapshot, straight from and to memory.
__device__ __forceinline__ void snapshot_row(int i, const float *__restrict__ mean,
                                             const float4 *__restrict__ rotation, const float *__restrict__ scale,
                                             const float *__restrict__ opacity, float athr, float pw, float gsf,
                                             float4 *__restrict__ geom, float4 *__restrict__ l2w,
                                             float4 *__restrict__ aabb, uint8_t *__restrict__ visible) {
    const float mu[3] = {mean[3 * i], mean[3 * i + 1], mean[3 * i + 2]};
    const float ls[3] = {scale[3 * i], scale[3 * i + 1], scale[3 * i + 2]};
    SnapRecord r;
    snapshot_one(mu, rotation[i], ls, opacity[i], athr, pw, gsf, r);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        geom[3 * i + k] = r.g[k];
        l2w[3 * i + k] = r.w[k];
    }
    aabb[2 * i] = r.bmin;
    aabb[2 * i + 1] = r.bmax;
    visible[i] = r.vis ? 1 : 0;
}

// One thread per Gaussian: the whole snapshot when there are fewer than a tile or a pointer is not
// 16-byte aligned.
__global__ void snapshot_kernel(int n, const float *__restrict__ mean, const float4 *__restrict__ rotation,
                                const float *__restrict__ scale, const float *__restrict__ opacity,
                                const float *__restrict__ cfg_alpha_threshold, const float *__restrict__ cfg_exp_power,
                                const float *__restrict__ cfg_gsf, float4 *__restrict__ geom, float4 *__restrict__ l2w,
                                float4 *__restrict__ aabb, uint8_t *__restrict__ visible) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        snapshot_row(i, mean, rotation, scale, opacity, *cfg_alpha_threshold, *cfg_exp_power, *cfg_gsf, geom, l2w,
                     aabb, visible);
}

// Bulk-pipelined snapshot: a persistent block takes tiles of kSnapTile consecutive Gaussians.  One
// thread loads a tile's parameter rows (mean, rotation, scale, opacity: 44 B per Gaussian, four
// contiguous ranges) into shared memory with bulk copies completing on an mbarrier, double-buffered
// so that the next tile's loads are in flight while this one is computed; each thread computes one
// Gaussian and writes its records into a shared-memory copy of the tile's output ranges, which one
// thread then stores with four bulk copies (geom, l2w, aabb, visible: 129 B per Gaussian) while the
// block goes on.  Every copy starts on a 16-byte boundary and spans a multiple of 16 bytes (the
// launcher checks the pointers; the tile is a multiple of 16 Gaussians).  Gaussians past the last
// full tile are the last block's, a thread each, while its first tile loads (in a launch of their own
// they held up the stream for 4 us).
constexpr int kSnapTile = 128;
static_assert(kSnapTile % 16 == 0, "every per-tile range must span a multiple of 16 bytes");

struct SnapIn {
    float mean[3 * kSnapTile];
    float4 rotation[kSnapTile];
    float scale[3 * kSnapTile];
    float opacity[kSnapTile];
};
struct SnapOut {
    float4 geom[3 * kSnapTile];
    float4 l2w[3 * kSnapTile];
    float4 aabb[2 * kSnapTile];
    uint8_t visible[kSnapTile];
};
constexpr uint32_t kSnapInBytes = 44u * kSnapTile;

__device__ __forceinline__ void snap_issue_loads(SnapIn &in, uint64_t *bar, int tile, const float *mean,
                                                 const float4 *rotation, const float *scale, const float *opacity) {
    const size_t g0 = (size_t)tile * kSnapTile;
    mbar_expect_tx(bar, kSnapInBytes);
    bulk_load(in.mean, mean + 3 * g0, 12u * kSnapTile, bar);
    bulk_load(in.rotation, rotation + g0, 16u * kSnapTile, bar);
    bulk_load(in.scale, scale + 3 * g0, 12u * kSnapTile, bar);
    bulk_load(in.opacity, opacity + g0, 4u * kSnapTile, bar);
}

__global__ void __launch_bounds__(kSnapTile) snapshot_bulk_kernel(
    int n, int tiles, const float *__restrict__ mean, const float4 *__restrict__ rotation, const float *__restrict__ scale,
    const float *__restrict__ opacity, const float *__restrict__ cfg_alpha_threshold,
    const float *__restrict__ cfg_exp_power, const float *__restrict__ cfg_gsf, float4 *__restrict__ geom,
    float4 *__restrict__ l2w, float4 *__restrict__ aabb, uint8_t *__restrict__ visible, int32_t *__restrict__ status) {
    __shared__ __align__(16) SnapIn in[2];
    __shared__ __align__(16) SnapOut out;
    __shared__ __align__(8) uint64_t bar[2];
    const int t = threadIdx.x;
    if (t == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
    }
    __syncthreads();
    const float athr = *cfg_alpha_threshold, pw = *cfg_exp_power, gsf = *cfg_gsf;
    int tile = blockIdx.x;
    if (t == 0 && tile < tiles) snap_issue_loads(in[0], &bar[0], tile, mean, rotation, scale, opacity);
    if (blockIdx.x == gridDim.x - 1 && tiles * kSnapTile + t < n)
        snapshot_row(tiles * kSnapTile + t, mean, rotation, scale, opacity, athr, pw, gsf, geom, l2w, aabb, visible);
    int it = 0;
    bool timed_out = false;
    for (; tile < tiles; it++, tile += gridDim.x) {
        const int st = it & 1;
        const int next = tile + gridDim.x;
        if (t == 0 && next < tiles) {
            // in[st ^ 1] was last read in the previous tile, before its barriers
            fence_proxy_async();
            snap_issue_loads(in[st ^ 1], &bar[st ^ 1], next, mean, rotation, scale, opacity);
        }
        const bool ok = __syncthreads_and(mbar_wait(&bar[st], (uint32_t)(it >> 1) & 1u, kBulkWaitNs));
        if (!ok) {
            if (t == 0) atomicOr(status, GRAY_STATUS_COPY_TIMEOUT);
            timed_out = true;
            break;
        }
        SnapRecord r;
        {
            const float mu[3] = {in[st].mean[3 * t], in[st].mean[3 * t + 1], in[st].mean[3 * t + 2]};
            const float ls[3] = {in[st].scale[3 * t], in[st].scale[3 * t + 1], in[st].scale[3 * t + 2]};
            snapshot_one(mu, in[st].rotation[t], ls, in[st].opacity[t], athr, pw, gsf, r);
        }
        if (t == 0) bulk_wait_read();  // the previous tile's stores have read the staging
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 3; k++) {
            out.geom[3 * t + k] = r.g[k];
            out.l2w[3 * t + k] = r.w[k];
        }
        out.aabb[2 * t] = r.bmin;
        out.aabb[2 * t + 1] = r.bmax;
        out.visible[t] = r.vis ? 1 : 0;
        fence_proxy_async();
        __syncthreads();
        if (t == 0) {
            const size_t g0 = (size_t)tile * kSnapTile;
            bulk_store(geom + 3 * g0, out.geom, 48u * kSnapTile);
            bulk_store(l2w + 3 * g0, out.l2w, 48u * kSnapTile);
            bulk_store(aabb + 2 * g0, out.aabb, 32u * kSnapTile);
            bulk_store(visible + g0, out.visible, kSnapTile);
            bulk_commit();
        }
    }
    if (t == 0) {
        bulk_wait_all();
        if (timed_out) {
            // the loads still in flight (this tile's and the next one's) get their own bounded
            // waits, so that no copy targets this block's shared memory after it exits
            mbar_wait(&bar[it & 1], (uint32_t)(it >> 1) & 1u, kBulkWaitNs);
            if (tile + (int)gridDim.x < tiles)
                mbar_wait(&bar[(it + 1) & 1], (uint32_t)((it + 1) >> 1) & 1u, kBulkWaitNs);
        }
    }
}

cudaError_t launch_snapshot(const gray_params &p, cudaStream_t s) {
    const gray_gaussians &g = p.gaussians;
    const int n = g.count;
    if (n <= 0) return cudaSuccess;
    const float4 *rot = reinterpret_cast<const float4 *>(g.rotation);
    float4 *geom = reinterpret_cast<float4 *>(p.scene.geom), *l2w = reinterpret_cast<float4 *>(p.scene.l2w),
           *aabb = reinterpret_cast<float4 *>(p.scene.aabb);
    const bool bulk = p.status && aligned16(g.mean) && aligned16(g.rotation) && aligned16(g.scale) &&
                      aligned16(g.opacity) && aligned16(geom) && aligned16(l2w) && aligned16(aabb) &&
                      aligned16(p.scene.visible);
    const int tiles = bulk ? n / kSnapTile : 0;
    if (tiles > 0) {
        int sms = 0, per_sm = 0;
        cudaError_t e = resident_blocks(reinterpret_cast<const void *>(&snapshot_bulk_kernel), kSnapTile, 0, &sms, &per_sm);
        if (e != cudaSuccess) return e;
        const int want = sms * per_sm;
        snapshot_bulk_kernel<<<tiles < want ? tiles : want, kSnapTile, 0, s>>>(
            n, tiles, g.mean, rot, g.scale, g.opacity, p.config.alpha_threshold, p.config.exp_power,
            p.config.global_scale_factor, geom, l2w, aabb, p.scene.visible, p.status);
        return cudaGetLastError();
    }
    snapshot_kernel<<<blocks_for(n), kThreads, 0, s>>>(n, g.mean, rot, g.scale, g.opacity, p.config.alpha_threshold,
                                                       p.config.exp_power, p.config.global_scale_factor, geom, l2w,
                                                       aabb, p.scene.visible);
    return cudaGetLastError();
}

// The bounded wait of the pipelines above, made to run out: 16 bytes are announced on the phase and
// none are copied, so it never completes.
__global__ void copy_wait_selftest_kernel(int32_t *status, uint64_t limit_ns) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
        mbar_expect_tx(&bar, 16u);
    }
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(&bar, 0u, limit_ns)) && threadIdx.x == 0)
        atomicOr(status, GRAY_STATUS_COPY_TIMEOUT);
}

cudaError_t launch_copy_wait_selftest(int32_t *status, uint64_t limit_ns, cudaStream_t s) {
    copy_wait_selftest_kernel<<<1, 32, 0, s>>>(status, limit_ns);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Per-forward preparation: live opacity and scaling factor for the intersection test
// (cuda/shaders.cu:21-24, 51-53 read them per hit), and the SH colour
// (reference: sh_forward_kernel, cuda/utils/sh.cu:224-247).  SH coefficient rows are staged
// through shared memory with coalesced loads.
// ---------------------------------------------------------------------------------------------
constexpr int kPrepThreads = 128;

template <typename SHT>
__device__ __forceinline__ float sh_load(const SHT *p);
template <>
__device__ __forceinline__ float sh_load<float>(const float *p) {
    return *p;
}
template <>
__device__ __forceinline__ float sh_load<__half>(const __half *p) {
    return __half2float(*p);
}

// SH colour of one Gaussian seen from cam (reference: sh_forward_kernel, cuda/utils/sh.cu:224-247);
// dc and row (its 3 * nb rest coefficients, coefficient-major) in the storage type.
template <typename SHT>
__device__ __forceinline__ void sh_colour(const float mu[3], const float *cam, const SHT *dc, const SHT *row, int nb,
                                          float out[3]) {
    float v[3];
#pragma unroll
    for (int k = 0; k < 3; k++) v[k] = mu[k] - cam[k];
    float len2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    float inv = 1.0f / sqrtf(fmaxf(len2, 1e-20f));
    float b[15];
    sh_basis(v[0] * inv, v[1] * inv, v[2] * inv, b);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        float acc = SH_C0 * sh_load<SHT>(dc + c);
#pragma unroll
        for (int j = 0; j < 15; j++)
            if (j < nb) acc = fmaf(b[j], sh_load<SHT>(row + 3 * j + c), acc);
        acc = acc + 0.5f;
        out[c] = fmaxf(acc, 0.0f);
    }
}

// One thread per Gaussian, SH rows staged through shared memory with coalesced loads: the whole pass when
// there are fewer than a tile or a pointer is not 16-byte aligned.
// reset_frame: this launch counts the forward call and empties the backward hit list too.
template <typename SHT>
__global__ void __launch_bounds__(kPrepThreads) forward_prep_kernel(
    int n, int num_rest, const float *__restrict__ opacity, const uint8_t *__restrict__ visible,
    const float *__restrict__ cfg_alpha_threshold, const float *__restrict__ cfg_exp_power,
    const uint8_t *__restrict__ cfg_enable_sh, const int32_t *__restrict__ current_sh_degree, int max_sh_degree,
    const float *__restrict__ mean, const float *__restrict__ cam_origin, const SHT *__restrict__ sh_dc,
    const SHT *__restrict__ sh_rest, float *__restrict__ channels, float2 *__restrict__ live,
    uint8_t *__restrict__ was_visible, uint32_t *__restrict__ total_num_calls, uint32_t *__restrict__ hit_counter,
    uint8_t *__restrict__ grads_enabled, int grads, int reset_frame) {
    extern __shared__ __align__(16) unsigned char prep_smem[];
    SHT *stage = reinterpret_cast<SHT *>(prep_smem);  // kPrepThreads * num_rest * 3 coefficients
    const int i0 = blockIdx.x * kPrepThreads;
    const int i = i0 + threadIdx.x;
    if (reset_frame && blockIdx.x == 0 && threadIdx.x == 0) {
        *total_num_calls += 1u;
        *hit_counter = 0u;
        if (grads >= 0) *grads_enabled = (uint8_t)grads;
    }
    const bool enable_sh = *cfg_enable_sh != 0;
    int degree = *current_sh_degree;
    degree = min(min(degree, 3), max_sh_degree);
    const int nb = enable_sh ? sh_count(degree) : 0;
    const int per = num_rest * 3;
    if (nb > 0) {
        const int rows = min(kPrepThreads, n - i0);
        const long long base = (long long)i0 * per;
        for (int t = threadIdx.x; t < rows * per; t += kPrepThreads) stage[t] = sh_rest[base + t];
    }
    __syncthreads();
    if (i >= n) return;
    if (reset_frame) was_visible[i] = 0;
    const float athr = *cfg_alpha_threshold, pw = *cfg_exp_power;
    float o = sigmoid_act(opacity[i]);
    float sf = scaling_factor(o, athr, pw);
    live[i] = make_float2(visible[i] ? o : __int_as_float(0xff800000), sf);
    if (!enable_sh) return;
    const float mu[3] = {mean[3 * i], mean[3 * i + 1], mean[3 * i + 2]};
    float col[3];
    sh_colour<SHT>(mu, cam_origin, sh_dc + 3 * i, stage + threadIdx.x * per, nb, col);
#pragma unroll
    for (int c = 0; c < 3; c++) channels[3 * i + c] = col[c];
}

// Bulk-pipelined forward preparation: a persistent block takes tiles of kPrepTile consecutive
// Gaussians; one thread loads a tile's inputs (opacity, mean, snapshot visibility, and with SH on
// the DC and rest coefficients: contiguous ranges) into one of two shared-memory stages with bulk
// copies completing on an mbarrier, so the next tile's loads are in flight while this one is
// computed; each thread computes one Gaussian into a shared-memory copy of the tile's outputs
// (live values, colours, the reset visited flags), stored by one thread with bulk copies.  Stage
// layout (byte offsets, T = kPrepTile, b = sizeof(SHT)): opacity 0, mean 4T, visible 16T, sh_dc 17T,
// sh_rest 17T + 3Tb; every range spans a multiple of 16 bytes.  Shared memory: 16 B of barriers,
// two stages, then the output copy (colours 12T, live 8T, flags T).
constexpr int kPrepTile = 64;
static_assert(kPrepTile % 16 == 0, "every per-tile range must span a multiple of 16 bytes");
constexpr int kPrepBlocksPerSm = 4;

__host__ __device__ __forceinline__ uint32_t prep_stage_bytes(int num_rest, uint32_t sb) {
    return 17u * kPrepTile + 3u * kPrepTile * sb + (uint32_t)kPrepTile * 3u * (uint32_t)num_rest * sb;
}
__host__ __device__ __forceinline__ uint32_t prep_smem_bytes(int num_rest, uint32_t sb) {
    return 16u + 2u * prep_stage_bytes(num_rest, sb) + 21u * kPrepTile;
}

template <typename SHT>
__device__ __forceinline__ void prep_issue_loads(unsigned char *stg, uint64_t *bar, int tile, int per, bool dc,
                                                 bool rest, const float *opacity, const float *mean,
                                                 const uint8_t *visible, const SHT *sh_dc, const SHT *sh_rest) {
    constexpr uint32_t T = kPrepTile, sb = sizeof(SHT);
    const size_t g0 = (size_t)tile * T;
    const uint32_t rest_bytes = T * (uint32_t)per * sb;
    mbar_expect_tx(bar, 17u * T + (dc ? 3u * T * sb : 0u) + (rest ? rest_bytes : 0u));
    bulk_load(stg, opacity + g0, 4u * T, bar);
    bulk_load(stg + 4 * T, mean + 3 * g0, 12u * T, bar);
    bulk_load(stg + 16 * T, visible + g0, T, bar);
    if (dc) bulk_load(stg + 17 * T, sh_dc + 3 * g0, 3u * T * sb, bar);
    if (rest) bulk_load(stg + 17 * T + 3 * T * sb, sh_rest + g0 * per, rest_bytes, bar);
}

template <typename SHT>
__global__ void __launch_bounds__(kPrepTile) forward_prep_bulk_kernel(
    int n, int tiles, int num_rest, const float *__restrict__ opacity, const uint8_t *__restrict__ visible,
    const float *__restrict__ cfg_alpha_threshold, const float *__restrict__ cfg_exp_power,
    const uint8_t *__restrict__ cfg_enable_sh, const int32_t *__restrict__ current_sh_degree, int max_sh_degree,
    const float *__restrict__ mean, const float *__restrict__ cam_origin, const SHT *__restrict__ sh_dc,
    const SHT *__restrict__ sh_rest, float *__restrict__ channels, float2 *__restrict__ live,
    uint8_t *__restrict__ was_visible, uint32_t *__restrict__ total_num_calls, uint32_t *__restrict__ hit_counter,
    uint8_t *__restrict__ grads_enabled, int grads, int reset_frame, int32_t *__restrict__ status) {
    constexpr uint32_t T = kPrepTile, sb = sizeof(SHT);
    extern __shared__ __align__(16) unsigned char prep_smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(prep_smem);
    const int per = 3 * num_rest;
    const uint32_t stage_bytes = prep_stage_bytes(num_rest, sb);
    unsigned char *stages = prep_smem + 16;
    unsigned char *outb = stages + 2 * stage_bytes;
    float *ch_out = reinterpret_cast<float *>(outb);
    float2 *live_out = reinterpret_cast<float2 *>(outb + 12 * T);
    uint8_t *wv_out = outb + 20 * T;
    const int t = threadIdx.x;
    if (reset_frame && blockIdx.x == 0 && t == 0) {
        *total_num_calls += 1u;
        *hit_counter = 0u;
        if (grads >= 0) *grads_enabled = (uint8_t)grads;
    }
    const bool enable_sh = *cfg_enable_sh != 0;
    int degree = *current_sh_degree;
    degree = min(min(degree, 3), max_sh_degree);
    const int nb = enable_sh ? sh_count(degree) : 0;
    const float athr = *cfg_alpha_threshold, pw = *cfg_exp_power;
    const float cam[3] = {cam_origin[0], cam_origin[1], cam_origin[2]};
    if (t == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        mbar_fence_init();
    }
    __syncthreads();
    int tile = blockIdx.x;
    if (t == 0 && tile < tiles)
        prep_issue_loads<SHT>(stages, &bar[0], tile, per, enable_sh, nb > 0, opacity, mean, visible, sh_dc, sh_rest);
    if (blockIdx.x == gridDim.x - 1 && tiles * (int)T + t < n) {
        // the Gaussians past the last full tile, while the block's first tile loads
        const size_t i = (size_t)tiles * T + t;
        const float o = sigmoid_act(opacity[i]);
        live[i] = make_float2(visible[i] ? o : __int_as_float(0xff800000), scaling_factor(o, athr, pw));
        if (enable_sh) {
            const float mu[3] = {mean[3 * i], mean[3 * i + 1], mean[3 * i + 2]};
            float col[3];
            sh_colour<SHT>(mu, cam, sh_dc + 3 * i, sh_rest + (size_t)per * i, nb, col);
#pragma unroll
            for (int c = 0; c < 3; c++) channels[3 * i + c] = col[c];
        }
        if (reset_frame) was_visible[i] = 0;
    }
    int it = 0;
    bool timed_out = false;
    for (; tile < tiles; it++, tile += gridDim.x) {
        const int st = it & 1;
        const int next = tile + gridDim.x;
        if (t == 0 && next < tiles) {
            fence_proxy_async();  // stage st ^ 1 was last read in the previous tile, before its barriers
            prep_issue_loads<SHT>(stages + (st ^ 1) * stage_bytes, &bar[st ^ 1], next, per, enable_sh, nb > 0,
                                  opacity, mean, visible, sh_dc, sh_rest);
        }
        const bool ok = __syncthreads_and(mbar_wait(&bar[st], (uint32_t)(it >> 1) & 1u, kBulkWaitNs));
        if (!ok) {
            if (t == 0) atomicOr(status, GRAY_STATUS_COPY_TIMEOUT);
            timed_out = true;
            break;
        }
        const unsigned char *stg = stages + st * stage_bytes;
        const float o = sigmoid_act(reinterpret_cast<const float *>(stg)[t]);
        const float sf = scaling_factor(o, athr, pw);
        const float2 lv = make_float2(stg[16 * T + t] ? o : __int_as_float(0xff800000), sf);
        float col[3] = {0.0f, 0.0f, 0.0f};
        if (enable_sh) {
            const float *m = reinterpret_cast<const float *>(stg + 4 * T) + 3 * t;
            const float mu[3] = {m[0], m[1], m[2]};
            const SHT *dc = reinterpret_cast<const SHT *>(stg + 17 * T) + 3 * t;
            const SHT *row = reinterpret_cast<const SHT *>(stg + 17 * T + 3 * T * sb) + per * t;
            sh_colour<SHT>(mu, cam, dc, row, nb, col);
        }
        if (t == 0) bulk_wait_read();  // the previous tile's stores have read the output copy
        __syncthreads();
        live_out[t] = lv;
#pragma unroll
        for (int c = 0; c < 3; c++) ch_out[3 * t + c] = col[c];
        wv_out[t] = 0;
        fence_proxy_async();
        __syncthreads();
        if (t == 0) {
            const size_t g0 = (size_t)tile * T;
            bulk_store(live + g0, live_out, 8u * T);
            if (enable_sh) bulk_store(channels + 3 * g0, ch_out, 12u * T);
            if (reset_frame) bulk_store(was_visible + g0, wv_out, T);
            bulk_commit();
        }
    }
    if (t == 0) {
        bulk_wait_all();
        if (timed_out) {
            // bounded waits for the loads still in flight before the block's shared memory goes
            mbar_wait(&bar[it & 1], (uint32_t)(it >> 1) & 1u, kBulkWaitNs);
            if (tile + (int)gridDim.x < tiles)
                mbar_wait(&bar[(it + 1) & 1], (uint32_t)((it + 1) >> 1) & 1u, kBulkWaitNs);
        }
    }
}

template <typename SHT>
static cudaError_t forward_prep_typed(const gray_params &p, bool reset_frame, int grads, cudaStream_t s) {
    const gray_gaussians &g = p.gaussians;
    const int n = g.count, num_rest = g.num_sh_coeffs;
    const SHT *dc = reinterpret_cast<const SHT *>(g.sh_coeffs_dc);
    const SHT *rest = reinterpret_cast<const SHT *>(g.sh_coeffs_rest);
    float2 *live = reinterpret_cast<float2 *>(p.scene.live);
    const uint32_t smem = prep_smem_bytes(num_rest, sizeof(SHT));
    const bool bulk = p.status && smem <= 48u * 1024u && aligned16(g.opacity) && aligned16(g.mean) &&
                      aligned16(p.scene.visible) && aligned16(dc) && (num_rest == 0 || aligned16(rest)) &&
                      aligned16(g.channels) && aligned16(live) && aligned16(g.was_visible);
    const int tiles = bulk ? n / kPrepTile : 0;
    cudaError_t e;
    if (tiles > 0) {
        int sms = 0, per_sm = 0;
        if ((e = resident_blocks(reinterpret_cast<const void *>(&forward_prep_bulk_kernel<SHT>), kPrepTile, smem, &sms,
                                 &per_sm)) != cudaSuccess)
            return e;
        // at most kPrepBlocksPerSm blocks per SM: the forward's tile schedule runs beside this kernel
        // on another stream, and its blocks need shared memory too
        const int want = sms * min(per_sm, kPrepBlocksPerSm);
        forward_prep_bulk_kernel<SHT><<<tiles < want ? tiles : want, kPrepTile, smem, s>>>(
            n, tiles, num_rest, g.opacity, p.scene.visible, p.config.alpha_threshold, p.config.exp_power,
            p.config.enable_sh, g.current_sh_degree, g.max_sh_degree, g.mean, p.camera.origin, dc, rest, g.channels,
            live, g.was_visible, p.metadata.total_num_calls, p.hitlist.total_words, p.metadata.grads_enabled, grads,
            reset_frame ? 1 : 0, p.status);
        return cudaGetLastError();
    }
    const size_t staged = (size_t)kPrepThreads * (size_t)(num_rest > 0 ? num_rest : 1) * 3 * sizeof(SHT);
    forward_prep_kernel<SHT><<<blocks_for(n, kPrepThreads), kPrepThreads, staged, s>>>(
        n, num_rest, g.opacity, p.scene.visible, p.config.alpha_threshold, p.config.exp_power, p.config.enable_sh,
        g.current_sh_degree, g.max_sh_degree, g.mean, p.camera.origin, dc, rest, g.channels, live, g.was_visible,
        p.metadata.total_num_calls, p.hitlist.total_words, p.metadata.grads_enabled, grads, reset_frame ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_forward_prep(const gray_params &p, bool reset_frame, int grads, cudaStream_t s) {
    const gray_gaussians &g = p.gaussians;
    if (reset_frame && g.count <= 0) {
        // still count the call and empty the hit list
        cudaError_t e = cudaMemsetAsync(p.hitlist.total_words, 0, sizeof(uint32_t), s);
        if (e == cudaSuccess && grads >= 0) e = cudaMemsetAsync(p.metadata.grads_enabled, grads, 1, s);
        return e;
    }
    if (g.count <= 0) return cudaSuccess;
    return g.sh_is_fp16 ? forward_prep_typed<__half>(p, reset_frame, grads, s)
                        : forward_prep_typed<float>(p, reset_frame, grads, s);
}

__global__ void set_view_kernel(gray_camera cam, uint8_t *rays_from_python, const float *origin, const float *c2w,
                                float fov, float znear, float zfar, int rays) {
    const int t = threadIdx.x;
    if (t < 3) cam.origin[t] = origin[t];
    if (t < 9) {
        const float r = c2w[t];
        cam.rotation_c2w[t] = r;
        cam.rotation_w2c[3 * (t % 3) + t / 3] = r;
    }
    if (t == 0) {
        *cam.vertical_fov_radians = fov;
        *cam.znear = znear;
        *cam.zfar = zfar;
        *rays_from_python = (uint8_t)rays;
    }
}

cudaError_t launch_set_view(const gray_params &p, const float *origin, const float *c2w, float fov, float znear,
                            float zfar, int rays_from_python, cudaStream_t s) {
    set_view_kernel<<<1, 32, 0, s>>>(p.camera, p.config.rays_from_python, origin, c2w, fov, znear, zfar,
                                     rays_from_python);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Batched preparation: live values once and the SH colour of every Gaussian for each of
// `nviews` camera origins (one pass over the SH coefficients serves all views).  Same
// arithmetic as forward_prep_kernel, so a view's colours are bit-identical to a plain forward.
// ---------------------------------------------------------------------------------------------
template <typename SHT>
__global__ void __launch_bounds__(kPrepThreads) batch_prep_kernel(
    int n, int num_rest, const float *__restrict__ opacity, const uint8_t *__restrict__ visible,
    const float *__restrict__ cfg_alpha_threshold, const float *__restrict__ cfg_exp_power,
    const uint8_t *__restrict__ cfg_enable_sh, const int32_t *__restrict__ current_sh_degree, int max_sh_degree,
    const float *__restrict__ mean, const float *__restrict__ origins, int nviews, const SHT *__restrict__ sh_dc,
    const SHT *__restrict__ sh_rest, const float *__restrict__ channels_in, float *__restrict__ channels_out,
    float2 *__restrict__ live) {
    extern __shared__ float stage[];
    const int i0 = blockIdx.x * kPrepThreads;
    const int i = i0 + threadIdx.x;
    const bool enable_sh = *cfg_enable_sh != 0;
    int degree = min(min(*current_sh_degree, 3), max_sh_degree);
    const int nb = enable_sh ? sh_count(degree) : 0;
    if (nb > 0) {
        const int rows = min(kPrepThreads, n - i0);
        const int per = num_rest * 3;
        const long long base = (long long)i0 * per;
        for (int t = threadIdx.x; t < rows * per; t += kPrepThreads) stage[t] = sh_load<SHT>(sh_rest + base + t);
    }
    __syncthreads();
    if (i >= n) return;
    const float athr = *cfg_alpha_threshold, pw = *cfg_exp_power;
    float o = sigmoid_act(opacity[i]);
    float sf = scaling_factor(o, athr, pw);
    live[i] = make_float2(visible[i] ? o : __int_as_float(0xff800000), sf);
    const float m0 = mean[3 * i], m1 = mean[3 * i + 1], m2 = mean[3 * i + 2];
    const float *row = stage + threadIdx.x * num_rest * 3;
    float dc[3];
#pragma unroll
    for (int c = 0; c < 3; c++) dc[c] = enable_sh ? sh_load<SHT>(sh_dc + 3 * i + c) : 0.0f;
    for (int v = 0; v < nviews; v++) {
        float *out = channels_out + ((size_t)v * n + i) * 3;
        if (!enable_sh) {
            out[0] = channels_in[3 * i];
            out[1] = channels_in[3 * i + 1];
            out[2] = channels_in[3 * i + 2];
            continue;
        }
        const float v0 = m0 - origins[3 * v], v1 = m1 - origins[3 * v + 1], v2 = m2 - origins[3 * v + 2];
        float len2 = v0 * v0 + v1 * v1 + v2 * v2;
        float inv = 1.0f / sqrtf(fmaxf(len2, 1e-20f));
        float b[15];
        sh_basis(v0 * inv, v1 * inv, v2 * inv, b);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float acc = SH_C0 * dc[c];
#pragma unroll
            for (int j = 0; j < 15; j++)
                if (j < nb) acc = fmaf(b[j], row[3 * j + c], acc);
            acc = acc + 0.5f;
            out[c] = fmaxf(acc, 0.0f);
        }
    }
}

cudaError_t launch_batch_prep(const gray_params &p, const float *origins, int nviews, float *channels_out,
                              cudaStream_t s) {
    const gray_gaussians &g = p.gaussians;
    if (g.count <= 0 || nviews <= 0) return cudaSuccess;
    const int num_rest = g.num_sh_coeffs;
    const size_t smem = (size_t)kPrepThreads * (size_t)(num_rest > 0 ? num_rest : 1) * 3 * sizeof(float);
    const unsigned int blocks = blocks_for(g.count, kPrepThreads);
    if (g.sh_is_fp16) {
        batch_prep_kernel<__half><<<blocks, kPrepThreads, smem, s>>>(
            g.count, num_rest, g.opacity, p.scene.visible, p.config.alpha_threshold, p.config.exp_power,
            p.config.enable_sh, g.current_sh_degree, g.max_sh_degree, g.mean, origins, nviews,
            reinterpret_cast<const __half *>(g.sh_coeffs_dc), reinterpret_cast<const __half *>(g.sh_coeffs_rest),
            g.channels, channels_out, reinterpret_cast<float2 *>(p.scene.live));
    } else {
        batch_prep_kernel<float><<<blocks, kPrepThreads, smem, s>>>(
            g.count, num_rest, g.opacity, p.scene.visible, p.config.alpha_threshold, p.config.exp_power,
            p.config.enable_sh, g.current_sh_degree, g.max_sh_degree, g.mean, origins, nviews,
            reinterpret_cast<const float *>(g.sh_coeffs_dc), reinterpret_cast<const float *>(g.sh_coeffs_rest),
            g.channels, channels_out, reinterpret_cast<float2 *>(p.scene.live));
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Gradient fold + SH backward.  The trace backward accumulates per-Gaussian gradients with
// 16-byte vector reductions into grad_acc ([n,16]: sums of q and q x^T, opacity, pruning weight, channels,
// count; replay_hit, trace.cu); this kernel carries them to mean, scale, rotation and opacity
// (fold_geometry), adds them to the reference-layout gradient arrays, sets was_visible, clears grad_acc and
// runs the SH backward for visible Gaussians (reference: sh_backward_kernel, cuda/utils/sh.cu:249-287).
//
// A view composites a part of the Gaussians only (11% at 3M / 1080p, 28% at 1M / 1600x1040), scattered over
// the rows.  A block reads the counts of kFoldScan rows, lists the visible ones and then folds those with
// every lane at work: a warp takes 32 of them, loads all it needs of them at once and moves their
// coefficient rows through shared memory, a row's words by consecutive lanes.  A thread per row had 3.5 of a
// warp's lanes follow the same chain of dependent loads (64 stall cycles per instruction) and wrote
// rows of 180 bytes word by word: 3M / 1080p 289 -> 140 us, 1M / 1600x1040 118 -> 79 us (176 and 93 since the
// geometric gradients are made here, which took 94 and 33 us of records and more from the replay).
// ---------------------------------------------------------------------------------------------
constexpr int kFoldThreads = 128;
constexpr int kFoldScan = 512;  // rows per block (1024: 1M 91 instead of 79 us; 256: 3M 165 instead of 140)
constexpr int kFoldRow = 45;     // words of a coefficient row at degree 3 (an odd stride: no bank conflicts)
constexpr int kFoldRows = 8;     // coefficient rows a warp loads at a time

// The geometric gradients of one Gaussian from its sums: with M (rows g0..g2) the world-to-object matrix, L
// the rows of the object-to-world one, x = sf u and s = exp(scale),
//   d/d mean = sf M^T sum(q),  d/d L = G = sf M^T sum(q x^T),
//   d/d scale_k = sum_r G_rk L_rk s_k / (s_k sf + eps)  (cuda/backward_pass.cu:101-111),
// and the rotation's is that of R = (G_rk s_k) pulled back to the quaternion through its normalisation
// (cuda/utils/activations.cu:68-70: (g - (g . qn) qn) / |q|).
struct FoldGeometry {
    float4 rot;
    float mean[3], scale[3];
};

__device__ __forceinline__ FoldGeometry fold_geometry(float4 a0, float4 a1, float4 a2, const float4 *__restrict__ g,
                                                      const float4 *__restrict__ l, float sf, const float ls[3],
                                                      float4 rotation, float eps) {
    const float M[3][3] = {{g[0].x, g[0].y, g[0].z}, {g[1].x, g[1].y, g[1].z}, {g[2].x, g[2].y, g[2].z}};
    const float L[3][3] = {{l[0].x, l[0].y, l[0].z}, {l[1].x, l[1].y, l[1].z}, {l[2].x, l[2].y, l[2].z}};
    const float q[3] = {a0.x, a0.y, a0.z};
    const float S[3][3] = {{a1.x, a1.y, a1.z}, {a1.y, a1.w, a2.x}, {a1.z, a2.x, a2.y}};
    FoldGeometry o;
    float R[3][3];
#pragma unroll
    for (int r = 0; r < 3; r++) o.mean[r] = (M[0][r] * q[0] + M[1][r] * q[1] + M[2][r] * q[2]) * sf;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float s = gexp(ls[k]), d = s * sf + eps;
        float acc = 0.0f;
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const float G = (M[0][r] * S[0][k] + M[1][r] * S[1][k] + M[2][r] * S[2][k]) * sf;
            acc = acc + G * (L[r][k] / d * s);
            R[r][k] = G * s;
        }
        o.scale[k] = acc;
    }
    const float qlen = sqrtf(rotation.x * rotation.x + rotation.y * rotation.y + rotation.z * rotation.z +
                             rotation.w * rotation.w);
    const float iq = 1.0f / qlen;
    const float qw = rotation.x / qlen, qx = rotation.y / qlen, qy = rotation.z / qlen, qz = rotation.w / qlen;
    const float g_r = 2.0f * qx * (R[2][1] - R[1][2]) + 2.0f * qy * (R[0][2] - R[2][0]) + 2.0f * qz * (R[1][0] - R[0][1]);
    const float g_x = -4.0f * qx * (R[1][1] + R[2][2]) + 2.0f * qy * (R[0][1] + R[1][0]) +
                      2.0f * qz * (R[0][2] + R[2][0]) + 2.0f * qw * (R[2][1] - R[1][2]);
    const float g_y = 2.0f * qx * (R[0][1] + R[1][0]) - 4.0f * qy * (R[0][0] + R[2][2]) +
                      2.0f * qz * (R[1][2] + R[2][1]) + 2.0f * qw * (R[0][2] - R[2][0]);
    const float g_z = 2.0f * qx * (R[0][2] + R[2][0]) + 2.0f * qy * (R[1][2] + R[2][1]) -
                      4.0f * qz * (R[0][0] + R[1][1]) + 2.0f * qw * (R[1][0] - R[0][1]);
    const float dq = g_r * qw + g_x * qx + g_y * qy + g_z * qz;
    o.rot = make_float4((g_r - dq * qw) * iq, (g_x - dq * qx) * iq, (g_y - dq * qy) * iq, (g_z - dq * qz) * iq);
    return o;
}

__global__ void __launch_bounds__(kFoldThreads) fold_sh_backward_kernel(
    int n, int num_rest, float4 *__restrict__ grad_acc, float4 *__restrict__ grad_rotation,
    float *__restrict__ grad_mean, float *__restrict__ grad_opacity, float *__restrict__ grad_scale,
    float *__restrict__ pruning_weight, float *__restrict__ grad_channels, uint8_t *__restrict__ was_visible,
    const uint8_t *__restrict__ cfg_enable_sh, const int32_t *__restrict__ current_sh_degree, int max_sh_degree,
    const float *__restrict__ mean, const float *__restrict__ cam_origin, const float *__restrict__ sh_rest,
    const float *__restrict__ channels, float *__restrict__ grad_sh_dc, float *__restrict__ grad_sh_rest,
    const float4 *__restrict__ geom, const float4 *__restrict__ l2w, const float2 *__restrict__ live,
    const float *__restrict__ scale, const float4 *__restrict__ rotation, const float *__restrict__ eps_scale_grad) {
    __shared__ float s_rows[kFoldThreads * kFoldRow];
    __shared__ uint16_t s_list[kFoldScan];
    __shared__ int s_count;
    const int t = threadIdx.x, lane = t & 31;
    const int base = blockIdx.x * kFoldScan;
    if (t == 0) s_count = 0;
    float w[kFoldScan / kFoldThreads];
#pragma unroll
    for (int k = 0; k < kFoldScan / kFoldThreads; k++) {
        const int i = base + k * kFoldThreads + t;
        w[k] = i < n ? grad_acc[4 * (size_t)i + 3].w : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kFoldScan / kFoldThreads; k++) {
        const bool vis = w[k] > 0.0f;  // untouched accumulator rows are already zero
        const uint32_t bal = __ballot_sync(0xffffffffu, vis);
        int at = 0;
        if (lane == 0 && bal) at = atomicAdd(&s_count, __popc(bal));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (vis) s_list[at + __popc(bal & ((1u << lane) - 1u))] = (uint16_t)(k * kFoldThreads + t);
    }
    __syncthreads();
    const int count = s_count;
    const bool sh = *cfg_enable_sh != 0;
    const int nb = sh ? sh_count(min(min(*current_sh_degree, 3), max_sh_degree)) : 0, words = 3 * nb;
    const size_t per = 3 * (size_t)num_rest;
    float *const rows = s_rows + (t & ~31) * kFoldRow;
    for (int c0 = t & ~31; c0 < count; c0 += kFoldThreads) {
        const bool on = c0 + lane < count;
        const int i = base + (on ? (int)s_list[c0 + lane] : 0);
        float4 a0, a1, a2, a3, gr, mr[3], lr[3], rot;
        float2 lv;
        float gm[3], gs[3], gc[3], m[3], col[3], ls[3], go = 0.0f, gp = 0.0f;
        if (on) {
            a0 = grad_acc[4 * (size_t)i];
            a1 = grad_acc[4 * (size_t)i + 1];
            a2 = grad_acc[4 * (size_t)i + 2];
            a3 = grad_acc[4 * (size_t)i + 3];
            gr = grad_rotation[i];
            go = grad_opacity[i];
            gp = pruning_weight[i];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                gm[k] = grad_mean[3 * (size_t)i + k];
                gs[k] = grad_scale[3 * (size_t)i + k];
                gc[k] = grad_channels[3 * (size_t)i + k];
                m[k] = sh ? mean[3 * (size_t)i + k] : 0.0f;
                col[k] = sh ? channels[3 * (size_t)i + k] : 0.0f;
                mr[k] = geom[3 * (size_t)i + k];
                lr[k] = l2w[3 * (size_t)i + k];
                ls[k] = scale[3 * (size_t)i + k];
            }
            rot = rotation[i];
            lv = live[i];
        }
        if (nb > 0) {
            for (int r0 = 0; r0 < 32 && c0 + r0 < count; r0 += kFoldRows) {
                float lo[kFoldRows], hi[kFoldRows];
#pragma unroll
                for (int r = 0; r < kFoldRows; r++) {
                    const float *row = sh_rest + per * (size_t)__shfl_sync(0xffffffffu, i, r0 + r);
                    lo[r] = lane < words ? row[lane] : 0.0f;
                    hi[r] = lane + 32 < words ? row[lane + 32] : 0.0f;
                }
#pragma unroll
                for (int r = 0; r < kFoldRows; r++) {
                    if (lane < words) rows[(r0 + r) * kFoldRow + lane] = lo[r];
                    if (lane + 32 < words) rows[(r0 + r) * kFoldRow + lane + 32] = hi[r];
                }
            }
            __syncwarp();
        }
        if (on) {
            const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            grad_acc[4 * (size_t)i] = z;
            grad_acc[4 * (size_t)i + 1] = z;
            grad_acc[4 * (size_t)i + 2] = z;
            grad_acc[4 * (size_t)i + 3] = z;
            was_visible[i] = 1;
            const FoldGeometry f = fold_geometry(a0, a1, a2, mr, lr, lv.y, ls, rot, *eps_scale_grad);
            grad_rotation[i] = make_float4(gr.x + f.rot.x, gr.y + f.rot.y, gr.z + f.rot.z, gr.w + f.rot.w);
            grad_opacity[i] = go + a0.w * lv.x * (1.0f - lv.x);
            pruning_weight[i] = gp + a2.z;
            gc[0] = gc[0] + a3.x;
            gc[1] = gc[1] + a3.y;
            gc[2] = gc[2] + a3.z;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                gm[k] = gm[k] + f.mean[k];
                grad_scale[3 * (size_t)i + k] = gs[k] + f.scale[k];
            }
#pragma unroll
            for (int c = 0; c < 3; c++) grad_channels[3 * (size_t)i + c] = gc[c];
            if (sh) {
                float v[3], g[3];
#pragma unroll
                for (int k = 0; k < 3; k++) v[k] = m[k] - cam_origin[k];
                const float len2 = fmaxf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2], 1e-20f);
                const float inv = 1.0f / sqrtf(len2);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    g[c] = col[c] <= 0.0f ? 0.0f : gc[c];
                    grad_sh_dc[3 * (size_t)i + c] = SH_C0 * g[c];
                }
                if (nb > 0) {
                    const float x = v[0] * inv, y = v[1] * inv, zc = v[2] * inv;
                    float b[15], dx[15], dy[15], dz[15];
                    sh_basis(x, y, zc, b);
                    sh_basis_grad(x, y, zc, dx, dy, dz);
                    float gd0 = 0.0f, gd1 = 0.0f, gd2 = 0.0f;
                    float *row = rows + lane * kFoldRow;  // coefficients in, gradients out
#pragma unroll
                    for (int j = 0; j < 15; j++) {
                        if (j < nb) {
                            const float q = row[3 * j] * g[0] + row[3 * j + 1] * g[1] + row[3 * j + 2] * g[2];
                            row[3 * j] = b[j] * g[0];
                            row[3 * j + 1] = b[j] * g[1];
                            row[3 * j + 2] = b[j] * g[2];
                            gd0 = fmaf(dx[j], q, gd0);
                            gd1 = fmaf(dy[j], q, gd1);
                            gd2 = fmaf(dz[j], q, gd2);
                        }
                    }
                    const float inv3 = inv * inv * inv;
                    const float dv = v[0] * gd0 + v[1] * gd1 + v[2] * gd2;
                    gm[0] = gm[0] + (gd0 * inv - v[0] * (dv * inv3));
                    gm[1] = gm[1] + (gd1 * inv - v[1] * (dv * inv3));
                    gm[2] = gm[2] + (gd2 * inv - v[2] * (dv * inv3));
                }
            }
#pragma unroll
            for (int k = 0; k < 3; k++) grad_mean[3 * (size_t)i + k] = gm[k];
        }
        if (nb > 0) {
            __syncwarp();
            const int left = min(32, count - c0);
#pragma unroll 4
            for (int r = 0; r < left; r++) {
                float *row = grad_sh_rest + per * (size_t)__shfl_sync(0xffffffffu, i, r);
                if (lane < words) row[lane] = rows[r * kFoldRow + lane];
                if (lane + 32 < words) row[lane + 32] = rows[r * kFoldRow + lane + 32];
            }
            __syncwarp();
        }
    }
}

cudaError_t launch_fold_and_sh_backward(const gray_params &p, cudaStream_t s) {
    const gray_gaussians &g = p.gaussians;
    if (g.count <= 0) return cudaSuccess;
    fold_sh_backward_kernel<<<blocks_for(g.count, kFoldScan), kFoldThreads, 0, s>>>(
        g.count, g.num_sh_coeffs, reinterpret_cast<float4 *>(p.scene.grad_acc),
        reinterpret_cast<float4 *>(g.grad_rotation), g.grad_mean, g.grad_opacity, g.grad_scale, g.pruning_weight,
        g.grad_channels, g.was_visible, p.config.enable_sh, g.current_sh_degree, g.max_sh_degree, g.mean,
        p.camera.origin, reinterpret_cast<const float *>(g.sh_coeffs_rest), g.channels, g.grad_sh_coeffs_dc,
        g.grad_sh_coeffs_rest, reinterpret_cast<const float4 *>(p.scene.geom),
        reinterpret_cast<const float4 *>(p.scene.l2w), reinterpret_cast<const float2 *>(p.scene.live), g.scale,
        reinterpret_cast<const float4 *>(g.rotation), p.config.eps_scale_grad);
    return cudaGetLastError();
}

}  // namespace gray
