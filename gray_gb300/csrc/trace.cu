// trace.cu -- forward and backward ray tracing of the Gaussians on the LBVH.
//
// Forward (replaces the OptiX launch of cuda/shaders.cu:69-106 with cuda/forward_pass.cu):
//   A block renders an 8x16-pixel tile of rays that share one origin, each warp a 4x8 (or 8x4)
//   pixel packet of it.  A per-tile kernel first walks the top of the BVH with the tile's frustum and
//   records the tile's frontier (the nodes of at most 16 to 64 leaves it reaches, sorted front to back);
//   the block's traversal starts there.  The block traverses as one frustum: each step pops up to
//   128 nodes (one per thread) from a shared-memory stack, tests both child boxes against the
//   frustum, pushes the nearer child last and queues leaves.  Queued leaves are taken in batches of
//   128: culled by an exact ellipsoid-frustum test and cached in shared memory with the conic their
//   support sphere projects to on the tile's pixels; every ray evaluates the conics at its pixel (a
//   conservative pretest of five FMAs) and the lanes then walk their masks of possible hits through
//   the intersection program of cuda/shaders.cu:10-67, which decides each hit.  The first traversal
//   accumulates, over ALL hits, the full transmittance
//   (an order-independent fixed-point sum of log(1 - alpha)) and the alpha-weighted colour sums of
//   the reference's truncated-tail estimate, and every traversal keeps the KB nearest hits above a
//   resume key in a per-lane shared-memory buffer of 64-bit keys (fp16 distance | gaussian id |
//   fp16 alpha).  The buffer is consumed by a state machine that reproduces the reference's
//   32-slot multi-pass selection exactly (pass boundaries, the strict `distance > tmin` drop of
//   equal distances, the 99-pass cap, zfar, t_threshold).  Composited ids are appended to the
//   backward hit list in warp-aggregated segments.  Jittered rays, and rays from the caller that share
//   their tile's origin within a cone (ray_cone), go the same way; other rays from the caller, and
//   tiles whose traversal overflows the shared stack, take a per-ray slab traversal instead.
// Backward (cuda/backward_pass.cu:2-142): one thread per pixel walks its segments back to front,
//   recomputes alpha in fp32 and adds the hit's 14 gradient sums and its count to the per-Gaussian
//   accumulator: lanes holding the same Gaussian combine in a tree, and the lowest issues four
//   16-byte vector reductions.
#include "gray_device.cuh"
#include "gray_internal.h"

namespace gray {

constexpr int kBlockWarpsX = 2, kBlockWarpsY = 2;  // 2x2 warp tiles per block
constexpr int kWarps = kBlockWarpsX * kBlockWarpsY;
constexpr int kFwdThreads = kWarps * 32;
constexpr int kStackWords = 2;               // warp-uniform stack of 64 entries in 2 registers per lane
constexpr int kStackMax = 32 * kStackWords;
constexpr int kPassSlots = 32;               // BUFFER_SIZE, cuda/forward_pass.cu:4
constexpr int kMaxPasses = 99;               // MAX_ITERATIONS, cuda/forward_pass.cu:3
constexpr int kMaxTraversals = 4 * kMaxPasses * 2;  // bound on re-traversals of one ray
constexpr unsigned kFull = 0xffffffffu;
constexpr int kBatch = 128;       // leaves fetched and tested together by a block (one per thread)
constexpr int kTileStack = 448;   // per-block traversal stack
constexpr int kSplitStack = 1536;  // of a block that traces a split tile's packet
constexpr int kStackReserve = 72;  // entries left to a depth-first descent (deeper than any tree)
constexpr int kTileQueue = kBatch + 2 * kFwdThreads;  // queued leaves: < kBatch before a step, + up to 2 per thread
static_assert(kBatch == kFwdThreads, "one leaf per thread");
constexpr int kSchedHeader = 64;  // schedule words before the per-tile estimates
constexpr int kSchedItems = 1;       // header word: tiles of the work order
constexpr int kSchedSplitNext = 2;   // work counter of the split tiles' packets
constexpr int kSchedSplitItems = 3;  // packets of split tiles
constexpr int kSchedRays = 4;        // tiles whose rays are traversed one by one (see kRayTile)
constexpr int kSchedRayNext = 5;     // work counter of their packets
constexpr uint32_t kRayTile = 0xffffffffu;  // estimate of such a tile
constexpr int kItemShift = 29;       // a split tile's packet: its tile, and the packet from this bit on
constexpr uint32_t kItemTile = (1u << kItemShift) - 1u;
constexpr int kOrderPerTile = 5;     // words of the work order per tile: itself, or its four packets
// Header words [kStatPackets, kStatChoice] outlive a forward: the automatic kernel choice (see
// plan_forward) keeps there the packet counts of the last scheduled forward and the choice the order
// kernel made from them.
constexpr int kStatPackets = 48;   // packets traced by the last scheduled forward
constexpr int kStatRetraced = 49;  // of them, packets that need more than one traversal with 16 slots
constexpr int kStatChoice = 50;    // kernel of the automatic choice: kChoiceNarrow or kChoiceWide
constexpr uint32_t kChoiceNarrow = 1u, kChoiceWide = 2u;
// The wide kernel (32 hit slots, four blocks per SM) is chosen when more than kWideLarge / 128 of the last
// forward's packets need more than one traversal with 16 slots (counted the same way by both kernels,
// so the choice does not depend on which one ran), the narrow one (16 slots, five blocks per SM)
// otherwise; with at most kWideTiles tiles per resident block, more than kWideSmall / 128.  A second
// traversal is repeated by the packet's whole tile, and in a small frame it is the launch's tail.  Measured,
// narrow against wide: 3M / 1080p with 5% of the packets 2.88 and 3.12 ms, with 31-38% 2.7-3.7 and 2.0-2.4;
// 1M / 1600x1040, 17-20%, 1.15-1.25 and 0.98-1.07; 500k / 1280x720 (7 tiles per block), 5.5-8.5%, 0.52-0.76
// and 0.46-0.53; 300k / 800x600, 1.5-3%, 0.36-0.50 and 0.28-0.32; equal within 3% where none or almost
// none do (100k / 320x240, 64 Gaussians / 256x256).
constexpr uint32_t kWideLarge = 10u, kWideSmall = 1u;
constexpr int kWideTiles = 8;
// Per pixel tile, or group of a batch, kFrontierWords words: the BVH frontier its frustum reaches (a count, then
// up to kFrontierMax node or leaf entries), and three that a batch uses: the group's estimate and, in slot
// i, entry i of the batch's work order (in slot 0 also whether there is one).  A count of kFrontierNone
// means "start at the root".  A frontier goes onto the traversal stack, so it leaves room there for the
// traversal's own pushes.
constexpr int kFrontierWords = GRAY_FRONTIER_WORDS;
constexpr int kFrontierMax = kFrontierWords - 4;
constexpr uint32_t kFrontierNone = 0xFFFFFFFFu;
constexpr int kBatchOrdered = kFrontierWords - 3, kBatchEst = kFrontierWords - 2, kBatchOrder = kFrontierWords - 1;
constexpr int kFrontierSort = 256;  // sort buffer of the frontier walk (a power of two > kFrontierMax)
constexpr int kFrontierCutDefault = 64;  // frontier nodes hold at most this many leaves

struct FwdArgs {
    uint32_t alloc_w, render_w, render_h;
    int n;
    int tile_w, tile_h;  // pixels of one warp packet (tile_w * tile_h == 32)
    const float *cam_origin, *fov, *w2c, *znear, *zfar;
    const float *exp_power, *alpha_threshold, *t_threshold, *eps_fwd, *bg;
    const uint8_t *render_depth, *needs_ray_output, *rays_from_python, *jitter, *grads_enabled;
    const uint8_t *render_ellipsoids;
    const float *ellipsoid_min_opacity;
    int display;  // forward_pass_display: colour only, whatever grads_enabled holds
    int auto_role;  // 0, or kChoiceNarrow / kChoiceWide: the launch of the automatic choice this is
    uint32_t *schedule;  // work order of the pixel tiles (null: tiles in launch order)
    int tiles_x, ntiles;
    int slots_split;  // blocks of the split kernel resident at once
    uint32_t *frontier;  // per-tile BVH frontiers (null: packets start at the root)
    uint32_t frontier_cut;
    uint32_t *super_frontier;  // per super-tile coarse frontiers seeding the tile walks (null: root)
    int super_x;               // super-tiles per row
    const uint32_t *total_num_calls;
    const float4 *geom, *l2w;
    const float2 *live;
    const float *channels;
    const float4 *nodes;
    const float *root_box;
    float *out_rgb, *out_depth, *out_T, *out_fullT, *out_rem, *ray_o, *ray_d;
    int32_t *stat_hit, *stat_acc;
    uint32_t *head, *counter, *pool;
    uint32_t pool_size;
    int32_t *status;
};

// PCG32 output hash (O'Neill 2014) for the optional sub-pixel jitter.
__device__ __forceinline__ uint32_t pcg_hash(uint32_t v) {
    uint32_t state = v * 747796405u + 2891336453u;
    uint32_t word = ((state >> ((state >> 28u) + 4u)) ^ state) * 277803737u;
    return (word >> 22u) ^ word;
}

// Ray against an axis-aligned box widened by the ray's rounding margin eps:
// t = (b -/+ eps - o) * inv computed as fma(b, inv, c) with c_lo = -(o + eps) inv, c_hi = (eps - o) inv.
struct SlabRay {
    f3 inv, clo, chi;
};

__device__ __forceinline__ SlabRay make_slab_ray(f3 ro, f3 rd, float eps) {
    SlabRay r;
    float dx = fabsf(rd.x) < 1e-20f ? (rd.x < 0.0f ? -1e-20f : 1e-20f) : rd.x;
    float dy = fabsf(rd.y) < 1e-20f ? (rd.y < 0.0f ? -1e-20f : 1e-20f) : rd.y;
    float dz = fabsf(rd.z) < 1e-20f ? (rd.z < 0.0f ? -1e-20f : 1e-20f) : rd.z;
    r.inv = mk3(1.0f / dx, 1.0f / dy, 1.0f / dz);
    r.clo = mk3(-(ro.x + eps) * r.inv.x, -(ro.y + eps) * r.inv.y, -(ro.z + eps) * r.inv.z);
    r.chi = mk3((eps - ro.x) * r.inv.x, (eps - ro.y) * r.inv.y, (eps - ro.z) * r.inv.z);
    return r;
}

__device__ __forceinline__ bool slab_hit(const float bmin[3], const float bmax[3], const SlabRay &r) {
    float ta = fmaf(bmin[0], r.inv.x, r.clo.x), tb = fmaf(bmax[0], r.inv.x, r.chi.x);
    float tn = fminf(ta, tb), tf = fmaxf(ta, tb);
    ta = fmaf(bmin[1], r.inv.y, r.clo.y);
    tb = fmaf(bmax[1], r.inv.y, r.chi.y);
    tn = fmaxf(tn, fminf(ta, tb));
    tf = fminf(tf, fmaxf(ta, tb));
    ta = fmaf(bmin[2], r.inv.z, r.clo.z);
    tb = fmaf(bmax[2], r.inv.z, r.chi.z);
    tn = fmaxf(tn, fminf(ta, tb));
    tf = fminf(tf, fmaxf(ta, tb));
    return tn <= tf && tf >= 0.0f;
}

struct LaneState {
    // all-hit accumulators (first traversal only); ft is set from lfx when the ray finishes
    long long lfx;
    float ft;
    long long afx, cfx0, cfx1, cfx2;
    int nhit;
    // selection buffer of the current traversal
    int kcount, ncand;
    unsigned long long kmax;
    float dfar;  // +inf, or once the buffer is full the fp16 distance after its last key's: a hit beyond it
                 // rounds to a larger distance than every kept key's (+inf too where the last key's distance
                 // is -0, which a negative znear keeps: keys order it after every other)
    // resume key for the next traversal
    unsigned long long resume;
    bool has_resume;
};

// What one ray traces against.
struct TraceScene {
    const float4 *geom;
    const float4 *l2w;  // rows (L | mu) for the leaf cull of the frustum traversal (may be null)
    const float2 *live;
    const float *channels;
    const float4 *nodes;
    const float *root_box;
    int n;
};

struct TraceKnobs {
    float znear, zfar, athr, pw, tthr;
    bool render_depth;
};

// Backward hit list sink (counter == nullptr: do not record).
struct HitSink {
    uint32_t *counter, *pool;
    uint32_t pool_size;
};

struct RayResult {
    float T, C0, C1, C2, depth;
    LaneState st;
    int nacc;
    uint32_t head;
    bool retraced;  // the packet traversed, or with 16 hit slots would have traversed, more than once
};

// Intersection program + all-hit sums + selection for one (ray, Gaussian) pair whose snapshot rows,
// live values and colour the caller has fetched.
// LO: the rows' w column holds the object-space origin (local_origin) instead of the mean.
template <int KB, bool LO = false>
__device__ __forceinline__ void on_leaf_data(uint32_t gid, const float4 g0, const float4 g1, const float4 g2,
                                             const float2 lv, int cf0, int cf1, int cf2, bool first, f3 ro, f3 rd,
                                             const TraceKnobs &k, LaneState &st,
                                             unsigned long long (*kbuf)[kFwdThreads]) {
    float dist, alpha;
    if constexpr (LO) {
        if (!intersect_lo(g0, g1, g2, lv.x, lv.y, rd, k.pw, k.znear, k.zfar, dist, alpha)) return;
    } else {
        if (!intersect(g0, g1, g2, lv.x, lv.y, ro, rd, k.athr, k.pw, k.znear, k.zfar, dist, alpha)) return;
    }
    const uint16_t a16 = f2h_bits(alpha);
    if (first) {
        add_log_transmittance(st.lfx, alpha);
        const long long a = alpha16_fixed(a16);
        st.afx += a;
        st.cfx0 += mul_fixed(a, cf0);
        st.cfx1 += mul_fixed(a, cf1);
        st.cfx2 += mul_fixed(a, cf2);
        st.nhit++;
    }
    if (dist > st.dfar) {  // beyond every key of a full buffer
        st.ncand++;
        return;
    }
    const uint16_t d16 = f2h_bits(dist);
    if (!(h2f_bits(d16) > k.znear)) return;
    const unsigned long long key =
        ((unsigned long long)d16 << 48) | ((unsigned long long)gid << 16) | (unsigned long long)a16;
    if (st.has_resume && !(key > st.resume)) return;
    st.ncand++;
    const int t = threadIdx.x;
    int pos;
    if (st.kcount < KB) {
        pos = st.kcount++;
    } else if (key < st.kmax) {
        pos = KB - 1;
    } else {
        return;
    }
    while (pos > 0) {
        unsigned long long prev = kbuf[pos - 1][t];
        if (prev < key) break;
        kbuf[pos][t] = prev;
        pos--;
    }
    kbuf[pos][t] = key;
    if (st.kcount == KB) {
        st.kmax = kbuf[KB - 1][t];
        st.dfar = h2f_bits((uint16_t)min((uint32_t)(st.kmax >> 48) + 1u, 0x7c00u));
    }
}

template <int KB>
__device__ __forceinline__ void on_leaf(const TraceScene &sc, uint32_t gid, bool want, bool first, f3 ro, f3 rd,
                                        const TraceKnobs &k, LaneState &st, unsigned long long (*kbuf)[kFwdThreads]) {
    if (!want) return;
    // every load up front (the colour too): one memory round trip per hit
    const float4 g0 = sc.geom[3 * gid], g1 = sc.geom[3 * gid + 1], g2 = sc.geom[3 * gid + 2];
    const float2 lv = sc.live[gid];
    const float *cp = sc.channels + 3 * (size_t)gid;
    on_leaf_data<KB>(gid, g0, g1, g2, lv, colour_fixed(cp[0]), colour_fixed(cp[1]), colour_fixed(cp[2]), first, ro,
                     rd, k, st, kbuf);
}

__device__ __forceinline__ void stack_push(uint32_t &stk0, uint32_t &stk1, int &sp, uint32_t v, int lane,
                                           int32_t *status) {
    if (sp < kStackMax) {
        if (lane == (sp & 31)) {
            if ((sp >> 5) == 0) stk0 = v;
            else stk1 = v;
        }
        sp++;
    } else {
        raise_status(status, GRAY_STATUS_STACK_OVERFLOW);
    }
}

// Frustum of a packet of primary rays sharing one origin o: four side planes through the origin and
// the plane through the origin orthogonal to the packet's mean direction (nothing behind it can be
// hit).  Normals n point inside.  Stored per warp in shared memory as per-plane constants of the
// two tests below: pn[p] = (n, box threshold), pa[p] = (|n|, ellipsoid threshold).
struct Frustum {
    float4 pn[5];
    float4 pa[5];
};

// Frustum of the rays through the pixels [x0, x1] x [y0, y1] of a pinhole camera: the rays of the
// corner pixels span a convex cone that contains every ray of the rectangle.  root_box bounds every
// box and mean the tests will see, which bounds their rounding error: with M the largest finite
// coordinate magnitude of the root box, the tests' sums have magnitude at most |n|_1 (4M + 2|o|_1)
// and a few roundings of 2^-24 each; the thresholds leave 1e-5 of that (about 170 roundings).
// Boxes with an infinite or NaN coordinate (beyond M) give an infinite or NaN sum and always pass.
__device__ __forceinline__ float3 camera_ray3(const float *w, float fov, int px, int py, uint32_t width,
                                              uint32_t height, float jx, float jy);

// Plane e of the frustum (e < 4: the side through corner rays e and e+1; e = 4: the near plane
// orthogonal to the corners' sum).
__device__ __forceinline__ void frustum_plane(int e, f3 o, const f3 d[4], const float *root_box, float4 &pn,
                                              float4 &pa) {
    const f3 sum = mk3(d[0].x + d[1].x + d[2].x + d[3].x, d[0].y + d[1].y + d[2].y + d[3].y,
                       d[0].z + d[1].z + d[2].z + d[3].z);
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const float v = fabsf(root_box[i]);
        if (i != 3 && i != 7 && v <= 0x1.fffffep127f) m = fmaxf(m, v);
    }
    const float o1 = fabsf(o.x) + fabsf(o.y) + fabsf(o.z);
    f3 nn = sum;
    if (e < 4) {
        // a x b as a x (b - a): exact differences of neighbouring rays, so that the normal's rounding is
        // relative to its own length and the plane holds both rays however narrow the cone is
        const f3 a = d[e], c = d[(e + 1) & 3], b = mk3(c.x - a.x, c.y - a.y, c.z - a.z);
        nn = mk3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
        if (dot3(nn, sum) < 0.0f) nn = mk3(-nn.x, -nn.y, -nn.z);
    }
    const float n1 = fabsf(nn.x) + fabsf(nn.y) + fabsf(nn.z);
    const float no = fdot3(nn, o);
    const float mbox = 1e-5f * n1 * (4.0f * m + 2.0f * o1) + 1e-30f;
    const float mell = 1e-5f * n1 * (3.0f * m + o1) + 1e-30f;
    pn = make_float4(nn.x, nn.y, nn.z, 2.0f * no - mbox);
    pa = make_float4(fabsf(nn.x), fabsf(nn.y), fabsf(nn.z), no - mell);
}

// The frustum built by a whole warp (every lane calls this): lanes 0-3 trace one corner ray each,
// lanes 0-4 write one plane each.  wide: the rays pass up to this many pixels beyond the pixels' centres.
__device__ __forceinline__ void make_frustum_warp(Frustum &fr, f3 o, const float *w2c, float fov, int x0, int y0,
                                                  int x1, int y1, uint32_t width, uint32_t height,
                                                  const float *root_box, float wide = 0.0f) {
    const int lane = threadIdx.x & 31;
    float3 dl = make_float3(0.0f, 0.0f, 0.0f);
    if (lane < 4) {
        const bool right = lane == 1 || lane == 2, low = lane >= 2;
        dl = camera_ray3(w2c, fov, right ? x1 : x0, low ? y1 : y0, width, height, right ? wide : -wide,
                         low ? wide : -wide);
    }
    f3 d[4];
#pragma unroll
    for (int e = 0; e < 4; e++)
        d[e] = mk3(__shfl_sync(0xffffffffu, dl.x, e), __shfl_sync(0xffffffffu, dl.y, e), __shfl_sync(0xffffffffu, dl.z, e));
    if (lane < 5) frustum_plane(lane, o, d, root_box, fr.pn[lane], fr.pa[lane]);
    __syncwarp();
}

// Conservative box-frustum test: false only when the box lies entirely outside one plane by more
// than a rounding margin.  The box's largest signed distance along n, times two, is
// n.(bmin + bmax) + |n|.(bmax - bmin) - 2 n.o.  A NaN never culls.
__device__ __forceinline__ bool frustum_box(const Frustum &fr, const float bmin[3], const float bmax[3]) {
    const float sx = bmin[0] + bmax[0], sy = bmin[1] + bmax[1], sz = bmin[2] + bmax[2];
    const float dx = bmax[0] - bmin[0], dy = bmax[1] - bmin[1], dz = bmax[2] - bmin[2];
#pragma unroll
    for (int p = 0; p < 5; p++) {
        const float4 n = fr.pn[p], a = fr.pa[p];
        const float v = fmaf(a.z, dz, fmaf(a.y, dy, fmaf(a.x, dx, fmaf(n.z, sz, fmaf(n.y, sy, n.x * sx)))));
        if (v < n.w) return false;
    }
    return true;
}

// Conservative frustum test of a Gaussian's support ellipsoid {mu + L u : |u| <= 1} (L, mu = the
// snapshot's l2w rows): false only when the ellipsoid lies outside one plane by more than a rounding
// margin.  The ellipsoid's extent along a normal n is |L^T n| (taken 3e-5 larger for its own
// rounding), compared squared with the gap between the plane's threshold and the centre's signed
// distance (no square root; a gap below 2^-60, so that its square stays a normal float, an
// infinite extent or a NaN never culls).
// A ray can only hit a Gaussian whose ellipsoid it crosses, so a leaf whose ellipsoid misses the
// packet's frustum holds no hit of the packet even when its box passed.
__device__ __forceinline__ bool frustum_ellipsoid(const Frustum &fr, const float4 *l2w) {
    const float4 r0 = l2w[0], r1 = l2w[1], r2 = l2w[2];
#pragma unroll
    for (int p = 0; p < 5; p++) {
        const float4 n = fr.pn[p];
        const float sd = fmaf(n.z, r2.w, fmaf(n.y, r1.w, n.x * r0.w));
        const float e0 = fmaf(r2.x, n.z, fmaf(r1.x, n.y, r0.x * n.x));
        const float e1 = fmaf(r2.y, n.z, fmaf(r1.y, n.y, r0.y * n.x));
        const float e2 = fmaf(r2.z, n.z, fmaf(r1.z, n.y, r0.z * n.x));
        const float gap = fr.pa[p].w - sd;
        if (gap > 0x1.0p-60f && fmaf(e2, e2, fmaf(e1, e1, e0 * e0)) * 1.00006f < gap * gap) return false;
    }
    return true;
}

// Division-free pretest of a block's candidates as conics in the tile's pixel plane.
//
// A tile's rays share the origin o and have (unnormalised) directions v(x, y) = v0 + x du + y dv, with
// (x, y) the pixel's offset from the tile's centre.  With lo = M (o - mu) and l = M v, a ray's line
// passes a Gaussian's unit sphere within its radius iff |lo x l|^2 <= |l|^2, and both sides are
// quadratic in (x, y).  The thread that fetches a candidate computes the six coefficients of
// h(x, y) = |l|^2 - |lo x l|^2 + margin once; every ray then evaluates h at its own (x, y) with five
// FMAs instead of transforming its direction into the candidate's frame (about 45 instructions).
// The coefficients are centred on the tile, so they carry no cancellation beyond the tile's own extent.
//
// Margin (u = 2^-24; norms are Euclidean): the ray direction the intersection program uses and v(x, y)
// differ by at most 32u V, V the sum of the magnitudes of the terms that make up a direction (camera_ray's
// and the basis' own roundings); M times either adds 3u |M|_F V on each side and the cross product 3u of
// its terms, so |lo x l| is known within eta = 64u (|lo| + 1) |M|_F V (48u + 6u of it from the terms above).
// A hit of the intersection program puts the line within 1 + 8u of the unit sphere (its max-density
// point lo + t ld is a point of the line up to one rounding), so |c| <= (1 + 8u) |l| + eta, and
// |c|^2 <= |l|^2 + 2.1 |l| eta + eta^2 + 17u |l|^2.  Coefficients and evaluation round by at most
// 24u (|l|^2 + |c|^2) of their largest values Lm, Cm over the tile; 48u is taken.  Outside the range in
// which every square stays a normal number the candidate is kept (h = +inf), and so it is on a NaN:
// rays read the sign bit of h, which is clear for +inf and for the NaN the arithmetic generates.
// The intersection program still decides every hit.
struct ConicBasis {
    float v0[3], du[3], dv[3];
    float hx, hy;  // largest |x| and |y| of the tile
    float mag;     // V
    // rays from the caller (ray_cone): their common origin, the axis and centre of their cone, and how many of
    // the tile's pixels have one
    float origin[3], axis[3], ca, cb, share;
};

// (a.x * b.x + c.x, a.y * b.y + c.y), each rounded once: one issue slot for two FMAs.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
        "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}

__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float norm_approx(f3 a) { return sqrt_approx(fdot3(a, a)); }

__device__ __forceinline__ f3 cross3(f3 a, f3 b) {
    return mk3(fmaf(a.y, b.z, -(a.z * b.y)), fmaf(a.z, b.x, -(a.x * b.z)), fmaf(a.x, b.y, -(a.y * b.x)));
}

// Coefficients (F, D, E, A, B, C) of h(x, y) = F + x (D + x A + y B) + y (E + y C) for the candidate
// with snapshot rows g0..g2 (columns M) and object-space origin lo.
__device__ __forceinline__ float conic_coefficients(const ConicBasis &cb, const float4 g0, const float4 g1,
                                                    const float4 g2, f3 lo, float q[6]) {
    const f3 v0 = mk3(cb.v0[0], cb.v0[1], cb.v0[2]), du = mk3(cb.du[0], cb.du[1], cb.du[2]),
             dv = mk3(cb.dv[0], cb.dv[1], cb.dv[2]);
    const f3 l0 = mk3(fdot3(g0, v0), fdot3(g1, v0), fdot3(g2, v0));
    const f3 lu = mk3(fdot3(g0, du), fdot3(g1, du), fdot3(g2, du));
    const f3 lv = mk3(fdot3(g0, dv), fdot3(g1, dv), fdot3(g2, dv));
    const f3 c0 = cross3(lo, l0), cu = cross3(lo, lu), cv = cross3(lo, lv);
    const float ll0 = fdot3(l0, l0), lluu = fdot3(lu, lu), llvv = fdot3(lv, lv);
    const float cc0 = fdot3(c0, c0), ccuu = fdot3(cu, cu), ccvv = fdot3(cv, cv);
    const float lm = fmaf(cb.hy, sqrt_approx(llvv), fmaf(cb.hx, sqrt_approx(lluu), sqrt_approx(ll0)));
    const float cm = fmaf(cb.hy, sqrt_approx(ccvv), fmaf(cb.hx, sqrt_approx(ccuu), sqrt_approx(cc0)));
    const float mf = sqrt_approx(g0.x * g0.x + g0.y * g0.y + g0.z * g0.z + g1.x * g1.x + g1.y * g1.y + g1.z * g1.z +
                                 g2.x * g2.x + g2.y * g2.y + g2.z * g2.z);
    const float nl = norm_approx(lo);
    const float eta = 0x1.0p-18f * (nl + 1.0f) * mf * cb.mag;
    const float margin = fmaf(eta, fmaf(2.1f, lm, eta), 0x1.8p-19f * fmaf(lm, lm, cm * cm));
    const bool ok = lm >= 0x1.0p-50f && lm <= 0x1.0p50f && cm <= 0x1.0p50f && nl <= 0x1.0p40f && eta <= 0x1.0p50f;
    q[0] = ok ? (ll0 - cc0) + margin : __int_as_float(0x7f800000);
    q[1] = ok ? 2.0f * (fdot3(l0, lu) - fdot3(c0, cu)) : 0.0f;
    q[2] = ok ? 2.0f * (fdot3(l0, lv) - fdot3(c0, cv)) : 0.0f;
    q[3] = ok ? lluu - ccuu : 0.0f;
    q[4] = ok ? 2.0f * (fdot3(lu, lv) - fdot3(cu, cv)) : 0.0f;
    q[5] = ok ? llvv - ccvv : 0.0f;
    return -__fdividef(fdot3(lo, l0), ll0);
}

// Shared memory of a block that traces one pixel tile (one ray per thread), or, SPLIT, a packet of one.
template <int KB, bool SPLIT>
struct TileShared {
    static constexpr bool kTiles = true;
    static constexpr int kStack = SPLIT ? kSplitStack : kTileStack;
    unsigned long long kbuf[KB][kFwdThreads];
    // the batch's candidates, filled once per batch by the block (one candidate per thread):
    float4 g[kBatch][3];       // snapshot rows with the tile's object-space origin: (M | M (o - mu))
    int4 c[kBatch];            // colour in 2^-24 fixed point (x, y, z), live opacity bits (w)
    float4 conic[kBatch / 2][3];  // coefficients of candidates 2i, 2i+1: (F F' D D') (E E' A A') (B B' C C')
    float sf[kBatch];          // live scaling factor
    uint32_t gid[kBatch];
    uint32_t stk[kStack];
    alignas(16) uint32_t queue[kTileQueue];
    Frustum fr;
    ConicBasis cb;
    uint32_t cnt[kWarps];      // per-warp counts of a step
};

// Shared memory of a block whose warps trace packets of rays one ray per lane, each lane by itself.
template <int KB>
struct RayShared {
    static constexpr bool kTiles = false;
    unsigned long long kbuf[KB][kFwdThreads];
};

// A batch: the block's queued leaves queue[0, take) (take <= kBatch, every thread calls this together;
// leaves beyond them move to the front of the queue).  (1) Thread j takes leaf j: it tests the leaf's
// ellipsoid against the tile's frustum, fetches its snapshot rows, live values and colour, computes
// its object-space ray origin (with local_origin, the arithmetic of local_ray) and its conic, and the
// survivors go to the shared cache in order of their max-density points along the tile's central ray
// (each thread ranks its key among the batch's 128: 32 16-byte loads), so that a ray finds its hits
// nearly front to back and its sorted buffer mostly appends: unsorted batches cost 2.60 instead of
// 2.38 ms at 3M / 1080p and 2.27 instead of 2.20 ms in a train step at 1M / 1600x1040; a scene of few
// hits per ray pays the ranking (500k / 640x480 0.671 to 0.686 ms).  A tile's four warps share the fetched records and
// the batch spans up to 128 candidates, where packets of their own batches fetched every record up to
// four times and tested 21 survivors at a time.  (2) Every ray evaluates the conics at its pixel, two
// candidates per step, into a bit mask of its possible hits.  (3) The lanes of a warp walk their masks
// together, one candidate per lane per step, through the intersection program, which decides the hit,
// and the selection.  The order in which a ray sees its hits does not matter: the all-hit sums are
// order-independent and the selection is by key.
template <int KB, bool SPLIT>
__device__ __forceinline__ void trace_batch_leaves(const TraceScene &sc, const TraceKnobs &k, f3 ro, f3 rd, float px,
                                                   float py, bool want, bool first, LaneState &st,
                                                   TileShared<KB, SPLIT> &sh, int take, int nc) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    {
        uint32_t gid = 0;
        bool keep = false;
        float4 g0, g1, g2;
        int4 cv;
        float sfv = 0.0f;
        float q[6];
        uint32_t key = 0xffffffffu;  // order along the tile's central ray; dropped leaves sort last
        if (t < take) {
            gid = sh.queue[t];
            g0 = sc.geom[3 * (size_t)gid];
            g1 = sc.geom[3 * (size_t)gid + 1];
            g2 = sc.geom[3 * (size_t)gid + 2];
            const float2 lv = sc.live[gid];
            const float *cp = sc.channels + 3 * (size_t)gid;
            const float c0 = cp[0], c1 = cp[1], c2 = cp[2];
            // no ray hits a Gaussian at or below the alpha threshold (intersect_lo's first test)
            keep = !(lv.x <= k.athr) && (sc.l2w ? frustum_ellipsoid(sh.fr, sc.l2w + 3 * (size_t)gid) : true);
            cv = make_int4(colour_fixed(c0), colour_fixed(c1), colour_fixed(c2), __float_as_int(lv.x));
            sfv = lv.y;
            const f3 lo = local_origin(g0, g1, g2, ro);
            const float at = conic_coefficients(sh.cb, g0, g1, g2, lo, q);
            if (keep) key = (__float_as_uint(fmaxf(at, 0.0f)) & ~(uint32_t)(kBatch - 1)) | (uint32_t)t;
            g0.w = lo.x;
            g1.w = lo.y;
            g2.w = lo.z;
        }
        const int rest = nc - take;
        const uint32_t r0 = t < rest ? sh.queue[take + t] : 0u;
        const uint32_t r1 = t + kFwdThreads < rest ? sh.queue[take + kFwdThreads + t] : 0u;
        const uint32_t bal = __ballot_sync(kFull, keep);
        if (lane == 0) sh.cnt[warp] = __popc(bal);
        __syncthreads();  // the counts; every read of the queue and of the previous batch's cache is done
        if (t < rest) sh.queue[t] = r0;
        if (t + kFwdThreads < rest) sh.queue[kFwdThreads + t] = r1;
        uint32_t *keys = sh.queue + kTileQueue - kBatch;  // (free: fewer than kTileQueue - kBatch leaves are left)
        keys[t] = key;
        __syncthreads();
        if (keep) {
            int slot = 0;
#pragma unroll 4
            for (int i = 0; i < kBatch / 4; i++) {
                const uint4 o = reinterpret_cast<const uint4 *>(keys)[i];
                slot += (o.x < key) + (o.y < key) + (o.z < key) + (o.w < key);
            }
            // split: pairs of ranks go round the four warps' words (see merge_split)
            if constexpr (SPLIT) slot = 32 * ((slot >> 1) & 3) + 2 * (slot >> 3) + (slot & 1);
            sh.g[slot][0] = g0;
            sh.g[slot][1] = g1;
            sh.g[slot][2] = g2;
            sh.c[slot] = cv;
            sh.sf[slot] = sfv;
            sh.gid[slot] = gid;
            float *cq = reinterpret_cast<float *>(sh.conic[slot >> 1]) + (slot & 1);
#pragma unroll
            for (int e = 0; e < 6; e++) cq[2 * e] = q[e];
        }
    }
    int kept = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) kept += (int)sh.cnt[w];
    __syncthreads();  // the cache is complete
    if (!__any_sync(kFull, want)) return;
    uint32_t m[kBatch / 32];
    const float2 x2 = make_float2(px, px), y2 = make_float2(py, py);
#pragma unroll
    for (int w = 0; w < kBatch / 32; w++) {
        m[w] = 0u;
        // candidates of this word (the rest of its slots are stale); split: of this warp's word alone
        int left = kept - 32 * w;
        if constexpr (SPLIT) {
            const int mine = kept - 2 * warp;  // ranks from 2 warp on, two of every eight
            left = w == warp ? 2 * (mine >> 3) + min(mine & 7, 2) : 0;
        }
        if (left > 0) {
            uint32_t miss = 0u;  // candidate 32 w + i ends up in bit 31 - i
#pragma unroll 4
            for (int i = 0; i < 16; i++) {
                const float4 qa = sh.conic[16 * w + i][0], qb = sh.conic[16 * w + i][1], qc = sh.conic[16 * w + i][2];
                float2 h = fma2(x2, make_float2(qb.z, qb.w), make_float2(qa.z, qa.w));
                h = fma2(y2, make_float2(qc.x, qc.y), h);
                h = fma2(x2, h, make_float2(qa.x, qa.y));
                h = fma2(y2, fma2(y2, make_float2(qc.z, qc.w), make_float2(qb.x, qb.y)), h);
                miss = __funnelshift_l(__float_as_uint(h.x), miss, 1);
                miss = __funnelshift_l(__float_as_uint(h.y), miss, 1);
            }
            const uint32_t valid = left >= 32 ? 0xffffffffu : ~(0xffffffffu >> left);
            m[w] = want ? ~miss & valid : 0u;
        }
    }
    int base = 0;
    for (;;) {
        if (m[0] == 0u) {
            base += 32;
#pragma unroll
            for (int w = 0; w + 1 < kBatch / 32; w++) m[w] = m[w + 1];
            m[kBatch / 32 - 1] = 0u;
        }
        uint32_t any = m[0];
#pragma unroll
        for (int w = 1; w < kBatch / 32; w++) any |= m[w];
        if (!__any_sync(kFull, any != 0u)) break;
        if (m[0] != 0u) {
            const int b = __clz((int)m[0]);
            m[0] &= ~(0x80000000u >> b);
            const int j = base + b;
            const int4 c = sh.c[j];
            on_leaf_data<KB, true>(sh.gid[j], sh.g[j][0], sh.g[j][1], sh.g[j][2],
                                   make_float2(__int_as_float(c.w), sh.sf[j]), c.x, c.y, c.z, first, ro, rd, k, st,
                                   sh.kbuf);
        }
    }
}

// One full traversal of the tile (rays with a common origin inside sh.fr) by the whole block, all of
// whose threads call this together: each step pops up to 128 nodes, one per thread, tests their child
// boxes against the tile's frustum, pushes surviving internal children and queues surviving leaves;
// every 128 queued leaves become a batch (trace_batch_leaves).  Four packets that walked the tree each
// for itself popped and fetched mostly the same nodes (per tile 270-690 pops and 90-260 queued leaves
// instead of 4 x 970 and 4 x 268 at 3M Gaussians; with the conics, the forward of 3M / 1080p went from
// 3.11 to 2.75 ms, 500k / 640x480 from 0.83 to 0.58 ms, 6M / 4K from 18.3 to 15.6 ms, the image and its
// colours included; the kernel is bound by instruction issue and the latency of each ray's own
// hit chain, at five or four blocks per SM).  With a frontier (count, entries; a count above
// kFrontierMax or a null pointer: none) the traversal starts there instead of at the root: the frontier
// goes onto the stack with its first entry on top, and a frontier leaf is queued when it is popped.
// px, py: the ray's offset from the tile's centre in the conics' basis.  Returns false if the stack
// filled up (a malformed tree; the caller then repeats the traversal per ray).
template <int KB, bool SPLIT>
__device__ __forceinline__ bool traverse_tile(const TraceScene &sc, const TraceKnobs &k, f3 ro, f3 rd, float px,
                                              float py, bool want, bool first, LaneState &st,
                                              TileShared<KB, SPLIT> &sh, const uint32_t *front, int32_t *status) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t lanemask_lt = (1u << lane) - 1u;
    const int n = sc.n;
    const float *rb = sc.root_box;
    const float rmin[3] = {rb[0], rb[1], rb[2]}, rmax[3] = {rb[4], rb[5], rb[6]};
    if (n <= 0 || !frustum_box(sh.fr, rmin, rmax)) return true;
    if (n == 1) {
        on_leaf<KB>(sc, 0u, want, first, ro, rd, k, st, sh.kbuf);
        return true;
    }
    const uint32_t fcount = front ? front[0] : kFrontierNone;
    int sp = 1, nc = 0;
    if (fcount <= (uint32_t)kFrontierMax) {
        sp = (int)fcount;
        for (int i = t; i < sp; i += kFwdThreads) sh.stk[sp - 1 - i] = front[1 + i];
    } else if (t == 0) {
        sh.stk[0] = 0u;
    }
    __syncthreads();
    int budget = n;  // a valid tree pushes each internal node at most once per traversal
    for (;;) {
        while (sp > 0 && nc < kBatch) {
            if (--budget < 0) {
                raise_status(status, GRAY_STATUS_STACK_OVERFLOW);
                sp = 0;
                break;
            }
            // a popped node frees its entry and pushes at most two: as many at once as fit below the reserve, and
            // in it one by one (a descent adds one entry per level, fewer than the reserve holds)
            const int room = TileShared<KB, SPLIT>::kStack - kStackReserve - sp;
            const int take = min(min(sp, kFwdThreads), max(room, 1));
            if (room + kStackReserve <= 1) return false;
            const uint32_t node = t < take ? sh.stk[sp - 1 - t] : GRAY_NULL;
            // children as (a, b) = (nearer, farther) along the tile's mean direction
            bool pa = false, pb = false;
            uint32_t ca = 0, cb = 0;
            if (node != GRAY_NULL) {
                if (node & GRAY_LEAF_BIT) {
                    ca = node;  // a leaf of the tile's frontier: queued below
                    pa = true;
                } else if (node >= (uint32_t)(n - 1)) {
                    raise_status(status, GRAY_STATUS_STACK_OVERFLOW);
                } else {
                    const float4 q0 = sc.nodes[4 * (size_t)node], q1 = sc.nodes[4 * (size_t)node + 1],
                                 q2 = sc.nodes[4 * (size_t)node + 2], q3 = sc.nodes[4 * (size_t)node + 3];
                    const float b0min[3] = {q0.x, q0.y, q0.z}, b0max[3] = {q0.w, q1.x, q1.y};
                    const float b1min[3] = {q1.z, q1.w, q2.x}, b1max[3] = {q2.y, q2.z, q2.w};
                    const uint32_t c0 = __float_as_uint(q3.x), c1 = __float_as_uint(q3.y);
                    const bool p0 = frustum_box(sh.fr, b0min, b0max), p1 = frustum_box(sh.fr, b1min, b1max);
                    // box centres (times 2) projected on the mean direction; the origin is common
                    const float4 c = sh.fr.pn[4];
                    const float s0 = fmaf(q0.z + q1.y, c.z, fmaf(q0.y + q1.x, c.y, (q0.x + q0.w) * c.x));
                    const float s1 = fmaf(q2.x + q2.w, c.z, fmaf(q1.w + q2.z, c.y, (q1.z + q2.y) * c.x));
                    const bool sw = s1 < s0;
                    ca = sw ? c1 : c0;
                    cb = sw ? c0 : c1;
                    pa = sw ? p1 : p0;
                    pb = sw ? p0 : p1;
                }
            }
            const bool ia = pa && !(ca & GRAY_LEAF_BIT), ib = pb && !(cb & GRAY_LEAF_BIT);
            const bool la = pa && (ca & GRAY_LEAF_BIT) && (ca & ~GRAY_LEAF_BIT) < (uint32_t)n;
            const bool lb = pb && (cb & GRAY_LEAF_BIT) && (cb & ~GRAY_LEAF_BIT) < (uint32_t)n;
            // The popped nodes are in visit order (thread 0 took the top).  Their internal children go
            // back so that the next pops see thread 0's nearer child first, then its farther one, then
            // thread 1's, ...; the leaves are queued in the same order.
            const uint32_t ma = __ballot_sync(kFull, ia), mb = __ballot_sync(kFull, ib);
            const uint32_t qa = __ballot_sync(kFull, la), qb = __ballot_sync(kFull, lb);
            if (lane == 0) sh.cnt[warp] = (uint32_t)(__popc(ma) + __popc(mb)) | (uint32_t)(__popc(qa) + __popc(qb)) << 16;
            __syncthreads();  // the counts; every pop has been read
            uint32_t before = 0u, total = 0u;  // (internal, leaves << 16) of the warps before this one, of all
#pragma unroll
            for (int w = 0; w < kWarps; w++) {
                const uint32_t c = sh.cnt[w];
                if (w < warp) before += c;
                total += c;
            }
            const int ni = (int)(total & 0xffffu);
            sp -= take;
            const int above = (int)(before & 0xffffu) + __popc(ma & lanemask_lt) + __popc(mb & lanemask_lt);
            if (ia) sh.stk[sp + ni - 1 - above] = ca;
            if (ib) sh.stk[sp + ni - 1 - above - (ia ? 1 : 0)] = cb;
            sp += ni;
            const int at = nc + (int)(before >> 16) + __popc(qa & lanemask_lt) + __popc(qb & lanemask_lt);
            if (la) sh.queue[at] = ca & ~GRAY_LEAF_BIT;
            if (lb) sh.queue[at + (la ? 1 : 0)] = cb & ~GRAY_LEAF_BIT;
            nc += (int)(total >> 16);
            __syncthreads();  // the pushes; the counts are free again
        }
        if (nc == 0) break;
        const int take = min(nc, kBatch);
        trace_batch_leaves<KB, SPLIT>(sc, k, ro, rd, px, py, want, first, st, sh, take, nc);
        nc -= take;
    }
    return true;
}

// A split tile's block traces one packet: its four warps hold the same 32 rays and each took a quarter of
// the candidates.  After a traversal every thread calls this together, and every warp then holds the
// rays' whole state: the all-hit sums added up (integers, so the order does not matter; a sum that
// stopped at its floor stays at or below it), and the order of the four warps' keys: entry (w, i) of
// rank r is named by src[32 r + lane] = 32 w + i.  The ranks are complete up to the last key of a
// buffer that was full and dropped keys; at most kSplitKeys of them are kept.  The cache's memory
// carries all of it, and the composited ids (see trace_rays).
constexpr int kSplitKeys = 64;

template <int KB>
struct SplitView {
    uint32_t *gids;  // [kSplitKeys][32]
    uint8_t *src;    // [kSplitKeys][32]
    int *bound;      // [kWarps][32]
    __device__ __forceinline__ explicit SplitView(TileShared<KB, true> &sh)
        : gids(reinterpret_cast<uint32_t *>(sh.g)), src(reinterpret_cast<uint8_t *>(sh.conic)),
          bound(reinterpret_cast<int *>(sh.sf)) {}
};

template <int KB>
__device__ __forceinline__ void merge_split(LaneState &st, TileShared<KB, true> &sh, bool first) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    long long *sums = reinterpret_cast<long long *>(sh.g);          // [5][128]
    int *counts = reinterpret_cast<int *>(sums + 5 * kFwdThreads);  // [3][128]
    const SplitView<KB> v(sh);
    static_assert((5 * 8 + 3 * 4) * kFwdThreads <= sizeof(sh.g) + sizeof(sh.c), "sums do not fit");
    static_assert(kSplitKeys * 32 * 4 <= sizeof(sh.g) + sizeof(sh.c) && kSplitKeys * 32 <= sizeof(sh.conic) &&
                      KB <= 32 && kWarps * 32 * 4 <= sizeof(sh.sf),
                  "a split packet's keys do not fit");
    __syncthreads();  // every warp is done with the cache
    if (first) {
        sums[t] = st.lfx;
        sums[kFwdThreads + t] = st.afx;
        sums[2 * kFwdThreads + t] = st.cfx0;
        sums[3 * kFwdThreads + t] = st.cfx1;
        sums[4 * kFwdThreads + t] = st.cfx2;
        counts[t] = st.nhit;
    }
    counts[kFwdThreads + t] = st.ncand;
    counts[2 * kFwdThreads + t] = st.kcount;
    __syncthreads();
    const int own = st.kcount;
    const bool full = st.ncand > st.kcount;  // this warp's buffer dropped keys
    int total = 0, kc[kWarps], at[kWarps];
    st.ncand = 0;
    if (first) {
        st.lfx = st.afx = st.cfx0 = st.cfx1 = st.cfx2 = 0;
        st.nhit = 0;
    }
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
        const int o = 32 * w + lane;
        if (first) {
            st.lfx += sums[o];
            st.afx += sums[kFwdThreads + o];
            st.cfx0 += sums[2 * kFwdThreads + o];
            st.cfx1 += sums[3 * kFwdThreads + o];
            st.cfx2 += sums[4 * kFwdThreads + o];
            st.nhit += counts[o];
        }
        st.ncand += counts[kFwdThreads + o];
        kc[w] = counts[2 * kFwdThreads + o];
        total += kc[w];
        at[w] = 0;
    }
    int bound = kSplitKeys;
    for (int i = 0; i < own; i++) {
        const unsigned long long key = sh.kbuf[i][t];
        int rank = i;
#pragma unroll
        for (int w = 0; w < kWarps; w++) {
            if (w != warp) {
                while (at[w] < kc[w] && sh.kbuf[at[w]][32 * w + lane] < key) at[w]++;
                rank += at[w];
            }
        }
        if (rank >= kSplitKeys) break;
        v.src[32 * rank + lane] = (uint8_t)(32 * warp + i);
        if (full && i == own - 1) bound = rank + 1;
    }
    v.bound[t] = bound;
    __syncthreads();  // the ranks; the sums have been read
#pragma unroll
    for (int w = 0; w < kWarps; w++) total = min(total, v.bound[32 * w + lane]);
    st.kcount = total;
}

// Trace a block's rays (one per thread; `alive` threads only) through the scene: traversal, selection,
// compositing (cuda/forward_pass.cu:6-151 minus the write-out).  tile: the block's rays share one origin
// and lie inside sh.fr, and are traversed together from the frontier `front` (see traverse_tile, px,
// py); else every warp traverses its own rays.  SPLIT: the four warps hold the same 32 rays and share
// their candidates (see merge_split); each ends with the same result, and warp 0 alone writes hit
// lists.  Every thread of the block calls this together; with RayShared (no tiles) the warps are on their own.
template <int KB, bool SPLIT, class Shared>
__device__ __forceinline__ void trace_rays(const TraceScene &sc, const TraceKnobs &k, f3 ro, f3 rd, float px, float py,
                                           bool alive, bool tile, bool grads, const HitSink &hs,
                                           int32_t *status, Shared &sh, const uint32_t *front,
                                           RayResult &res) {
    if constexpr (!Shared::kTiles) tile = false;
    unsigned long long(*kbuf)[kFwdThreads] = sh.kbuf;
    const int lane = threadIdx.x & 31;
    LaneState &st = res.st;
    st.lfx = 0;
    st.afx = st.cfx0 = st.cfx1 = st.cfx2 = 0;
    st.nhit = 0;
    st.kcount = 0;
    st.ncand = 0;
    st.kmax = 0;
    st.resume = 0;
    st.has_resume = false;
    float T = 1.0f, C0 = 0.0f, C1 = 0.0f, C2 = 0.0f, depth = 0.0f;
    int pass = 0, slots = 0, nacc = 0;
    float tmin_sel = k.znear, last_d = k.znear;
    bool done = !alive;
    uint32_t head = GRAY_NULL;

    bool first = true;
    int traversals = 0;
    // the packet needs a second traversal with a 16-slot buffer: some lane of a 32-slot kernel goes
    // on past the 16 nearest keys of its first traversal (the same 16 the narrow kernel holds)
    bool deep = false;
    const int n = sc.n;
    while (tile ? __syncthreads_or(!done) : __any_sync(kFull, !done)) {
        const bool want = !done;
        st.kcount = 0;
        st.ncand = 0;
        st.dfar = __int_as_float(0x7f800000);
        // ---------------- traversal ----------------
        bool per_ray = !tile;
        bool ranked = false;  // the keys are those of the four warps, in merge_split's order
        if constexpr (Shared::kTiles) {
            if (tile && traverse_tile<KB, SPLIT>(sc, k, ro, rd, px, py, want, first, st, sh, front, status)) {
                if constexpr (SPLIT) {
                    merge_split<KB>(st, sh, first);
                    ranked = true;
                }
            } else if (tile) {
                // the tile's stack filled up: discard what was gathered, trace per ray
                st.kcount = 0;
                st.ncand = 0;
                st.dfar = __int_as_float(0x7f800000);
                if (first) {
                    st.lfx = 0;
                    st.afx = st.cfx0 = st.cfx1 = st.cfx2 = 0;
                    st.nhit = 0;
                }
                per_ray = true;
            }
        }
        if (!per_ray) {
        } else if (n == 1) {
            // (the per-ray path's ray data is built here, so it holds no registers in the frustum path)
            const SlabRay sr = make_slab_ray(ro, rd, 2.0e-6f * (fabsf(ro.x) + fabsf(ro.y) + fabsf(ro.z)));
            const float *rb = sc.root_box;
            const float bmin[3] = {rb[0], rb[1], rb[2]}, bmax[3] = {rb[4], rb[5], rb[6]};
            bool h = want && slab_hit(bmin, bmax, sr);
            if (__any_sync(kFull, h)) on_leaf<KB>(sc, 0u, h, first, ro, rd, k, st, kbuf);
        } else if (n > 1) {
            const SlabRay sr = make_slab_ray(ro, rd, 2.0e-6f * (fabsf(ro.x) + fabsf(ro.y) + fabsf(ro.z)));
            // packet lead direction for the near/far child order (any deterministic choice is valid)
            float lx = alive ? rd.x : 0.0f, ly = alive ? rd.y : 0.0f, lz = alive ? rd.z : 0.0f;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                lx += __shfl_xor_sync(kFull, lx, off);
                ly += __shfl_xor_sync(kFull, ly, off);
                lz += __shfl_xor_sync(kFull, lz, off);
            }
            uint32_t stk0 = 0, stk1 = 0;  // entry e lives in lane e%32, word e/32
            int sp = 0;
            {
                const float *rb = sc.root_box;
                const float bmin[3] = {rb[0], rb[1], rb[2]}, bmax[3] = {rb[4], rb[5], rb[6]};
                bool h = want && slab_hit(bmin, bmax, sr);
                if (__any_sync(kFull, h)) {
                    if (lane == 0) stk0 = 0u;
                    sp = 1;
                }
            }
            long long budget = 2LL * n;  // pops of a valid tree per traversal are < n
            while (sp > 0) {
                if (--budget < 0) {
                    raise_status(status, GRAY_STATUS_STACK_OVERFLOW);
                    break;
                }
                sp--;
                const uint32_t word = (sp >> 5) == 0 ? stk0 : stk1;
                const uint32_t node = __shfl_sync(kFull, word, sp & 31);
                if (node >= (uint32_t)(n - 1)) {
                    raise_status(status, GRAY_STATUS_STACK_OVERFLOW);
                    continue;
                }
                const float4 q0 = sc.nodes[4 * node], q1 = sc.nodes[4 * node + 1], q2 = sc.nodes[4 * node + 2],
                             q3 = sc.nodes[4 * node + 3];
                const float b0min[3] = {q0.x, q0.y, q0.z}, b0max[3] = {q0.w, q1.x, q1.y};
                const float b1min[3] = {q1.z, q1.w, q2.x}, b1max[3] = {q2.y, q2.z, q2.w};
                const uint32_t c0 = __float_as_uint(q3.x), c1 = __float_as_uint(q3.y);
                const bool h0 = want && slab_hit(b0min, b0max, sr);
                const bool h1 = want && slab_hit(b1min, b1max, sr);
                const bool any0 = __any_sync(kFull, h0), any1 = __any_sync(kFull, h1);
                if (!any0 && !any1) continue;
                // near child first along the packet's lead direction
                const float p0 = (b0min[0] + b0max[0]) * lx + (b0min[1] + b0max[1]) * ly + (b0min[2] + b0max[2]) * lz;
                const float p1 = (b1min[0] + b1max[0]) * lx + (b1min[1] + b1max[1]) * ly + (b1min[2] + b1max[2]) * lz;
                const bool swap = p1 < p0;
                const uint32_t cn = swap ? c1 : c0, cf = swap ? c0 : c1;
                const bool an = swap ? any1 : any0, af = swap ? any0 : any1;
                const bool hn = swap ? h1 : h0, hf = swap ? h0 : h1;
                // far internal child goes deeper in the stack, near internal child on top;
                // leaves are processed right away, near first
                if (af && !(cf & GRAY_LEAF_BIT)) stack_push(stk0, stk1, sp, cf, lane, status);
                if (an && (cn & GRAY_LEAF_BIT)) {
                    const uint32_t gid = cn & ~GRAY_LEAF_BIT;
                    if (gid < (uint32_t)n) on_leaf<KB>(sc, gid, hn, first, ro, rd, k, st, kbuf);
                }
                if (af && (cf & GRAY_LEAF_BIT)) {
                    const uint32_t gid = cf & ~GRAY_LEAF_BIT;
                    if (gid < (uint32_t)n) on_leaf<KB>(sc, gid, hf, first, ro, rd, k, st, kbuf);
                }
                if (an && !(cn & GRAY_LEAF_BIT)) stack_push(stk0, stk1, sp, cn, lane, status);
            }
        }
        // ---------------- consume (cuda/forward_pass.cu:46-125) ----------------
        int nc = 0;
        const auto key_at = [&](int i) -> unsigned long long {
            if constexpr (SPLIT) {
                if (ranked) {
                    const uint32_t s = SplitView<KB>(sh).src[32 * i + lane];
                    return kbuf[s & 31u][(s & ~31u) + lane];
                }
            }
            return kbuf[i][threadIdx.x];
        };
        // composited ids replace the keys already looked at (split: the keys are shared by the warps,
        // so every warp writes the same ids beside them)
        const auto gid_at = [&](int i) -> uint32_t & {
            if constexpr (SPLIT) {
                if (ranked) return SplitView<KB>(sh).gids[32 * i + lane];
            }
            return *reinterpret_cast<uint32_t *>(&kbuf[i][threadIdx.x]);
        };
        if (want) {
            const unsigned long long last_key = st.kcount > 0 ? key_at(st.kcount - 1) : 0ull;
            // the next entry and its colour are fetched while this one is composited
            unsigned long long next = st.kcount > 0 ? key_at(0) : 0ull;
            const float *nc0 = sc.channels + 3 * (size_t)(uint32_t)(next >> 16);
            float nx = 0.0f, ny = 0.0f, nz = 0.0f;
            if (st.kcount > 0) {
                nx = nc0[0];
                ny = nc0[1];
                nz = nc0[2];
            }
            for (int i = 0; i < st.kcount; i++) {
                if constexpr (KB > 16 || SPLIT) {
                    if (i == 16 && first) deep = true;
                }
                const unsigned long long key = next;
                const float cx = nx, cy = ny, cz = nz;
                if (i + 1 < st.kcount) {
                    next = key_at(i + 1);
                    const float *c = sc.channels + 3 * (size_t)(uint32_t)(next >> 16);
                    nx = c[0];
                    ny = c[1];
                    nz = c[2];
                }
                const float d = h2f_bits((uint16_t)(key >> 48));
                if (!(d > tmin_sel)) continue;
                if (slots == kPassSlots) {
                    pass++;
                    if (pass >= kMaxPasses) {
                        done = true;
                        break;
                    }
                    tmin_sel = last_d;
                    if (!(tmin_sel < k.zfar)) {
                        done = true;
                        break;
                    }
                    slots = 0;
                    if (!(d > tmin_sel)) continue;
                }
                slots++;
                last_d = d;
                if (!(d < k.zfar)) {
                    done = true;
                    break;
                }
                const uint32_t gid = (uint32_t)(key >> 16);
                const float al = h2f_bits((uint16_t)(key & 0xFFFFu));
                const long long a = alpha16_fixed((uint16_t)(key & 0xFFFFu));
                st.afx -= a;
                st.cfx0 -= mul_fixed(a, colour_fixed(cx));
                st.cfx1 -= mul_fixed(a, colour_fixed(cy));
                st.cfx2 -= mul_fixed(a, colour_fixed(cz));
                const float w = T * al;
                C0 = C0 + cx * w;
                C1 = C1 + cy * w;
                C2 = C2 + cz * w;
                if (k.render_depth) depth = depth + d * w;
                T = T * (1.0f - al);
                gid_at(nc) = gid;
                nc++;
                nacc++;
                if (T < k.tthr) {
                    done = true;
                    break;
                }
            }
            if (!done) {
                if (st.ncand > st.kcount) {
                    // resume after the last key looked at; entries at or below the active pass
                    // threshold would be dropped anyway, so skip them at the traversal
                    unsigned long long r = last_key;
                    const bool exact = pass > 0 || slots == kPassSlots;
                    if (exact) {
                        const float thr = slots == kPassSlots ? fmaxf(last_d, tmin_sel) : tmin_sel;
                        const unsigned long long skip = ((unsigned long long)f2h_bits(thr) << 48) | 0xFFFFFFFFFFFFull;
                        r = skip > r ? skip : r;
                    }
                    st.resume = r;
                    st.has_resume = true;
                    if (++traversals > kMaxTraversals) {
                        raise_status(status, GRAY_STATUS_STACK_OVERFLOW);
                        done = true;
                    }
                } else {
                    done = true;
                }
            }
        }
        // ---------------- backward hit list segment (warp aggregated) ----------------
        if (grads) {
            const uint32_t need = nc > 0 && (!SPLIT || threadIdx.x < 32) ? (uint32_t)nc + 2u : 0u;
            uint32_t incl = need;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                uint32_t v = __shfl_up_sync(kFull, incl, off);
                if (lane >= off) incl += v;
            }
            const uint32_t total = __shfl_sync(kFull, incl, 31);
            uint32_t base = 0;
            if (total > 0) {
                if (lane == 31) base = atomicAdd(hs.counter, total);
                base = __shfl_sync(kFull, base, 31);
            }
            if (need > 0) {
                const uint32_t off = base + incl - need;
                const bool fits = base <= hs.pool_size && total <= hs.pool_size - base;
                if (fits) {
                    hs.pool[off] = head;
                    hs.pool[off + 1] = (uint32_t)nc;
                    for (int j = 0; j < nc; j++) hs.pool[off + 2 + j] = gid_at(j);
                    head = off;
                } else {
                    raise_status(status, GRAY_STATUS_HITLIST_OVERFLOW);
                }
            }
        }
        first = false;
    }
    res.T = T;
    res.C0 = C0;
    res.C1 = C1;
    res.C2 = C2;
    st.ft = full_transmittance(st.lfx);
    res.depth = depth;
    res.nacc = nacc;
    res.head = head;
    res.retraced = __any_sync(kFull, traversals > 0 || deep);
}

// Truncated-tail estimate and background (cuda/forward_pass.cu:131-142).
__device__ __forceinline__ void finish_ray(RayResult &r, const float *bg, float eps_fwd, bool render_depth,
                                           float &r0, float &r1, float &r2) {
    const LaneState &st = r.st;
    const float rT = r.T - st.ft;
    r0 = r1 = r2 = 0.0f;
    if (st.afx > 0) {
        const float sa = __ll2float_rn(st.afx) * 0x1.0p-24f;
        r0 = (__ll2float_rn(st.cfx0) * 0x1.0p-48f) / sa;
        r1 = (__ll2float_rn(st.cfx1) * 0x1.0p-48f) / sa;
        r2 = (__ll2float_rn(st.cfx2) * 0x1.0p-48f) / sa;
    }
    r.C0 = r.C0 + rT * r0;
    r.C1 = r.C1 + rT * r1;
    r.C2 = r.C2 + rT * r2;
    if (render_depth) r.depth = r.depth / fmaxf(1.0f - r.T, eps_fwd);
    r.C0 = r.C0 + bg[0] * st.ft;
    r.C1 = r.C1 + bg[1] * st.ft;
    r.C2 = r.C2 + bg[2] * st.ft;
}

// Primary ray of pixel (px, py) of a width x height pinhole camera (cuda/core/camera.h:17-36).
__device__ __forceinline__ f3 camera_ray(const float *w, float fov, int px, int py, uint32_t width, uint32_t height,
                                         float jx, float jy) {
    const float view_size = tanf(fov / 2.0f);
    const float aspect = (float)width / (float)height;
    const float fx = (float)px + jx, fy = (float)py + jy;
    const float y = view_size * (1.0f - 2.0f * (fy + 0.5f) / (float)height);
    const float x = aspect * view_size * (2.0f * (fx + 0.5f) / (float)width - 1.0f);
    f3 v = mk3(w[0] * x + w[3] * y - w[6], w[1] * x + w[4] * y - w[7], w[2] * x + w[5] * y - w[8]);
    const float inv = 1.0f / sqrtf(dot3(v, v));
    return mk3(v.x * inv, v.y * inv, v.z * inv);
}

__device__ __forceinline__ float3 camera_ray3(const float *w, float fov, int px, int py, uint32_t width,
                                              uint32_t height, float jx, float jy) {
    const f3 r = camera_ray(w, fov, px, py, width, height, jx, jy);
    return make_float3(r.x, r.y, r.z);
}

// The tile's ray basis for the conics: directions v(x, y) = v0 + x du + y dv of the pinhole camera's
// pixels at the offset (x, y) from pixel position (cx, cy), as camera_ray forms them.  One thread.
__device__ __forceinline__ void make_conic_basis(ConicBasis &cb, const float *w, float fov, float cx, float cy,
                                                 float hx, float hy, uint32_t width, uint32_t height) {
    const float vs = tanf(fov / 2.0f), ax = (float)width / (float)height * vs;
    const float x0 = ax * (2.0f * (cx + 0.5f) / (float)width - 1.0f), y0 = vs * (1.0f - 2.0f * (cy + 0.5f) / (float)height);
    const float dx = 2.0f * ax / (float)width, dy = -2.0f * vs / (float)height;
    float n0 = 0.0f, n1 = 0.0f, n2 = 0.0f;
#pragma unroll
    for (int e = 0; e < 3; e++) {
        cb.v0[e] = w[e] * x0 + w[3 + e] * y0 - w[6 + e];
        cb.du[e] = w[e] * dx;
        cb.dv[e] = w[3 + e] * dy;
        n0 += w[e] * w[e];
        n1 += w[3 + e] * w[3 + e];
        n2 += w[6 + e] * w[6 + e];
    }
    cb.hx = hx;
    cb.hy = hy;
    // V's terms: the pixel's (2 (x + 0.5) / width is below 2) and the basis' own, which are larger where a tile
    // reaches past a small image (one pixel wide, x0 is 7 or 15 ax).  The block waits for this chain: with
    // square roots rounded to nearest a light frame's tiles took 1% longer (20k Gaussians, 1920x1080).
    const float mx = fmaxf(2.0f * fabsf(ax), fabsf(x0) + hx * fabsf(dx));
    const float my = fmaxf(2.0f * fabsf(vs), fabsf(y0) + hy * fabsf(dy));
    cb.mag = sqrt_approx(n0) * mx + sqrt_approx(n1) * my + sqrt_approx(n2);
}

// Rays that the caller supplied for the pixels [x0, x1] x [y0, y1]: when those that are alive share
// their origin and lie within about 53 degrees of their mean direction, the T threads of a block (they call
// this together, and wait for one another afterwards; part: scratch of a row per warp) build their frustum
// and the conics' basis and return true.  With the axis m and unit vectors u, v across it, a ray is the direction m + a u + b v up to its
// length; the frustum spans the rectangle of the rays' (a, b), widened by 4e-6 (some 60 roundings of what
// they are computed from), and the conics' plane is that of (a, b) about its centre.  Lengths outside
// [2^-10, 2^10] (whose object-space squares could leave the normal range) and NaNs are left to the
// per-ray traversal.
// Not inlined: its registers would cost the camera rays' kernels 2%.
constexpr int kConePart = 16;

template <int T>
__device__ __noinline__ bool ray_cone(const float *__restrict__ ray_o, const float *__restrict__ ray_d,
                                      uint32_t alloc_w, const float *__restrict__ root_box, int x0, int y0,
                                      int x1, int y1, Frustum &fr, ConicBasis &cb, float (*part)[kConePart]) {
    constexpr int W = T / 32;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int w = x1 - x0 + 1, count = w * (y1 - y0 + 1);
    if (w <= 0 || y1 < y0) return false;  // a split tile's packet beyond the image
    bool have = false, bad = false;
    int rays = 0;
    f3 ref = mk3(0.0f, 0.0f, 0.0f), m = mk3(0.0f, 0.0f, 0.0f);
    for (int i0 = 0; i0 < count; i0 += T) {
        const int i = i0 + t;
        const size_t px = 3 * ((size_t)(y0 + i / w) * alloc_w + (size_t)(x0 + i % w));
        f3 d = mk3(0.0f, 0.0f, 0.0f), o = d;
        if (i < count) {
            d = mk3(ray_d[px], ray_d[px + 1], ray_d[px + 2]);
            o = mk3(ray_o[px], ray_o[px + 1], ray_o[px + 2]);
        }
        const float len2 = dot3(d, d);
        const bool on = !(sqrtf(len2) == 0.0f);
        const uint32_t who = __ballot_sync(kFull, on);
        rays += __popc(who);
        if (!have && who != 0u) {
            const int lead = __ffs((int)who) - 1;
            ref = mk3(__shfl_sync(kFull, o.x, lead), __shfl_sync(kFull, o.y, lead), __shfl_sync(kFull, o.z, lead));
            have = true;
        }
        if (on) {
            if (!(len2 >= 0x1.0p-20f && len2 <= 0x1.0p20f)) bad = true;
            if (!(o.x == ref.x && o.y == ref.y && o.z == ref.z)) bad = true;
            const float inv = 1.0f / sqrtf(len2);
            m = mk3(fmaf(d.x, inv, m.x), fmaf(d.y, inv, m.y), fmaf(d.z, inv, m.z));
        }
        if (__any_sync(kFull, bad)) break;  // (origins of their own: the first round tells)
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        m = mk3(m.x + __shfl_xor_sync(kFull, m.x, off), m.y + __shfl_xor_sync(kFull, m.y, off),
                m.z + __shfl_xor_sync(kFull, m.z, off));
    bad = __any_sync(kFull, bad);
    if constexpr (W > 1) {
        if (lane == 0) {
            float *p = part[warp];
            p[0] = m.x;
            p[1] = m.y;
            p[2] = m.z;
            p[3] = ref.x;
            p[4] = ref.y;
            p[5] = ref.z;
            p[6] = bad ? -1.0f : (float)rays;
        }
        __syncthreads();
        m = mk3(0.0f, 0.0f, 0.0f);
        have = bad = false;
        rays = 0;
        for (int q = 0; q < W; q++) {
            const float *p = part[q];
            if (p[6] < 0.0f) bad = true;
            if (!(p[6] > 0.0f)) continue;  // no ray of this warp
            if (!have) ref = mk3(p[3], p[4], p[5]);
            have = true;
            if (!(p[3] == ref.x && p[4] == ref.y && p[5] == ref.z)) bad = true;
            m = mk3(m.x + p[0], m.y + p[1], m.z + p[2]);
            rays += (int)p[6];
        }
    }
    if (bad || rays == 0) return false;
    const float inv = 1.0f / sqrtf(dot3(m, m));
    m = mk3(m.x * inv, m.y * inv, m.z * inv);
    if (!(dot3(m, m) > 0.99f)) return false;  // (directions that cancel, NaN)
    f3 u = fabsf(m.x) < 0.7f ? mk3(0.0f, m.z, -m.y) : mk3(-m.z, 0.0f, m.x);
    const float ul = 1.0f / sqrtf(dot3(u, u));
    u = mk3(u.x * ul, u.y * ul, u.z * ul);
    const f3 v = cross3(m, u);
    const float big = __int_as_float(0x7f800000);
    float a0 = big, a1 = -big, b0 = big, b1 = -big;
    for (int i = t; i < count; i += T) {
        const size_t px = 3 * ((size_t)(y0 + i / w) * alloc_w + (size_t)(x0 + i % w));
        const f3 d = mk3(ray_d[px], ray_d[px + 1], ray_d[px + 2]);
        const float len = sqrtf(dot3(d, d));
        if (len == 0.0f) continue;
        const float c = fdot3(d, m);
        if (!(c >= 0.6f * len)) bad = true;
        const float ra = fdot3(d, u) / c, rb = fdot3(d, v) / c;
        a0 = fminf(a0, ra);
        a1 = fmaxf(a1, ra);
        b0 = fminf(b0, rb);
        b1 = fmaxf(b1, rb);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a0 = fminf(a0, __shfl_xor_sync(kFull, a0, off));
        a1 = fmaxf(a1, __shfl_xor_sync(kFull, a1, off));
        b0 = fminf(b0, __shfl_xor_sync(kFull, b0, off));
        b1 = fmaxf(b1, __shfl_xor_sync(kFull, b1, off));
    }
    bad = __any_sync(kFull, bad);
    if constexpr (W > 1) {
        if (lane == 0) {
            float *p = part[warp];
            p[8] = a0;
            p[9] = a1;
            p[10] = b0;
            p[11] = b1;
            p[12] = bad ? 1.0f : 0.0f;
        }
        __syncthreads();
        for (int q = 0; q < W; q++) {
            const float *p = part[q];
            a0 = fminf(a0, p[8]);
            a1 = fmaxf(a1, p[9]);
            b0 = fminf(b0, p[10]);
            b1 = fmaxf(b1, p[11]);
            if (p[12] != 0.0f) bad = true;
        }
    }
    if (bad) return false;
    const float wide = 4e-6f * (1.0f + fmaxf(fabsf(a0), fabsf(a1)) + fmaxf(fabsf(b0), fabsf(b1)));
    a0 -= wide;
    a1 += wide;
    b0 -= wide;
    b1 += wide;
    if (t < 5) {
        f3 d[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const float ea = e == 1 || e == 2 ? a1 : a0, eb = e >= 2 ? b1 : b0;
            d[e] = mk3(fmaf(eb, v.x, fmaf(ea, u.x, m.x)), fmaf(eb, v.y, fmaf(ea, u.y, m.y)),
                       fmaf(eb, v.z, fmaf(ea, u.z, m.z)));
        }
        frustum_plane(t, ref, d, root_box, fr.pn[t], fr.pa[t]);
    }
    if (t == 0) {
        const float ca = 0.5f * (a0 + a1), cc = 0.5f * (b0 + b1);
        const float mm[3] = {m.x, m.y, m.z}, uu[3] = {u.x, u.y, u.z}, vv[3] = {v.x, v.y, v.z};
        const float oo[3] = {ref.x, ref.y, ref.z};
#pragma unroll
        for (int e = 0; e < 3; e++) {
            cb.v0[e] = fmaf(cc, vv[e], fmaf(ca, uu[e], mm[e]));
            cb.du[e] = uu[e];
            cb.dv[e] = vv[e];
            cb.origin[e] = oo[e];
            cb.axis[e] = mm[e];
        }
        cb.ca = ca;
        cb.cb = cc;
        cb.hx = 0.5f * (a1 - a0);
        cb.hy = 0.5f * (b1 - b0);
        cb.mag = 2.0f * (1.0f + fmaxf(fabsf(a0), fabsf(a1)) + fmaxf(fabsf(b0), fabsf(b1)));
        cb.share = (float)rays / (float)count;
    }
    __syncwarp();
    return true;
}

__device__ __forceinline__ TraceKnobs trace_knobs(const FwdArgs &a) {
    TraceKnobs k;
    k.znear = *a.znear;
    k.zfar = *a.zfar;
    k.athr = *a.alpha_threshold;
    k.pw = *a.exp_power;
    k.tthr = *a.t_threshold;
    k.render_depth = *a.render_depth != 0;
    return k;
}

// What a traced ray leaves behind (cuda/forward_pass.cu:131-151).
__device__ __forceinline__ void store_ray(const FwdArgs &a, const TraceKnobs &k, bool grads, uint32_t pixel, f3 ro,
                                          f3 rd, RayResult &r) {
    float r0, r1, r2;
    finish_ray(r, a.bg, *a.eps_fwd, k.render_depth, r0, r1, r2);
    a.out_rgb[3 * pixel] = r.C0;
    a.out_rgb[3 * pixel + 1] = r.C1;
    a.out_rgb[3 * pixel + 2] = r.C2;
    if (grads) {
        a.out_depth[pixel] = r.depth;
        a.out_T[pixel] = r.T;
        a.out_fullT[pixel] = r.st.ft;
        a.out_rem[3 * pixel] = r0;
        a.out_rem[3 * pixel + 1] = r1;
        a.out_rem[3 * pixel + 2] = r2;
        a.ray_o[3 * pixel] = ro.x;
        a.ray_o[3 * pixel + 1] = ro.y;
        a.ray_o[3 * pixel + 2] = ro.z;
        a.ray_d[3 * pixel] = rd.x;
        a.ray_d[3 * pixel + 1] = rd.y;
        a.ray_d[3 * pixel + 2] = rd.z;
        a.stat_hit[pixel] += r.st.nhit;
        a.stat_acc[pixel] += r.nacc;
        a.head[pixel] = r.head;
    } else {
        const bool nro = *a.needs_ray_output != 0;
        if (k.render_depth || nro) a.out_depth[pixel] = r.depth;
        if (nro) {
            a.ray_d[3 * pixel] = rd.x;
            a.ray_d[3 * pixel + 1] = rd.y;
            a.ray_d[3 * pixel + 2] = rd.z;
        }
        a.head[pixel] = GRAY_NULL;
    }
}

// Where a tile's rays come from: the camera; whatever rays_from_python says, supplied rays of a tile that
// share a cone being traversed together; or the same, supplied rays being traversed one by one.
constexpr int kCamera = 0, kCones = 1, kSingles = 2;

// The block's pixel tile (bx, by): 2x2 packets of tile_w x tile_h pixels, one packet per warp; or, SPLIT:
// packet sub of it alone, its candidates shared by the four warps.  Returns whether the calling
// warp's packet needs more than one traversal with 16 hit slots (RayResult::retraced).
// RAYS: other rays than the camera's cost its kernels registers (1.8% of the forward).
template <int KB, bool SPLIT, int RAYS>
__device__ __forceinline__ bool forward_tile(const FwdArgs &a, int bx, int by, int sub, TileShared<KB, SPLIT> &sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int rw = SPLIT ? a.tile_w : a.tile_w * kBlockWarpsX, rh = SPLIT ? a.tile_h : a.tile_h * kBlockWarpsY;
    const int pk = SPLIT ? sub : warp;  // the warp's packet
    const int px0 = bx * (a.tile_w * kBlockWarpsX) + (pk % kBlockWarpsX) * a.tile_w;
    const int py0 = by * (a.tile_h * kBlockWarpsY) + (pk / kBlockWarpsX) * a.tile_h;
    // the pixels the block traces start at (tx0, ty0)
    const int tx0 = SPLIT ? px0 : bx * (a.tile_w * kBlockWarpsX), ty0 = SPLIT ? py0 : by * (a.tile_h * kBlockWarpsY);
    const int px = px0 + (lane % a.tile_w), py = py0 + (lane / a.tile_w);
    const bool inside = px < (int)a.render_w && py < (int)a.render_h;
    const uint32_t pixel = (uint32_t)py * a.alloc_w + (uint32_t)px;

    const TraceKnobs k = trace_knobs(a);
    const bool grads = !a.display && *a.grads_enabled != 0;
    const TraceScene sc{a.geom, a.l2w, a.live, a.channels, a.nodes, a.root_box, a.n};
    const HitSink hs{a.counter, a.pool, a.pool_size};

    // ---- ray generation (cuda/shaders.cu:76-88) ----
    f3 ro = mk3(0.0f, 0.0f, 0.0f), rd = mk3(0.0f, 0.0f, 0.0f);
    float jx = 0.0f, jy = 0.0f;
    bool alive = false;
    // every thread holds the camera origin, inactive ones too (a tile's candidates get their
    // object-space origin from whichever thread fetches them)
    const bool given = RAYS != kCamera && *a.rays_from_python;
    if (!given) ro = mk3(a.cam_origin[0], a.cam_origin[1], a.cam_origin[2]);
    if (inside) {
        if (given) {
            ro = mk3(a.ray_o[3 * pixel], a.ray_o[3 * pixel + 1], a.ray_o[3 * pixel + 2]);
            rd = mk3(a.ray_d[3 * pixel], a.ray_d[3 * pixel + 1], a.ray_d[3 * pixel + 2]);
        } else {
            ro = mk3(a.cam_origin[0], a.cam_origin[1], a.cam_origin[2]);
            if (*a.jitter) {
                uint32_t h = pcg_hash(pixel ^ pcg_hash(*a.total_num_calls));
                jx = (float)(h & 0xFFFFu) * 0x1.0p-16f - 0.5f;
                jy = (float)(h >> 16) * 0x1.0p-16f - 0.5f;
            }
            rd = camera_ray(a.w2c, *a.fov, px, py, a.render_w, a.render_h, jx, jy);
        }
        alive = !(sqrtf(dot3(rd, rd)) == 0.0f);
    }

    // rays that share their origin: the block traverses its tile together
    bool tile = true;
    float x = 0.0f, y = 0.0f;  // the ray's place in the conics' plane
    if (given) {
        tile = false;
        if constexpr (RAYS == kCones) {
            static_assert(sizeof(sh.kbuf) >= sizeof(float) * kWarps * kConePart, "the cone's scratch does not fit");
            tile = ray_cone<kFwdThreads>(a.ray_o, a.ray_d, a.alloc_w, a.root_box, tx0, ty0,
                                         min(tx0 + rw, (int)a.render_w) - 1, min(ty0 + rh, (int)a.render_h) - 1, sh.fr,
                                         sh.cb, reinterpret_cast<float(*)[kConePart]>(sh.kbuf));
            __syncthreads();
            if (tile) {
                const f3 m = mk3(sh.cb.axis[0], sh.cb.axis[1], sh.cb.axis[2]);
                const float c = fdot3(rd, m);
                x = fdot3(rd, mk3(sh.cb.du[0], sh.cb.du[1], sh.cb.du[2])) / c - sh.cb.ca;
                y = fdot3(rd, mk3(sh.cb.dv[0], sh.cb.dv[1], sh.cb.dv[2])) / c - sh.cb.cb;
                if (!alive) ro = mk3(sh.cb.origin[0], sh.cb.origin[1], sh.cb.origin[2]);
            }
        }
    } else {
        const float wide = *a.jitter ? 0.5f : 0.0f;
        const float hx = (float)(rw - 1) * 0.5f, hy = (float)(rh - 1) * 0.5f;
        // (the loop of trace_rays starts with a block barrier)
        if (warp == 0)
            make_frustum_warp(sh.fr, ro, a.w2c, *a.fov, tx0, ty0, tx0 + rw - 1, ty0 + rh - 1, a.render_w, a.render_h,
                              a.root_box, wide);
        if (threadIdx.x == kFwdThreads - 1)
            make_conic_basis(sh.cb, a.w2c, *a.fov, (float)tx0 + hx, (float)ty0 + hy, hx + wide, hy + wide, a.render_w,
                             a.render_h);
        // (pixel plus jitter as camera_ray rounds it; the differences are exact)
        x = ((float)px + jx) - ((float)tx0 + hx);
        y = ((float)py + jy) - ((float)ty0 + hy);
    }
    const uint32_t *front =
        tile && a.frontier ? a.frontier + (size_t)(by * a.tiles_x + bx) * kFrontierWords : nullptr;
    RayResult r;
    trace_rays<KB, SPLIT>(sc, k, ro, rd, x, y, alive, tile, grads, hs, a.status, sh, front, r);
    if (SPLIT && warp != 0) return false;
    if (!inside) return r.retraced;
    if (!alive) {
        a.head[pixel] = GRAY_NULL;  // inactive pixel: empty list, nothing else written
        return r.retraced;
    }
    store_ray(a, k, grads, pixel, ro, rd, r);
    return r.retraced;
}

// Packet sub of the pixel tile (bx, by) on the caller's rays, traced by one warp ray by ray.
template <int KB>
__device__ __forceinline__ bool forward_ray_packet(const FwdArgs &a, int bx, int by, int sub, RayShared<KB> &sh) {
    const int lane = threadIdx.x & 31;
    const int px = (bx * kBlockWarpsX + sub % kBlockWarpsX) * a.tile_w + lane % a.tile_w;
    const int py = (by * kBlockWarpsY + sub / kBlockWarpsX) * a.tile_h + lane / a.tile_w;
    const bool inside = px < (int)a.render_w && py < (int)a.render_h;
    const uint32_t pixel = (uint32_t)py * a.alloc_w + (uint32_t)px;
    const TraceKnobs k = trace_knobs(a);
    const bool grads = !a.display && *a.grads_enabled != 0;
    const TraceScene sc{a.geom, a.l2w, a.live, a.channels, a.nodes, a.root_box, a.n};
    const HitSink hs{a.counter, a.pool, a.pool_size};
    f3 ro = mk3(0.0f, 0.0f, 0.0f), rd = ro;
    if (inside) {
        ro = mk3(a.ray_o[3 * pixel], a.ray_o[3 * pixel + 1], a.ray_o[3 * pixel + 2]);
        rd = mk3(a.ray_d[3 * pixel], a.ray_d[3 * pixel + 1], a.ray_d[3 * pixel + 2]);
    }
    const bool alive = inside && !(sqrtf(dot3(rd, rd)) == 0.0f);
    RayResult r;
    trace_rays<KB, false>(sc, k, ro, rd, 0.0f, 0.0f, alive, false, grads, hs, a.status, sh, nullptr, r);
    if (alive) store_ray(a, k, grads, pixel, ro, rd, r);
    else if (inside) a.head[pixel] = GRAY_NULL;
    return r.retraced;
}

// Programmatic launches (see launch_trace_forward): a kernel of the chain lets the next one start once
// all of its blocks have (griddepcontrol.launch_dependents), and block 0 of each waits at its end for
// the launch before it to complete (griddepcontrol.wait; nothing to wait for in an ordinary launch), so
// that the last one's completion is the chain's.  The other blocks leave their SM to the next kernel.
__device__ __forceinline__ void grid_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait_before() {
    if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Grid launch: block (x, y) renders tile (x, y).
template <int KB, int MINB>
__global__ void __launch_bounds__(kFwdThreads, MINB) trace_forward_kernel(const FwdArgs a) {
    __shared__ TileShared<KB, false> sh;
    if (*a.render_ellipsoids) return;  // the ellipsoid view (ellipsoid_kernel) renders this frame
    forward_tile<KB, false, kSingles>(a, blockIdx.x, blockIdx.y, 0, sh);
}

// Persistent launch: the blocks take tiles from the schedule's order, densest first, until none is
// left (a separate kernel, so the grid launch keeps its register allocation).
// The packets it traced, and those that traverse more than once with a 16-slot buffer (whatever KB
// is), are added to the schedule's statistics words (the automatic kernel choice of the next forward
// reads them).
template <int KB, int MINB>
__global__ void __launch_bounds__(kFwdThreads, MINB) trace_forward_sched_kernel(const FwdArgs a) {
    __shared__ TileShared<KB, false> sh;
    __shared__ uint32_t s_next, s_packets, s_retraced;
    grid_launch_next();
    // automatic choice: both kernels are launched, the one the order kernel did not choose leaves
    // (rays from the caller are the split packets' kernel's)
    if (*a.render_ellipsoids || *a.rays_from_python ||
        (a.auto_role != 0 && a.schedule[kStatChoice] != (uint32_t)a.auto_role)) {
        grid_wait_before();
        return;
    }
    if (threadIdx.x == 0) {
        s_packets = 0u;
        s_retraced = 0u;
    }
    const uint32_t items = a.schedule[kSchedItems];
    for (;;) {
        __syncthreads();  // every thread is done with the previous tile (s_next, the frontier, counts)
        if (threadIdx.x == 0) s_next = atomicAdd(a.schedule, 1u);
        __syncthreads();
        const uint32_t t = s_next;
        if (t >= items) break;
        const uint32_t tile = a.schedule[kSchedHeader + a.ntiles + t];
        const bool again =
            forward_tile<KB, false, kCamera>(a, (int)(tile % (uint32_t)a.tiles_x), (int)(tile / (uint32_t)a.tiles_x), 0, sh);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&s_packets, 1u);
            if (again) atomicAdd(&s_retraced, 1u);
        }
    }
    if (threadIdx.x == 0 && s_packets > 0u) {
        atomicAdd(&a.schedule[kStatPackets], s_packets);
        atomicAdd(&a.schedule[kStatRetraced], s_retraced);
    }
    grid_wait_before();
}

// The tiles whose rays, the caller's, are traversed one by one (kRayTile): a warp traces a packet.  The last of a
// forward's kernels: without such tiles its blocks leave at once, which costs the camera's frames nothing
// there (as the first, 500k / 640x480 336 to 344 us).  A block begins with the four packets of one tile (so that a few tiles spread over all SMs), and its
// warps then take the next packets each by itself, so that none waits for its tile's slowest.  The packets
// have 32 hit slots at four blocks per SM, whatever trace_variant says: origins of their own, with 16 or 32
// slots as for the camera's rays at six or four blocks and these, 19 000 Gaussians in a box / 256x200 752 and
// 661 us, 100k / 160x120 433 and 361, 100k / 1280x720 606 and 599, shuffled 9.25 and 9.36 ms (five blocks:
// 707, 391, 588 us, 8.9 ms, but 16x16 rays over 1M 3.36 to 3.53 ms).
constexpr int kRaySlots = 32, kRayBlocks = 4;

template <int KB, int MINB>
__global__ void __launch_bounds__(kFwdThreads, MINB) trace_forward_rays_kernel(const FwdArgs a) {
    __shared__ RayShared<KB> sh;
    grid_launch_next();
    if (*a.render_ellipsoids || !*a.rays_from_python || a.schedule[kSchedRays] == 0u) {
        grid_wait_before();
        return;
    }
    const uint32_t packets = kWarps * a.schedule[kSchedRays];
    const int lane = threadIdx.x & 31;
    uint32_t traced = 0u, retraced = 0u;
    for (uint32_t q = blockIdx.x * kWarps + (threadIdx.x >> 5); q < packets;) {
        const uint32_t tile = a.schedule[kSchedHeader + 2 * a.ntiles - 1 - q / kWarps];
        const bool again = forward_ray_packet<KB>(a, (int)(tile % (uint32_t)a.tiles_x),
                                                  (int)(tile / (uint32_t)a.tiles_x), (int)(q % kWarps), sh);
        traced++;
        retraced += again ? 1u : 0u;
        if (lane == 0) q = gridDim.x * kWarps + atomicAdd(a.schedule + kSchedRayNext, 1u);
        q = __shfl_sync(kFull, q, 0);
    }
    if (lane == 0 && traced > 0u) {
        atomicAdd(&a.schedule[kStatPackets], traced);
        atomicAdd(&a.schedule[kStatRetraced], retraced);
    }
    grid_wait_before();
}

// The split tiles' packets (see sched_order_kernel), and the tiles of the caller's rays that are traversed
// together; launched before the kernel of the whole tiles, which starts as soon as this one's blocks have
// and fills what they leave free.  A kernel of its own: with both bodies in one, the whole tiles' loop lost
// registers (3M / 1080p 2.28 to 2.33 ms with a run-time switch, 2.44 ms with two inlined bodies, 2.40 ms
// with a call).
template <int KB, int MINB>
__global__ void __launch_bounds__(kFwdThreads, MINB) trace_forward_split_kernel(const FwdArgs a) {
    __shared__ TileShared<KB, true> sh;
    auto &whole_sh = reinterpret_cast<TileShared<KB, false> &>(sh);
    static_assert(sizeof(TileShared<KB, false>) <= sizeof(sh), "whole tiles use the same memory");
    __shared__ uint32_t s_next, s_packets, s_retraced;
    grid_launch_next();
    if (*a.render_ellipsoids) return;
    const uint32_t items = a.schedule[kSchedSplitItems], whole = *a.rays_from_python ? a.schedule[kSchedItems] : 0u;
    if (items + whole == 0u) return;
    if (threadIdx.x == 0) {
        s_packets = 0u;
        s_retraced = 0u;
    }
    for (;;) {
        __syncthreads();  // every thread is done with the previous packet
        if (threadIdx.x == 0) s_next = atomicAdd(a.schedule + kSchedSplitNext, 1u);
        __syncthreads();
        const uint32_t t = s_next;
        if (t >= items + whole) break;
        bool again;
        if (t < items) {
            const uint32_t item = a.schedule[kSchedHeader + 2 * a.ntiles + t], tile = item & kItemTile;
            again = forward_tile<KB, true, kCones>(a, (int)(tile % (uint32_t)a.tiles_x),
                                                   (int)(tile / (uint32_t)a.tiles_x), (int)(item >> kItemShift), sh);
        } else {
            const uint32_t tile = a.schedule[kSchedHeader + a.ntiles + t - items];
            again = forward_tile<KB, false, kCones>(a, (int)(tile % (uint32_t)a.tiles_x),
                                                    (int)(tile / (uint32_t)a.tiles_x), 0, whole_sh);
        }
        if ((threadIdx.x & 31) == 0 && (threadIdx.x == 0 || t >= items)) {
            atomicAdd(&s_packets, 1u);
            if (again) atomicAdd(&s_retraced, 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_packets > 0u) {
        atomicAdd(&a.schedule[kStatPackets], s_packets);
        atomicAdd(&a.schedule[kStatRetraced], s_retraced);
    }
}

// ---------------------------------------------------------------------------------------------
// Work order of the forward's tiles and their BVH frontiers.  A tile's work follows the number of
// Gaussians its rays meet (per-packet time correlates 0.92 with hits), so the estimate is the number
// of leaves under the BVH nodes its frustum reaches, cut where a node holds at most `cut` leaves.
// Tiles are then counting-sorted by log2 of the estimate, largest first, so the launch does not end
// with a dense tile started late.  The nodes at the cut (and leaves reached above it) are the tile's
// frontier: every ray of the tile that hits a Gaussian reaches it through one of them, so the tile's
// packets start their traversals there instead of at the root (the top levels are walked once per
// tile, not once per packet traversal).  The frontier is sorted by its boxes' centres along the
// tile's mean direction, so packets visit it roughly front to back.  The tiles' walks share their
// top: a first pass walks each super-tile (kSuperTiles x kSuperTiles tiles) down to nodes of at
// most kSuperCut leaves and stores them with their boxes; a tile's walk then starts from its
// super-tile's entries, testing each entry's own box against the tile's frustum, instead of from the
// root.  Every leaf a ray of the tile can hit lies under an entry of the super-tile (its ancestors
// meet the tile's frustum, hence the super-tile's), so the tile still reaches it.  Schedule words:
// [0..5] work counters and lengths, [kSchedHeader, +ntiles) estimates, [kSchedHeader + ntiles, +ntiles) order of
// the whole tiles and, from its end backwards, the tiles of single rays, [kSchedHeader + 2 ntiles, +4 ntiles) the
// split tiles' packets, then (when frontiers are on) kFrontierWords words per tile, then kSuperWords words per
// super-tile.
// ---------------------------------------------------------------------------------------------
constexpr int kCostCut = 512;
constexpr int kCostStack = 512;  // (a super-tile's entries and what their walk pushes)
constexpr int kSuperTiles = 4;
constexpr uint32_t kSuperCut = 1024;
constexpr int kSuperMax = 255;          // entries of a super-tile frontier (fits the walk's buffer)
constexpr int kSuperEntryWords = 8;     // link, leaves below, box min xyz, box max xyz
constexpr int kSuperWords = 1 + kSuperMax * kSuperEntryWords;

struct FrontierScratch {
    Frustum fr;
    uint32_t stk[kCostStack];
    float key[kFrontierSort];
    uint32_t val[kFrontierSort];
    int entries;  // of val that the last walk filled
};

// What the super-tile walk also keeps of each frontier entry.
struct SuperScratch {
    float box[kFrontierSort][6];
    uint32_t leaves[kFrontierSort];
};

// Bitonic sort of the warp's nf (key, link) frontier entries (fs.key / fs.val, nf <= 32 * E) by key,
// written to out[1 .. nf].  The network runs in registers: element i sits in lane i % 32, slot i / 32;
// the partner at distance j < 32 is the same slot of lane ^ j (a shuffle), at j >= 32 the slot
// e ^ (j / 32) of the same lane.  Padding keys are +inf (sorted last); each pair (lower, upper)
// swaps iff (ascending ? k_upper < k_lower : k_lower < k_upper), so NaN keys never move and ties
// keep their places.
template <int E>
__device__ __forceinline__ void frontier_sort_out(const FrontierScratch &fs, int nf, uint32_t *out) {
    const int lane = threadIdx.x & 31;
    float k[E];
    uint32_t v[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int i = e * 32 + lane;
        k[e] = i < nf ? fs.key[i] : __int_as_float(0x7f800000);
        v[e] = i < nf ? fs.val[i] : GRAY_NULL;
    }
#pragma unroll
    for (int kk = 2; kk <= 32 * E; kk <<= 1) {
#pragma unroll
        for (int j = kk >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const int f = e ^ (j >> 5);
                    if (f > e) {
                        const bool up = ((e * 32 + lane) & kk) == 0;
                        const float kl = k[e], ku = k[f];
                        if (up ? (ku < kl) : (kl < ku)) {
                            k[e] = ku;
                            k[f] = kl;
                            const uint32_t t = v[e];
                            v[e] = v[f];
                            v[f] = t;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const float ko = __shfl_xor_sync(kFull, k[e], j);
                    const uint32_t vo = __shfl_xor_sync(kFull, v[e], j);
                    const bool up = ((e * 32 + lane) & kk) == 0;
                    const bool lower = (lane & j) == 0;
                    const float kl = lower ? k[e] : ko, ku = lower ? ko : k[e];
                    if (up ? (ku < kl) : (kl < ku)) {
                        k[e] = ko;
                        v[e] = vo;
                    }
                }
            }
        }
    }
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int i = e * 32 + lane;
        if (i < nf) out[1 + i] = v[e];
    }
}

// One warp walks the top of the BVH for a pixel rectangle whose frustum is in fs.fr: returns (on
// every lane) the number of leaves under the frontier, the nodes of at most `cut` leaves (and the
// leaves) it reaches; with `out`, writes the frontier there sorted front to back (count + entries),
// or a count of kFrontierNone when the frontier does not fit or the tree is malformed.  The walk ends
// there (or when its stack is full), and the leaves under the nodes it has not opened count in full: the
// densest tiles, whose frontiers do not fit, must not seem light (stopped with what had been reached, one
// tile of 6M Gaussians at 1280x720 was the last to start, 9.1 ms for a view that takes 2.2).  n > 1.
// seed (may be null; a count above kSuperMax means none): a super-tile frontier
// to start from instead of the root -- each entry whose box meets this frustum is walked further
// (more than `cut` leaves) or is a frontier entry.  SUPER: the walk of a super-tile; with `out` it
// writes its entries unsorted with their leaf counts and boxes (kSuperWords words), or
// kFrontierNone when they do not fit.
template <bool SUPER>
__device__ __forceinline__ uint32_t frontier_walk(const float4 *nodes, int n, uint32_t cut, FrontierScratch &fs,
                                               SuperScratch *ss, uint32_t *out, const uint32_t *seed) {
    const int lane = threadIdx.x & 31;
    const uint32_t lanemask_lt = (1u << lane) - 1u;
    const Frustum &fr = fs.fr;
    const float4 cdir = fr.pn[4];  // the near plane's normal: the rectangle's mean direction
    uint32_t est = 0;
    uint32_t pending = 0;  // leaves under the nodes on the stack (this lane's pushes less its pops, modulo 2^32)
    int nf = 0, sp = 0;
    bool complete = true, stop = false;
    const uint32_t nseed = seed ? seed[0] : kFrontierNone;
    if (nseed <= (uint32_t)kSuperMax) {
        for (int b0 = 0; b0 < (int)nseed; b0 += 32) {
            const int i = b0 + lane;
            bool push = false, rec = false, bad = false;
            uint32_t link = 0;
            float key = 0.0f;
            if (i < (int)nseed) {
                const uint32_t *e = seed + 1 + (size_t)i * kSuperEntryWords;
                link = e[0];
                const uint32_t lv = e[1];
                const float bmin[3] = {__uint_as_float(e[2]), __uint_as_float(e[3]), __uint_as_float(e[4])};
                const float bmax[3] = {__uint_as_float(e[5]), __uint_as_float(e[6]), __uint_as_float(e[7])};
                if (frustum_box(fr, bmin, bmax)) {
                    if (link & GRAY_LEAF_BIT) {
                        rec = (link & ~GRAY_LEAF_BIT) < (uint32_t)n;
                        bad = !rec;
                        est += rec ? 1u : 0u;
                    } else if (link < (uint32_t)(n - 1)) {
                        push = lv > cut;
                        rec = !push;
                        if (rec) est += lv;
                    } else {
                        bad = true;
                    }
                    if (push) pending += lv;
                    key = fmaf(bmin[2] + bmax[2], cdir.z, fmaf(bmin[1] + bmax[1], cdir.y, (bmin[0] + bmax[0]) * cdir.x));
                }
            }
            if (__any_sync(kFull, bad)) complete = false;
            const uint32_t mp = __ballot_sync(kFull, push);
            if (push) fs.stk[sp + __popc(mp & lanemask_lt)] = link;
            sp += __popc(mp);
            const uint32_t mr = __ballot_sync(kFull, rec);
            const int at = nf + __popc(mr & lanemask_lt);
            if (rec && at < kFrontierSort) {
                fs.key[at] = key;
                fs.val[at] = link;
            }
            nf += __popc(mr);
        }
    } else {
        if (lane == 0) {
            fs.stk[0] = 0u;
            pending = (uint32_t)n;
        }
        sp = 1;
    }
    __syncwarp();
    for (int guard = 0; sp > 0; guard++) {
        // a popped node frees its entry and pushes at most two
        const int take = min(min(sp, 32), kCostStack - sp);
        if (guard >= 4096 || nf > (SUPER ? kSuperMax : kFrontierMax) || take <= 0) {
            complete = false;
            stop = true;
            break;
        }
        uint32_t node = GRAY_NULL;
        if (lane < take) node = fs.stk[sp - 1 - lane];
        __syncwarp();
        sp -= take;
        // children as (a, b) = (nearer, farther) along the rectangle's mean direction, as the forward
        uint32_t ca = 0, cb = 0, la = 0, lb = 0;  // children and the leaves below them
        bool pa = false, pb = false, bad = false;
        float sa = 0.0f, sb = 0.0f;
        float boxa[6], boxb[6];
        if (node != GRAY_NULL) {
            if (node >= (uint32_t)(n - 1)) {
                bad = true;
            } else {
                const float4 q0 = nodes[4 * node], q1 = nodes[4 * node + 1], q2 = nodes[4 * node + 2],
                             q3 = nodes[4 * node + 3];
                const float b0min[3] = {q0.x, q0.y, q0.z}, b0max[3] = {q0.w, q1.x, q1.y};
                const float b1min[3] = {q1.z, q1.w, q2.x}, b1max[3] = {q2.y, q2.z, q2.w};
                const uint32_t c0 = __float_as_uint(q3.x), c1 = __float_as_uint(q3.y);
                const uint32_t l0 = __float_as_uint(q3.w), l1 = __float_as_uint(q3.z) - l0;
                pending -= l0 + l1;
                const bool p0 = frustum_box(fr, b0min, b0max), p1 = frustum_box(fr, b1min, b1max);
                const float s0 = fmaf(q0.z + q1.y, cdir.z, fmaf(q0.y + q1.x, cdir.y, (q0.x + q0.w) * cdir.x));
                const float s1 = fmaf(q2.x + q2.w, cdir.z, fmaf(q1.w + q2.z, cdir.y, (q1.z + q2.y) * cdir.x));
                const bool sw = s1 < s0;
                ca = sw ? c1 : c0;
                cb = sw ? c0 : c1;
                pa = sw ? p1 : p0;
                pb = sw ? p0 : p1;
                sa = sw ? s1 : s0;
                sb = sw ? s0 : s1;
                la = sw ? l1 : l0;
                lb = sw ? l0 : l1;
                if constexpr (SUPER) {
                    const float c0b[6] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y};
                    const float c1b[6] = {q1.z, q1.w, q2.x, q2.y, q2.z, q2.w};
#pragma unroll
                    for (int k = 0; k < 6; k++) {
                        boxa[k] = sw ? c1b[k] : c0b[k];
                        boxb[k] = sw ? c0b[k] : c1b[k];
                    }
                }
            }
        }
        // internal children above the cut are walked further; leaves and nodes at the cut are
        // frontier entries
        bool ia = false, ib = false, fa = false, fb = false;
        if (pa) {
            if (ca & GRAY_LEAF_BIT) {
                fa = (ca & ~GRAY_LEAF_BIT) < (uint32_t)n;
                bad = bad || !fa;
                est += fa ? 1u : 0u;
            } else if (ca < (uint32_t)(n - 1)) {
                ia = la > cut;
                fa = !ia;
                if (fa) est += la;
            } else {
                bad = true;
            }
        }
        if (pb) {
            if (cb & GRAY_LEAF_BIT) {
                fb = (cb & ~GRAY_LEAF_BIT) < (uint32_t)n;
                bad = bad || !fb;
                est += fb ? 1u : 0u;
            } else if (cb < (uint32_t)(n - 1)) {
                ib = lb > cut;
                fb = !ib;
                if (fb) est += lb;
            } else {
                bad = true;
            }
        }
        // a malformed tree: leave it to the forward's own checks (root start)
        if (__any_sync(kFull, bad)) complete = false;
        if (ia) pending += la;
        if (ib) pending += lb;
        const uint32_t ma = __ballot_sync(kFull, ia), mb = __ballot_sync(kFull, ib);
        const int ni = __popc(ma) + __popc(mb);
        const int above = __popc(ma & lanemask_lt) + __popc(mb & lanemask_lt);
        if (ia) fs.stk[sp + ni - 1 - above] = ca;
        if (ib) fs.stk[sp + ni - 1 - above - (ia ? 1 : 0)] = cb;
        sp += ni;
        const uint32_t qa = __ballot_sync(kFull, fa), qb = __ballot_sync(kFull, fb);
        const int before = nf + __popc(qa & lanemask_lt) + __popc(qb & lanemask_lt);
        if (fa && before < kFrontierSort) {
            fs.key[before] = sa;
            fs.val[before] = ca;
            if constexpr (SUPER) {
                ss->leaves[before] = (ca & GRAY_LEAF_BIT) ? 1u : la;
#pragma unroll
                for (int k = 0; k < 6; k++) ss->box[before][k] = boxa[k];
            }
        }
        const int bb = before + (fa ? 1 : 0);
        if (fb && bb < kFrontierSort) {
            fs.key[bb] = sb;
            fs.val[bb] = cb;
            if constexpr (SUPER) {
                ss->leaves[bb] = (cb & GRAY_LEAF_BIT) ? 1u : lb;
#pragma unroll
                for (int k = 0; k < 6; k++) ss->box[bb][k] = boxb[k];
            }
        }
        nf += __popc(qa) + __popc(qb);
        __syncwarp();
    }
    if (stop) est += pending;
    if (lane == 0) fs.entries = min(nf, kFrontierSort);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) est += __shfl_xor_sync(kFull, est, off);
    if (!out) return est;
    if constexpr (SUPER) {
        if (complete && nf <= kSuperMax) {
            for (int i = lane; i < nf; i += 32) {
                uint32_t *e = out + 1 + (size_t)i * kSuperEntryWords;
                e[0] = fs.val[i];
                e[1] = ss->leaves[i];
#pragma unroll
                for (int k = 0; k < 6; k++) e[2 + k] = __float_as_uint(ss->box[i][k]);
            }
            if (lane == 0) out[0] = (uint32_t)nf;
        } else if (lane == 0) {
            out[0] = kFrontierNone;
        }
        return est;
    }
    if (complete && nf <= kFrontierMax) {
        if (nf <= 32) frontier_sort_out<1>(fs, nf, out);
        else if (nf <= 64) frontier_sort_out<2>(fs, nf, out);
        else if (nf <= 128) frontier_sort_out<4>(fs, nf, out);
        else frontier_sort_out<8>(fs, nf, out);
        if (lane == 0) out[0] = (uint32_t)nf;
    } else if (lane == 0) {
        out[0] = kFrontierNone;
    }
    return est;
}

// The frustum of the camera's rays through a pixel rectangle (a warp together).
__device__ __forceinline__ void make_tile_frustum(const FwdArgs &a, int x0, int y0, int x1, int y1, Frustum &fr) {
    make_frustum_warp(fr, mk3(a.cam_origin[0], a.cam_origin[1], a.cam_origin[2]), a.w2c, *a.fov, x0, y0, x1, y1,
                      a.render_w, a.render_h, a.root_box, *a.jitter ? 0.5f : 0.0f);
}

// Coarse frontiers of the super-tiles (kSuperTiles x kSuperTiles block tiles each), one warp each.  Not for the
// caller's rays: a warp would read 2048 of them first (60 us), more than the walks that start at the root take.
__global__ void __launch_bounds__(32) super_cost_kernel(const FwdArgs a, int bw, int bh, int nsuper) {
    __shared__ FrontierScratch fs;
    __shared__ SuperScratch ss;
    const int st = blockIdx.x, lane = threadIdx.x;
    if (st >= nsuper) return;
    uint32_t *out = a.super_frontier + (size_t)st * kSuperWords;
    const int n = a.n;
    if (*a.render_ellipsoids || *a.rays_from_python || n <= 1) {
        if (lane == 0) out[0] = kFrontierNone;
        return;
    }
    const int x0 = (st % a.super_x) * kSuperTiles * bw, y0 = (st / a.super_x) * kSuperTiles * bh;
    const int x1 = min(x0 + kSuperTiles * bw, (int)a.render_w) - 1;
    const int y1 = min(y0 + kSuperTiles * bh, (int)a.render_h) - 1;
    make_tile_frustum(a, x0, y0, x1, y1, fs.fr);
    frontier_walk<true>(a.nodes, n, kSuperCut, fs, &ss, out, nullptr);
}

// Whether the Gaussians that the rays in cb's cone may hit are met by fewer than `least` of them on average:
// each lane follows one of the walk's frontier entries down to a Gaussian and compares its extent, seen
// from the rays' origin, with the cone's; up to three times more while the answer is within a factor of two.
// Not inlined: its registers would cost the walks of the camera's tiles (1M Gaussians, 64x64 537 to 543 us).
__device__ __noinline__ bool sparse_tile(const float4 *__restrict__ nodes, const float4 *__restrict__ l2w, int n,
                                         const FrontierScratch &fs, const ConicBasis &cb, float least) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const int entries = fs.entries, take = min(entries, 32);
    float sum = 0.0f, found = 0.0f;
    for (int round = 0; round < 4; round++) {
        uint32_t link = lane < take ? fs.val[(4 * lane + round) * entries / (4 * take)] : GRAY_NULL;
        for (int guard = 0; guard < 64 && !(link & GRAY_LEAF_BIT); guard++) {
            if (link >= (uint32_t)(n - 1)) {
                link = GRAY_NULL;
                break;
            }
            const float4 q0 = nodes[4 * (size_t)link], q1 = nodes[4 * (size_t)link + 1],
                         q2 = nodes[4 * (size_t)link + 2], q3 = nodes[4 * (size_t)link + 3];
            const float b0min[3] = {q0.x, q0.y, q0.z}, b0max[3] = {q0.w, q1.x, q1.y};
            const float b1min[3] = {q1.z, q1.w, q2.x}, b1max[3] = {q2.y, q2.z, q2.w};
            const bool p0 = frustum_box(fs.fr, b0min, b0max), p1 = frustum_box(fs.fr, b1min, b1max);
            const bool second = p0 && p1 ? (((lane ^ (7 * round)) >> (guard % 5)) & 1) != 0 : p1;
            link = !(p0 || p1) ? GRAY_NULL : __float_as_uint(second ? q3.y : q3.x);
        }
        const uint32_t gid = link & ~GRAY_LEAF_BIT;
        const bool on = link != GRAY_NULL && (link & GRAY_LEAF_BIT) && gid < (uint32_t)n;
        float met = 0.0f;
        if (on) {
            const float4 r0 = l2w[3 * (size_t)gid], r1 = l2w[3 * (size_t)gid + 1], r2 = l2w[3 * (size_t)gid + 2];
            const float size = (2.0f / 3.0f) * (norm_approx(mk3(r0.x, r0.y, r0.z)) + norm_approx(mk3(r1.x, r1.y, r1.z)) +
                                                norm_approx(mk3(r2.x, r2.y, r2.z)));
            const float z = (r0.w - cb.origin[0]) * cb.axis[0] + (r1.w - cb.origin[1]) * cb.axis[1] +
                            (r2.w - cb.origin[2]) * cb.axis[2];
            const float seen = z > size ? size / z : 1.0f;
            met = cb.share * (float)kFwdThreads * fminf(1.0f, seen / (2.0f * cb.hx)) * fminf(1.0f, seen / (2.0f * cb.hy));
            met = fminf(met, 4.0f * least);  // (a few near or large ones say little of the rest)
        }
        found += (float)__popc(__ballot_sync(kFull, on));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) met += __shfl_xor_sync(kFull, met, off);
        sum += met;
        if (!(sum > 0.5f * least * found && sum < 2.0f * least * found)) break;
    }
    return sum < least * found;
}

// Which tiles of the caller's rays are traversed together: those whose rays share a cone (ray_cone), over more than a
// few Gaussians, unless the candidates are many and met by few of the rays (rays all over the view in any
// order, thumbnails, 16x16 rays for a whole scene).  The others' estimate is kRayTile.  A tile's time grows with its
// candidates, est; that of its rays one by one with the hits and more slowly.  Measured, rays met per
// candidate, est, together against one by one:
//   tiles that fill the SMs: 0.02, 7e3: 3.1 and 2.3 ms; 0.37, 2e4: 58 and 43; 0.05, 3.5e4: 15.0 and 6.9;
//     0.08, 3.5e5: 364 and 35; 0.7 (0.2 to 17), 2e3: 0.17 and 0.57
//   few tiles: 0.014, 7e3: 0.14 and 0.29; 0.05, 3.5e4: 0.30 and 0.73; 0.015, 6.5e4: 1.3 and 0.76; 0.08,
//     3.5e5: 2.8 and 4.8; 0.03, 6.5e5: 15 and 4.1; 0.11, 1e6: 8.3 and 10.9
// so the line is at 3.2e-3 and 1.1e-4 sqrt(est) rays.  Without candidates to speak of, one by one is faster:
// 64 Gaussians / 64x64 40 us and 49 (105 when every tile was walked), 200 / 1280x720 126 us and 161, 400 / 1280x720
// 1.00 to 1.07 times.
constexpr int kTogetherIdle = 128, kTogetherLoaded = 512;
constexpr uint32_t kSparseFrom = 512;
constexpr float kSparseIdle = 1.2e-8f, kSparseLoaded = 1.0e-5f;  // squares of the factors

__global__ void __launch_bounds__(32, 32) tile_cost_kernel(const FwdArgs a, int bw, int bh) {
    __shared__ FrontierScratch fs;
    __shared__ ConicBasis cb;
    __shared__ float s_sparse;  // factor of the caller's rays, 0 for the camera's (in no register over the walk)
    const int tile = blockIdx.x, lane = threadIdx.x;
    uint32_t *out = a.frontier ? a.frontier + (size_t)tile * kFrontierWords : nullptr;
    const int n = a.n;
    bool walk = !*a.render_ellipsoids && n > 1, single = false;
    if (walk) {
        const int x0 = (tile % a.tiles_x) * bw, y0 = (tile / a.tiles_x) * bh;
        const int x1 = min(x0 + bw, (int)a.render_w) - 1, y1 = min(y0 + bh, (int)a.render_h) - 1;
        if (*a.rays_from_python) {
            const bool loaded = 2 * a.ntiles > a.slots_split;
            if (lane == 0) s_sparse = loaded ? kSparseLoaded : kSparseIdle;
            walk = n > (loaded ? kTogetherLoaded : kTogetherIdle) &&
                   ray_cone<32>(a.ray_o, a.ray_d, a.alloc_w, a.root_box, x0, y0, x1, y1, fs.fr, cb, nullptr);
            single = !walk;
        } else {
            if (lane == 0) s_sparse = 0.0f;
            make_tile_frustum(a, x0, y0, x1, y1, fs.fr);
        }
    }
    if (!walk) {
        if (lane == 0) {
            if (out) out[0] = kFrontierNone;
            a.schedule[kSchedHeader + tile] = single ? kRayTile : 0u;
        }
        return;
    }
    const uint32_t *seed = nullptr;
    if (a.super_frontier) {
        const int sx = (tile % a.tiles_x) / kSuperTiles, sy = (tile / a.tiles_x) / kSuperTiles;
        seed = a.super_frontier + (size_t)(sy * a.super_x + sx) * kSuperWords;
    }
    uint32_t est = frontier_walk<false>(a.nodes, n, a.frontier_cut > 0 ? a.frontier_cut : (uint32_t)kCostCut, fs,
                                        nullptr, out, seed);
    const float factor = *(volatile float *)&s_sparse;
    if (factor > 0.0f && est > kSparseFrom && sparse_tile(a.nodes, a.l2w, n, fs, cb, sqrt_approx((float)est * factor)))
        est = kRayTile;
    if (lane == 0) a.schedule[kSchedHeader + tile] = est;
}

// The work order, one block: the tiles counting-sorted by log2 of their estimates, densest first, so that
// the launch does not end with a dense tile started late; and the automatic kernel choice for this
// forward from the last scheduled forward's packet counts (the narrow kernel when there are none yet).
//
// Dense tiles are split.  A tile whose estimate exceeds kSplitEighths / 8 of what the resident blocks
// have to do on average (the sum of the estimates over the blocks resident at once) may still run when
// the others are done: it is entered as its four packets, each traced by a block whose four warps share
// its candidates (merge_split).  Below kSplitLeast leaves a tile is too short for that to pay.  Split, a
// tile costs more (all of them split: 3M / 1080p 2.27 -> 5.09 ms), so all such tiles are only in frames of up
// to slots / 4 tiles (a tile or so per SM) and where the densest has kSplitSteep times the average: the
// others are done long before it.  Half that will do from kSplitLong leaves on, where the densest tile takes
// about as long as such a frame and a block's share is some long tiles (5.5M / 357x204: at most 50 split 2439
// us, all 1763; 200 000 in a box / 480x360, all alike and as dense: 17 split 3500, 450 4460).  Else the
// densest are, about slots / 12 in a frame of up to slots tiles
// and slots / 6 in a larger one.  "About": a quarter octave of estimates is split or left together, so that a
// frame of tiles alike is left whole.  Measured over 215 frames (scenes of 1000 to 5.5M Gaussians, 89x69 to
// 3840x2160, seen from outside and within), each with 2 to 16 thresholds: this rule is 4.0% (geometric mean)
// and at most 26% above the best threshold and at most 1% above splitting all candidates, which is 10% and
// 91% above it; none split is 27% and 347%.  10 000 in a box / 640x480 from afar: none 191 us, 64 tiles 243,
// all 420 candidates 322; 500k / 640x480 none 394, 32 379, 64 286, 169 324, all tiles 559; 1.9M / 260x349
// (the densest 5.4 times the average) none 2154, 64 1179, 304 656.  On the caller's rays up to slots / 2: whole,
// their tiles have 16 hit slots, split 64 (160 thumbnail tiles over 1M: whole 30 ms, split 3).
constexpr int kOrderThreads = 1024;
constexpr int kOrderAhead = 8;
constexpr int kOrderBuckets = 33;  // leading zeros of an estimate
constexpr unsigned long long kSplitEighths = 5;
constexpr uint32_t kSplitLeast = 96;
constexpr int kSplitBuckets = 128;  // four per octave of an estimate

__device__ __forceinline__ int split_bucket(uint32_t e) {  // e >= kSplitLeast
    const int octave = 31 - __clz((int)e);
    return 4 * octave + (int)((e >> (octave - 2)) & 3u);
}

constexpr unsigned long long kSplitSteep = 5;
constexpr uint32_t kSplitLong = 16384;

// The lowest bucket edge with at most `limit` candidates from it on (counts: candidates per bucket), less one;
// 0xffffffff if the densest bucket holds more.  One warp.
__device__ __forceinline__ uint32_t split_above(const uint32_t *counts, uint32_t limit) {
    const int lane = threadIdx.x & 31, first = kSplitBuckets - 4 - 4 * lane;  // the densest in lane 0
    const uint32_t own = counts[first] + counts[first + 1] + counts[first + 2] + counts[first + 3];
    uint32_t from = own;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, from, off);
        if (lane >= off) from += v;
    }
    from -= own;  // candidates of the denser lanes
    uint32_t edge = 0xffffffffu;
#pragma unroll
    for (int j = 3; j >= 0; j--) {
        const int b = first + j;
        from += counts[b];
        if (counts[b] > 0u && from <= limit) edge = ((uint32_t)(4 + (b & 3)) << (b / 4 - 2)) - 1u;
    }
    return __reduce_min_sync(kFull, edge);
}

constexpr int kSplitBlocks = 4;  // blocks per SM of the split kernel

__global__ void __launch_bounds__(kOrderThreads) sched_order_kernel(uint32_t *sched, int ntiles, int slots_narrow,
                                                                    int slots_wide, int slots_split, int never_split,
                                                                    const uint8_t *rays_from_python) {
    __shared__ unsigned long long s_sum[32];
    __shared__ uint32_t s_max[32], s_dense[kSplitBuckets], s_candidates, s_limit;
    __shared__ uint32_t s_bucket[2 * kOrderBuckets + 1];  // whole tiles, then split ones; tiles of single rays
    __shared__ uint32_t s_split;
    const int t = threadIdx.x, lane = t & 31;
    const uint32_t *est = sched + kSchedHeader;
    const bool given = *rays_from_python;
    unsigned long long sum = 0ull;
    uint32_t most = 0u;
#pragma unroll 8
    for (int i = t; i < ntiles; i += kOrderThreads) {
        const uint32_t e = est[i] != kRayTile ? est[i] : 0u;
        sum += e;
        most = max(most, e);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(kFull, sum, off);
    most = __reduce_max_sync(kFull, most);
    if (lane == 0) {
        s_sum[t >> 5] = sum;
        s_max[t >> 5] = most;
    }
    if (t < kSplitBuckets) s_dense[t] = 0u;
    if (t == 0) s_candidates = 0u;
    if (t <= 2 * kOrderBuckets) s_bucket[t] = 0u;
    __syncthreads();
    if (t == 0) {
        const uint32_t packets = sched[kStatPackets], retraced = sched[kStatRetraced];
        uint32_t choice = sched[kStatChoice];
        if (choice != kChoiceNarrow && choice != kChoiceWide) choice = kChoiceNarrow;
        if (packets > 0u && retraced <= packets) {
            const uint32_t most = ntiles <= kWideTiles * slots_narrow ? kWideSmall : kWideLarge;
            choice = (unsigned long long)retraced * 128ull > (unsigned long long)packets * most ? kChoiceWide
                                                                                                 : kChoiceNarrow;
        }
        sched[kStatChoice] = choice;
        sched[kStatPackets] = 0u;
        sched[kStatRetraced] = 0u;
        sched[0] = 0u;
        sched[kSchedSplitNext] = 0u;
        sched[kSchedRayNext] = 0u;
        unsigned long long total = 0ull;
        for (int w = 0; w < kOrderThreads / 32; w++) total += s_sum[w];
        // (the split kernel has all tiles of the caller's rays)
        const unsigned long long slots = (unsigned long long)(given                   ? slots_split
                                                              : choice == kChoiceWide ? slots_wide
                                                                                      : slots_narrow);
        const unsigned long long thr = total * kSplitEighths / (8ull * (slots > 0ull ? slots : 1ull));
        uint32_t densest = 0u;
        for (int w = 0; w < kOrderThreads / 32; w++) densest = max(densest, s_max[w]);
        const uint32_t above = thr < kSplitLeast ? kSplitLeast : thr < 0xffffffffull ? (uint32_t)thr : 0xffffffffu;
        s_split = never_split || densest <= above ? 0xffffffffu : above;
        const uint32_t n = (uint32_t)ntiles, places = (uint32_t)slots;
        const bool steep = 2ull * densest * slots >= (densest >= kSplitLong ? kSplitSteep : 2ull * kSplitSteep) * total;
        s_limit = n <= places / (given ? 2u : 4u) || steep ? 0xffffffffu : places / (n <= places ? 12u : 6u);
    }
    __syncthreads();
    uint32_t split = s_split;
    if (split != 0xffffffffu) {
        for (int i0 = 0; i0 < ntiles; i0 += kOrderThreads) {
            const uint32_t e = i0 + t < ntiles ? est[i0 + t] : 0u;
            const bool dense = e > split && e != kRayTile;
            if (dense) atomicAdd(&s_dense[split_bucket(e)], 1u);
            const uint32_t c = (uint32_t)__popc(__ballot_sync(kFull, dense));
            if (lane == 0 && c > 0u) atomicAdd(&s_candidates, c);
        }
        __syncthreads();
        if (t < 32) {
            if (s_candidates > s_limit) split = split_above(s_dense, s_limit);
            if (t == 0) s_split = split;
        }
        __syncthreads();
        split = s_split;
    }
    for (int pass = 0; pass < 2; pass++) {
        // pass 0 counts the buckets' tiles, pass 1 writes them; the lanes of a warp that fall in one
        // bucket share an atomic
        uint32_t ahead[kOrderAhead];  // estimates of the next rounds, loaded together
        for (int i0 = 0, r = 0; i0 < ntiles; i0 += kOrderThreads, r = (r + 1) % kOrderAhead) {
            const int i = i0 + t;
            if (r == 0) {
#pragma unroll
                for (int j = 0; j < kOrderAhead; j++)
                    ahead[j] = i + j * kOrderThreads < ntiles ? est[i + j * kOrderThreads] : 0u;
            }
            const uint32_t e = ahead[0];
#pragma unroll
            for (int j = 0; j + 1 < kOrderAhead; j++) ahead[j] = ahead[j + 1];
            const bool single = e == kRayTile, four = e > split && !single;
            const uint32_t key = i >= ntiles ? 2u * kOrderBuckets + 1u
                                 : single    ? 2u * kOrderBuckets
                                             : (uint32_t)__clz((int)e) + (four ? (uint32_t)kOrderBuckets : 0u);  // dense first
            const uint32_t peers = __match_any_sync(kFull, key);
            const int lead = __ffs((int)peers) - 1;
            uint32_t base = 0u;
            if (lane == lead && i < ntiles) base = atomicAdd(&s_bucket[key], (uint32_t)__popc(peers));
            base = __shfl_sync(kFull, base, lead) + __popc(peers & ((1u << lane) - 1u));
            if (pass == 1 && i < ntiles) {
                uint32_t *out = sched + kSchedHeader + ntiles;
                if (single) {
                    out[ntiles - 1 - (int)base] = (uint32_t)i;  // (the whole tiles' order fills from the front)
                } else if (four) {
                    out += ntiles + 4u * base;
                    for (uint32_t s = 0; s < 4u; s++) out[s] = (uint32_t)i | s << kItemShift;
                } else {
                    out[base] = (uint32_t)i;
                }
            }
        }
        __syncthreads();
        if (pass == 0 && t < 2) {
            uint32_t acc = 0u;
            for (int k = 0; k < kOrderBuckets; k++) {
                const uint32_t c = s_bucket[t * kOrderBuckets + k];
                s_bucket[t * kOrderBuckets + k] = acc;
                acc += c;
            }
            sched[t == 0 ? kSchedItems : kSchedSplitItems] = t == 0 ? acc : 4u * acc;
        }
        if (pass == 0 && t == 2) {
            sched[kSchedRays] = s_bucket[2 * kOrderBuckets];
            s_bucket[2 * kOrderBuckets] = 0u;
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------------
// Ellipsoid view (reference: cuda/ellipsoid_viewer.cu:1-94): closest-hit ray tracing of each
// Gaussian's support ellipsoid (the unit sphere of its snapshot frame), flat-shaded.  A Gaussian
// takes part if its snapshot marked it visible and its live opacity is >= ellipsoid_min_opacity.
// Per Gaussian the hit distance is the near root t0 = (s - h) / |ld| of the object-space ray when
// t0 >= znear, else the far root t1 = (s + h) / |ld|; the ray keeps the smallest distance in
// [znear, zfar] (equal distances: the smaller gaussian id, where OptiX keeps whichever its
// traversal reported first).  Output: RGB = max(0.5, <-view, normal>) (colour + 0.15) and depth =
// t, or the background and depth 0 on a miss; an inactive pixel (zero direction) is left as is.
// ---------------------------------------------------------------------------------------------
constexpr int kEllStack = 64;

// Distance of the ray's hit on Gaussian gid's ellipsoid, if it has one at or beyond tmin.
__device__ __forceinline__ bool ellipsoid_hit(const float4 g0, const float4 g1, const float4 g2, f3 ro, f3 rd,
                                              float tmin, float &t) {
    LocalHit h;
    local_ray(g0, g1, g2, ro, rd, h);
    if (h.b > 0.0f) return false;  // centre behind the ray
    const float norm = sqrtf(fdot3(h.ld, h.ld));
    const f3 dn = mk3(h.ld.x / norm, h.ld.y / norm, h.ld.z / norm);
    const float smid = -fdot3(h.lo, dn);
    const f3 u = mk3(fmaf(smid, dn.x, h.lo.x), fmaf(smid, dn.y, h.lo.y), fmaf(smid, dn.z, h.lo.z));
    const float sq = fdot3(u, u);
    if (sq > 1.0f) return false;
    const float hc = sqrtf(1.0f - sq);
    const float t0 = (smid - hc) / norm, t1 = (smid + hc) / norm;
    t = t0 >= tmin ? t0 : t1;
    return t >= tmin;
}

// Flat shading of the winning hit: object-space normal at the hit, carried to world space by the
// transpose of the snapshot matrix M (the inverse-transpose of the instance transform).
__device__ __forceinline__ void ellipsoid_shade(const float4 g0, const float4 g1, const float4 g2, f3 ro, f3 rd,
                                                float t, const float *c, float &r0, float &r1, float &r2) {
    LocalHit h;
    local_ray(g0, g1, g2, ro, rd, h);
    const float norm = sqrtf(fdot3(h.ld, h.ld));
    const f3 dn = mk3(h.ld.x / norm, h.ld.y / norm, h.ld.z / norm);
    const float tn = t * norm;
    f3 ln = mk3(fmaf(tn, dn.x, h.lo.x), fmaf(tn, dn.y, h.lo.y), fmaf(tn, dn.z, h.lo.z));
    const float ll = sqrtf(fdot3(ln, ln));
    ln = mk3(ln.x / ll, ln.y / ll, ln.z / ll);
    f3 wn = mk3(fmaf(ln.z, g2.x, fmaf(ln.y, g1.x, ln.x * g0.x)), fmaf(ln.z, g2.y, fmaf(ln.y, g1.y, ln.x * g0.y)),
                fmaf(ln.z, g2.z, fmaf(ln.y, g1.z, ln.x * g0.z)));
    const float wl = sqrtf(fdot3(wn, wn));
    wn = mk3(wn.x / wl, wn.y / wl, wn.z / wl);
    const float dl = sqrtf(fdot3(rd, rd));
    const f3 vd = mk3(rd.x / dl, rd.y / dl, rd.z / dl);
    const float align = fmaxf(0.5f, -fdot3(vd, wn));
    r0 = align * (c[0] + 0.15f);
    r1 = align * (c[1] + 0.15f);
    r2 = align * (c[2] + 0.15f);
}

// Entry distance of the ray into a box (slab test of SlabRay), or false if it misses.
__device__ __forceinline__ bool slab_enter(const float bmin[3], const float bmax[3], const SlabRay &r, float &tn) {
    float ta = fmaf(bmin[0], r.inv.x, r.clo.x), tb = fmaf(bmax[0], r.inv.x, r.chi.x);
    float n0 = fminf(ta, tb), f0 = fmaxf(ta, tb);
    ta = fmaf(bmin[1], r.inv.y, r.clo.y);
    tb = fmaf(bmax[1], r.inv.y, r.chi.y);
    n0 = fmaxf(n0, fminf(ta, tb));
    f0 = fminf(f0, fmaxf(ta, tb));
    ta = fmaf(bmin[2], r.inv.z, r.clo.z);
    tb = fmaf(bmax[2], r.inv.z, r.chi.z);
    n0 = fmaxf(n0, fminf(ta, tb));
    f0 = fminf(f0, fmaxf(ta, tb));
    tn = n0;
    return n0 <= f0 && f0 >= 0.0f;
}

__device__ __forceinline__ void ellipsoid_leaf(const FwdArgs &a, uint32_t gid, f3 ro, f3 rd, float znear, float minop,
                                               float &best, uint32_t &bid) {
    if (a.live[gid].x < minop) return;
    float t;
    if (!ellipsoid_hit(a.geom[3 * gid], a.geom[3 * gid + 1], a.geom[3 * gid + 2], ro, rd, znear, t)) return;
    if (t < best || (t == best && gid < bid)) {
        best = t;
        bid = gid;
    }
}

constexpr int kEllTileX = 16, kEllTileY = 8;

__device__ __forceinline__ void ellipsoid_pixel(const FwdArgs &a, int px, int py) {
    if (px >= (int)a.render_w || py >= (int)a.render_h) return;
    const uint32_t pixel = (uint32_t)py * a.alloc_w + (uint32_t)px;
    if (!a.display && *a.grads_enabled) raise_status(a.status, GRAY_STATUS_BAD_MODE);
    f3 ro, rd;
    if (*a.rays_from_python) {
        ro = mk3(a.ray_o[3 * pixel], a.ray_o[3 * pixel + 1], a.ray_o[3 * pixel + 2]);
        rd = mk3(a.ray_d[3 * pixel], a.ray_d[3 * pixel + 1], a.ray_d[3 * pixel + 2]);
    } else {
        ro = mk3(a.cam_origin[0], a.cam_origin[1], a.cam_origin[2]);
        float jx = 0.0f, jy = 0.0f;
        if (*a.jitter) {
            uint32_t h = pcg_hash(pixel ^ pcg_hash(*a.total_num_calls));
            jx = (float)(h & 0xFFFFu) * 0x1.0p-16f - 0.5f;
            jy = (float)(h >> 16) * 0x1.0p-16f - 0.5f;
        }
        rd = camera_ray(a.w2c, *a.fov, px, py, a.render_w, a.render_h, jx, jy);
    }
    a.head[pixel] = GRAY_NULL;  // no backward hit list for this frame
    if (sqrtf(dot3(rd, rd)) == 0.0f) return;
    const float znear = *a.znear, minop = *a.ellipsoid_min_opacity;
    float best = *a.zfar;
    uint32_t bid = GRAY_NULL;
    const int n = a.n;
    const SlabRay sr = make_slab_ray(ro, rd, 2.0e-6f * (fabsf(ro.x) + fabsf(ro.y) + fabsf(ro.z)));
    if (n == 1) {
        ellipsoid_leaf(a, 0u, ro, rd, znear, minop, best, bid);
    } else if (n > 1) {
        uint32_t stk[kEllStack];
        int sp = 0;
        float tr;
        const float *rb = a.root_box;
        const float rmin[3] = {rb[0], rb[1], rb[2]}, rmax[3] = {rb[4], rb[5], rb[6]};
        if (slab_enter(rmin, rmax, sr, tr) && tr <= best) stk[sp++] = 0u;
        long long budget = 2LL * n;
        while (sp > 0) {
            if (--budget < 0) {
                raise_status(a.status, GRAY_STATUS_STACK_OVERFLOW);
                break;
            }
            const uint32_t node = stk[--sp];
            if (node >= (uint32_t)(n - 1)) {
                raise_status(a.status, GRAY_STATUS_STACK_OVERFLOW);
                continue;
            }
            const float4 q0 = a.nodes[4 * node], q1 = a.nodes[4 * node + 1], q2 = a.nodes[4 * node + 2],
                         q3 = a.nodes[4 * node + 3];
            const float b0min[3] = {q0.x, q0.y, q0.z}, b0max[3] = {q0.w, q1.x, q1.y};
            const float b1min[3] = {q1.z, q1.w, q2.x}, b1max[3] = {q2.y, q2.z, q2.w};
            const uint32_t c0 = __float_as_uint(q3.x), c1 = __float_as_uint(q3.y);
            float t0, t1;
            bool h0 = slab_enter(b0min, b0max, sr, t0) && t0 <= best;
            bool h1 = slab_enter(b1min, b1max, sr, t1) && t1 <= best;
            // leaves right away (they may shrink `best` before the boxes are pushed)
            if (h0 && (c0 & GRAY_LEAF_BIT)) {
                if ((c0 & ~GRAY_LEAF_BIT) < (uint32_t)n) ellipsoid_leaf(a, c0 & ~GRAY_LEAF_BIT, ro, rd, znear, minop, best, bid);
                h0 = false;
            }
            if (h1 && (c1 & GRAY_LEAF_BIT)) {
                if ((c1 & ~GRAY_LEAF_BIT) < (uint32_t)n) ellipsoid_leaf(a, c1 & ~GRAY_LEAF_BIT, ro, rd, znear, minop, best, bid);
                h1 = false;
            }
            h0 = h0 && t0 <= best;
            h1 = h1 && t1 <= best;
            // far child deeper in the stack, near child on top
            const bool near1 = h0 && h1 && t1 < t0;
            const uint32_t first = near1 ? c0 : c1, second = near1 ? c1 : c0;
            const bool hf = near1 ? h0 : h1, hs = near1 ? h1 : h0;
            if (sp + (int)hf + (int)hs > kEllStack) {
                raise_status(a.status, GRAY_STATUS_STACK_OVERFLOW);
                break;
            }
            if (hf) stk[sp++] = first;
            if (hs) stk[sp++] = second;
        }
    }
    float r0 = a.bg[0], r1 = a.bg[1], r2 = a.bg[2], depth = 0.0f;
    if (bid != GRAY_NULL) {
        ellipsoid_shade(a.geom[3 * bid], a.geom[3 * bid + 1], a.geom[3 * bid + 2], ro, rd, best,
                        a.channels + 3 * (size_t)bid, r0, r1, r2);
        depth = best;
    }
    a.out_rgb[3 * pixel] = r0;
    a.out_rgb[3 * pixel + 1] = r1;
    a.out_rgb[3 * pixel + 2] = r2;
    a.out_depth[pixel] = depth;
}

// Grid-stride over 16x8-pixel tiles (a few blocks per SM): the launch made on every forward costs
// little when the view is off.
__global__ void __launch_bounds__(kEllTileX * kEllTileY) ellipsoid_kernel(const FwdArgs a, int tiles_x, int ntiles) {
    if (*a.render_ellipsoids)
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x)
            ellipsoid_pixel(a, (t % tiles_x) * kEllTileX + threadIdx.x, (t / tiles_x) * kEllTileY + threadIdx.y);
    grid_wait_before();
}

// ---------------------------------------------------------------------------------------------
// Batched render: many views (of one or several resident scenes) in one persistent launch.
// Blocks pull groups of 2x2 packets from a global counter (the groups of all views counted in order of
// the views; with frontiers, the densest first) and trace them as the plain forward's blocks trace a tile.  Forward only (no gradients, no
// hit lists); per view the output is RGB.  With a frontier buffer (group_offset numbers the groups
// in it), batch_frontier_kernel first writes each group's BVH frontier, and the traversals start there.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(32) batch_frontier_kernel(const gray_batch_scene *__restrict__ scenes,
                                                            const gray_batch_view *__restrict__ views, int nviews,
                                                            uint32_t *__restrict__ frontier, int tile_w,
                                                            uint32_t cut) {
    __shared__ FrontierScratch fs;
    const uint32_t group = blockIdx.x;
    const int lane = threadIdx.x;
    int v = 0;
    while (v + 1 < nviews && views[v + 1].group_offset <= group) v++;
    const gray_batch_view &vw = views[v];
    const gray_batch_scene &bs = scenes[vw.scene];
    uint32_t *out = frontier + (size_t)group * kFrontierWords;
    if (group == 0u && lane == 0) out[kBatchOrdered] = 0u;  // (batch_order_kernel's to set)
    const int tile_h = 32 / tile_w;
    const uint32_t tiles_x = (vw.width + tile_w - 1) / tile_w;
    const uint32_t gxn = (tiles_x + 1) / 2, local = group - vw.group_offset;
    const int x0 = (int)((local % gxn) * 2 * tile_w), y0 = (int)((local / gxn) * 2 * tile_h);
    if (bs.n <= 1 || x0 >= (int)vw.width || y0 >= (int)vw.height) {
        if (lane == 0) {
            out[0] = kFrontierNone;
            out[kBatchEst] = 0u;
        }
        return;
    }
    const int x1 = min(x0 + 2 * tile_w, (int)vw.width) - 1, y1 = min(y0 + 2 * tile_h, (int)vw.height) - 1;
    make_frustum_warp(fs.fr, mk3(vw.origin[0], vw.origin[1], vw.origin[2]), vw.w2c, vw.fov_y, x0, y0, x1, y1, vw.width,
                      vw.height, bs.root_box);
    const uint32_t est = frontier_walk<false>(reinterpret_cast<const float4 *>(bs.nodes), bs.n, cut, fs, nullptr, out,
                                              nullptr);
    if (lane == 0) out[kBatchEst] = est;
}

constexpr unsigned int kBatchOrderFrom = 4;  // groups per block from which the order is made

__device__ __forceinline__ uint32_t batch_groups_of(const gray_batch_view &v, int tile_w) {
    const uint32_t tile_h = 32u / tile_w;
    const uint32_t tx = (v.width + tile_w - 1) / tile_w, ty = (v.height + tile_h - 1) / tile_h;
    return ((tx + 1) / 2) * ((ty + 1) / 2);
}

// The batch's work order, one block: the groups of all views counting-sorted by log2 of their estimates,
// densest first, as the plain forward's tiles: in the views' order a dense group near the end was the
// launch's tail (two views of 3M Gaussians at up to 1920x1080 4.69 -> 3.31 ms, four of 1M at up to 1280x720
// 1.37 -> 0.99, sixteen of 3M 24.8 -> 24.6).  Views whose group_offset does not number their groups one after another get
// no order.
__global__ void __launch_bounds__(kOrderThreads) batch_order_kernel(const gray_batch_view *__restrict__ views,
                                                                    int nviews, uint32_t *__restrict__ frontier,
                                                                    uint32_t total_groups, int tile_w) {
    __shared__ uint32_t s_bucket[kOrderBuckets];
    __shared__ int s_ok;
    const int t = threadIdx.x, lane = t & 31;
    if (t < kOrderBuckets) s_bucket[t] = 0u;
    if (t == 0) {
        uint32_t g = 0u;
        bool ok = true;
        for (int v = 0; v < nviews; v++) {
            ok = ok && views[v].group_offset == g;
            g += batch_groups_of(views[v], tile_w);
        }
        s_ok = ok && g == total_groups ? 1 : 0;
        frontier[kBatchOrdered] = (uint32_t)s_ok;
    }
    __syncthreads();
    if (!s_ok) return;
    for (int pass = 0; pass < 2; pass++) {
        uint32_t ahead[kOrderAhead];
        uint32_t r = 0u;
        for (uint32_t i0 = 0; i0 < total_groups; i0 += kOrderThreads, r = (r + 1) % kOrderAhead) {
            const uint32_t i = i0 + t;
            if (r == 0u) {
#pragma unroll
                for (int j = 0; j < kOrderAhead; j++) {
                    const uint32_t k = i + j * kOrderThreads;
                    ahead[j] = k < total_groups ? frontier[(size_t)k * kFrontierWords + kBatchEst] : 0u;
                }
            }
            const uint32_t key = i < total_groups ? (uint32_t)__clz((int)ahead[0]) : (uint32_t)kOrderBuckets;
#pragma unroll
            for (int j = 0; j + 1 < kOrderAhead; j++) ahead[j] = ahead[j + 1];
            const uint32_t peers = __match_any_sync(kFull, key);
            const int lead = __ffs((int)peers) - 1;
            uint32_t base = 0u;
            if (lane == lead && i < total_groups) base = atomicAdd(&s_bucket[key], (uint32_t)__popc(peers));
            base = __shfl_sync(kFull, base, lead) + __popc(peers & ((1u << lane) - 1u));
            if (pass == 1 && i < total_groups) frontier[(size_t)base * kFrontierWords + kBatchOrder] = i;
        }
        __syncthreads();
        if (pass == 0 && t == 0) {
            uint32_t acc = 0u;
            for (int k = 0; k < kOrderBuckets; k++) {
                const uint32_t c = s_bucket[k];
                s_bucket[k] = acc;
                acc += c;
            }
        }
        __syncthreads();
    }
}

template <int KB, int MINB>
__global__ void __launch_bounds__(kFwdThreads, MINB)
    trace_batch_kernel(const gray_batch_scene *__restrict__ scenes, const gray_batch_view *__restrict__ views,
                       int nviews, uint32_t total_packets, float *__restrict__ out, uint32_t *__restrict__ counter,
                       int tile_w, const uint32_t *__restrict__ frontier, uint32_t total_groups,
                       int32_t *status) {
    __shared__ TileShared<KB, false> sh;
    // the group's scene and view parameters live in shared memory (read where used), which keeps
    // them out of the registers the traversal needs
    __shared__ TraceScene s_sc;
    __shared__ TraceKnobs s_k;
    __shared__ uint32_t s_view, s_local;  // view of the block's group, group inside the view
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile_h = 32 / tile_w;
    const float hx = (float)(tile_w * kBlockWarpsX - 1) * 0.5f, hy = (float)(tile_h * kBlockWarpsY - 1) * 0.5f;
    const bool ordered = frontier && total_groups > 0u && frontier[kBatchOrdered] != 0u;
    for (;;) {
        __syncthreads();  // every thread is done with the previous group
        if (threadIdx.x == 0) {
            uint32_t g = atomicAdd(counter, 1u);
            if (ordered && g < total_groups) g = frontier[(size_t)g * kFrontierWords + kBatchOrder];
            int v = 0;
            for (; v < nviews; v++) {
                const uint32_t groups = batch_groups_of(views[v], tile_w);
                if (g < groups) break;
                g -= groups;
            }
            s_view = (uint32_t)v;
            s_local = g;
            if (v < nviews) {
                const gray_batch_view &vw = views[v];
                const gray_batch_scene &bs = scenes[vw.scene];
                s_k.znear = vw.znear;
                s_k.zfar = vw.zfar;
                s_k.athr = bs.alpha_threshold;
                s_k.pw = bs.exp_power;
                s_k.tthr = bs.t_threshold;
                s_k.render_depth = false;
                s_sc = TraceScene{reinterpret_cast<const float4 *>(bs.geom), reinterpret_cast<const float4 *>(bs.l2w),
                                  reinterpret_cast<const float2 *>(bs.live), vw.channels,
                                  reinterpret_cast<const float4 *>(bs.nodes), bs.root_box, bs.n};
            }
        }
        __syncthreads();
        if (s_view >= (uint32_t)nviews) break;
        const gray_batch_view &vw = views[s_view];
        const TraceScene &sc = s_sc;
        const TraceKnobs &k = s_k;
        const uint32_t tiles_x = (vw.width + tile_w - 1) / tile_w, gxn = (tiles_x + 1) / 2;
        const uint32_t gx = s_local % gxn, gy = s_local / gxn;
        const uint32_t wx = 2 * gx + warp % kBlockWarpsX, wy = 2 * gy + warp / kBlockWarpsX;
        const int x0 = (int)(gx * 2 * tile_w), y0 = (int)(gy * 2 * tile_h);
        const int px = (int)(wx * tile_w) + lane % tile_w, py = (int)(wy * tile_h) + lane / tile_w;
        // (packets past the launch's total, and past the view's edges, render nothing)
        const bool inside = px < (int)vw.width && py < (int)vw.height &&
                            vw.packet_offset + wy * tiles_x + wx < total_packets;
        const f3 ro = mk3(vw.origin[0], vw.origin[1], vw.origin[2]);
        f3 rd = mk3(0.0f, 0.0f, 0.0f);
        if (inside) rd = camera_ray(vw.w2c, vw.fov_y, px, py, vw.width, vw.height, 0.0f, 0.0f);
        // (the loop of trace_rays starts with a block barrier)
        if (warp == 0)
            make_frustum_warp(sh.fr, ro, vw.w2c, vw.fov_y, x0, y0, x0 + 2 * tile_w - 1, y0 + 2 * tile_h - 1, vw.width,
                              vw.height, s_sc.root_box);
        if (threadIdx.x == kFwdThreads - 1)
            make_conic_basis(sh.cb, vw.w2c, vw.fov_y, (float)x0 + hx, (float)y0 + hy, hx, hy, vw.width, vw.height);
        // the group's frontier (a group beyond the launch's total starts at the root)
        const uint32_t grp = vw.group_offset + s_local;
        const uint32_t *front = frontier && grp < total_groups ? frontier + (size_t)grp * kFrontierWords : nullptr;
        RayResult r;
        trace_rays<KB, false>(sc, k, ro, rd, (float)(px - x0) - hx, (float)(py - y0) - hy, inside, true, false,
                              HitSink{nullptr, nullptr, 0}, status, sh, front, r);
        if (!inside) continue;
        float r0, r1, r2;
        finish_ray(r, scenes[vw.scene].bg, 1e-12f, false, r0, r1, r2);
        float *o = out + vw.out_offset + 3 * ((size_t)py * vw.width + px);
        o[0] = r.C0;
        o[1] = r.C1;
        o[2] = r.C2;
    }
}

static FwdArgs forward_args(const gray_params &p, bool display) {
    FwdArgs a;
    a.display = display ? 1 : 0;
    a.auto_role = 0;
    a.alloc_w = p.image_width;
    a.render_w = p.render_width;
    a.render_h = p.render_height;
    a.n = p.gaussians.count;
    a.cam_origin = p.camera.origin;
    a.fov = p.camera.vertical_fov_radians;
    a.w2c = p.camera.rotation_w2c;
    a.znear = p.camera.znear;
    a.zfar = p.camera.zfar;
    a.exp_power = p.config.exp_power;
    a.alpha_threshold = p.config.alpha_threshold;
    a.t_threshold = p.config.t_threshold;
    a.eps_fwd = p.config.eps_forward_normalization;
    a.bg = p.config.background_channels;
    a.render_depth = p.config.render_depth;
    a.needs_ray_output = p.config.needs_ray_output;
    a.rays_from_python = p.config.rays_from_python;
    a.jitter = p.config.jitter_primary_rays;
    a.grads_enabled = p.metadata.grads_enabled;
    a.total_num_calls = p.metadata.total_num_calls;
    a.geom = reinterpret_cast<const float4 *>(p.scene.geom);
    a.l2w = reinterpret_cast<const float4 *>(p.scene.l2w);
    a.live = reinterpret_cast<const float2 *>(p.scene.live);
    a.channels = p.gaussians.channels;
    a.nodes = reinterpret_cast<const float4 *>(p.scene.nodes);
    a.root_box = p.scene.root_box;
    a.out_rgb = p.framebuffer.output_channels;
    a.out_depth = p.framebuffer.output_depth;
    a.out_T = p.framebuffer.transmittance;
    a.out_fullT = p.framebuffer.full_transmittance;
    a.out_rem = p.framebuffer.remaining_channels_estimate;
    a.ray_o = p.framebuffer.ray_origin;
    a.ray_d = p.framebuffer.ray_direction;
    a.stat_hit = p.stats.num_gaussians_hit;
    a.stat_acc = p.stats.num_gaussians_accumulated;
    a.head = p.hitlist.head_per_pixel;
    a.counter = p.hitlist.total_words;
    a.pool = p.hitlist.pool;
    a.pool_size = p.hitlist.size;
    a.status = p.status;
    a.render_ellipsoids = p.config.render_ellipsoids;
    a.ellipsoid_min_opacity = p.config.ellipsoid_min_opacity;
    a.slots_split = 1;
    a.tile_w = 8;
    a.tile_h = 4;
    a.schedule = nullptr;
    a.frontier = nullptr;
    a.frontier_cut = 0;
    a.super_frontier = nullptr;
    a.super_x = 0;
    return a;
}

cudaError_t launch_ellipsoids(const gray_params &p, bool display, cudaStream_t s) {
    const FwdArgs a = forward_args(p, display);
    const int tiles_x = (int)((p.render_width + kEllTileX - 1) / kEllTileX);
    const int ntiles = tiles_x * (int)((p.render_height + kEllTileY - 1) / kEllTileY);
    if (ntiles <= 0) return cudaSuccess;
    int sms = 0, per_sm = 0;
    cudaError_t e;
    if ((e = resident_blocks(reinterpret_cast<const void *>(&ellipsoid_kernel), kEllTileX * kEllTileY, 0, &sms,
                             &per_sm)) != cudaSuccess)
        return e;
    // the last of the forward's programmatic launches: what it reads was there before the chain's first
    int tx = tiles_x, nt = ntiles;
    FwdArgs args_a = a;
    void *args[] = {&args_a, &tx, &nt};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ntiles < 8 * sms ? ntiles : 8 * sms);
    cfg.blockDim = dim3(kEllTileX, kEllTileY);
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, reinterpret_cast<const void *>(&ellipsoid_kernel), args);
}

// Launch shape of one forward: the kernel arguments, the trace kernel and its grid, and whether the
// tile schedule (work estimate, densest-first order, per-tile BVH frontier) is used.
struct FwdPlan {
    FwdArgs a;
    const void *kern;
    const void *kern_wide;  // automatic choice: the wide kernel, launched after `kern` (else null)
    dim3 grid;
    int bw, bh;
    bool sched, split;  // split: dense tiles may be traced as their four packets
    int nsuper;  // super-tiles whose coarse frontiers seed the tile walks (0: tiles walk from the root)
};

// The automatic choice's frontier cut.  Finer frontiers shorten the tiles' traversals and sharpen their
// estimates, and lengthen the tile walks, which take as long as the preparation beside them from about
// 2M Gaussians on.  Measured, display at cuts 16, 32 and 64 (us): 30k / 1280x720 228, 241, 248; 300k /
// 1920x1080 653, 670, 690; 500k / 640x480 326, 340, 384; 1M / 1920x1080 1030, 1042, 1066, 1M / 640x480 547,
// 476, 513; 2M / 1920x1080 1583, 1528, 1526; 3M / 1920x1080 2078, 1997, 1965; 6M / 4K 9233, 9107, 9008.
static uint32_t automatic_cut(int n) { return n <= 600000 ? 16u : n <= 1500000 ? 32u : (uint32_t)kFrontierCutDefault; }

static FwdPlan plan_forward(const gray_params &p, bool display) {
    FwdPlan q;
    q.nsuper = 0;
    FwdArgs &a = q.a;
    a = forward_args(p, display);
    // variant: bits 0-1 select (buffer size, register cap), bit 2 the packet shape, bits 3-4 the
    // tile frontier's cut (64 leaves, 32, 128, no frontier), bit 5 leaves dense tiles whole
    // variant 0 (the default) chooses between the narrow and the wide kernel of kDefaultTraceVariant's
    // packet shape, with automatic_cut's frontiers, from the last scheduled forward's re-traversals: the 16-slot hit buffer with
    // five blocks per SM (4, 5, 6: 3.08, 2.83, 2.91 ms on the benchmark's training view at 3M / 1080p; six leave
    // 80 registers, with twice the spills) is faster where few rays composite more than 16 hits, the 32-slot one with
    // four blocks where many do (a re-traversal repeats the packet's whole traversal)
    const bool automatic = p.trace_variant <= 0;
    const int v = p.trace_variant > 0 ? p.trace_variant : kDefaultTraceVariant;
    const int fcut = (v >> 3) & 3;
    q.split = (v & 32) == 0;
    q.kern_wide = nullptr;
    a.tile_w = (v & 4) ? 4 : 8;
    a.tile_h = 32 / a.tile_w;
    q.bw = a.tile_w * kBlockWarpsX;
    q.bh = a.tile_h * kBlockWarpsY;
    q.grid = dim3((p.render_width + q.bw - 1) / q.bw, (p.render_height + q.bh - 1) / q.bh);
    a.tiles_x = (int)q.grid.x;
    a.ntiles = (int)(q.grid.x * q.grid.y);
    a.schedule = nullptr;
    const size_t words = gray_schedule_words_for(p.image_width, p.image_height);
    q.sched = p.hitlist.schedule && a.ntiles > 0 &&
              (size_t)a.ntiles <= (words - kSchedHeader) / (1 + kOrderPerTile);
#define GRAY_FWD_KERNEL(KB, MINB)                                                                   \
    (!q.sched ? reinterpret_cast<const void *>(&trace_forward_kernel<KB, MINB>)                     \
              : reinterpret_cast<const void *>(&trace_forward_sched_kernel<KB, MINB>))
    switch (v & 3) {
        case 0: q.kern = GRAY_FWD_KERNEL(32, 3); break;
        case 1: q.kern = GRAY_FWD_KERNEL(32, 4); break;
        case 2: q.kern = GRAY_FWD_KERNEL(16, 3); break;
        default: q.kern = GRAY_FWD_KERNEL(16, 5); break;
    }
#undef GRAY_FWD_KERNEL
    if (q.sched) {
        a.schedule = p.hitlist.schedule;
        if (automatic) {
            q.kern = reinterpret_cast<const void *>(&trace_forward_sched_kernel<16, 5>);
            q.kern_wide = reinterpret_cast<const void *>(&trace_forward_sched_kernel<32, 4>);
        }
        a.frontier_cut = automatic   ? automatic_cut(a.n)
                         : fcut == 0 ? kFrontierCutDefault
                         : fcut == 1 ? 32u
                         : fcut == 2 ? 128u
                                     : 0u;
        if (a.frontier_cut > 0 && (size_t)a.ntiles <= (words - kSchedHeader) / (1 + kOrderPerTile + kFrontierWords))
            a.frontier = a.schedule + kSchedHeader + (1 + kOrderPerTile) * (size_t)a.ntiles;
        if (a.frontier) {
            // super-tiles after the tiles' frontiers, when the buffer holds them
            const int sx = (a.tiles_x + kSuperTiles - 1) / kSuperTiles;
            const int sy = ((int)q.grid.y + kSuperTiles - 1) / kSuperTiles;
            const size_t used =
                (size_t)kSchedHeader + (size_t)(1 + kOrderPerTile + kFrontierWords) * (size_t)a.ntiles;
            // (in a small tree they leave the tiles' walks two levels to save, and are a launch more)
            if (a.n > (int)(4 * kSuperCut) && used + (size_t)sx * (size_t)sy * kSuperWords <= words) {
                a.super_frontier = a.frontier + (size_t)a.ntiles * kFrontierWords;
                a.super_x = sx;
                q.nsuper = sx * sy;
            }
        }
    }
    return q;
}

bool trace_forward_has_schedule(const gray_params &p) { return plan_forward(p, false).sched; }

cudaError_t launch_trace_schedule(const gray_params &p, bool display, cudaStream_t s) {
    const FwdPlan q = plan_forward(p, display);
    if (!q.sched) return cudaSuccess;
    // densest tiles first: per-tile estimate and frontier, then the work order
    FwdArgs a = q.a;
    const void *kerns[3] = {q.kern, q.kern_wide ? q.kern_wide : q.kern,
                            reinterpret_cast<const void *>(&trace_forward_split_kernel<16, kSplitBlocks>)};
    int slots[3] = {0, 0, 0};
    for (int i = 0; i < 3; i++) {
        int sms = 0, per_sm = 0;
        const cudaError_t e = resident_blocks(kerns[i], kFwdThreads, 0, &sms, &per_sm);
        if (e != cudaSuccess) return e;
        slots[i] = sms * per_sm;
    }
    a.slots_split = slots[2];
    if (q.nsuper > 0) super_cost_kernel<<<q.nsuper, 32, 0, s>>>(a, q.bw, q.bh, q.nsuper);
    tile_cost_kernel<<<a.ntiles, 32, 0, s>>>(a, q.bw, q.bh);
    sched_order_kernel<<<1, kOrderThreads, 0, s>>>(a.schedule, a.ntiles, slots[0], slots[1], slots[2],
                                                   q.split ? 0 : 1, a.rays_from_python);
    return cudaGetLastError();
}

cudaError_t launch_trace_forward(const gray_params &p, bool display, bool schedule_ready, cudaStream_t s) {
    FwdPlan q = plan_forward(p, display);
    cudaError_t e;
    if (!q.sched) {
        void *args[] = {&q.a};
        if ((e = cudaLaunchKernel(q.kern, q.grid, dim3(kFwdThreads), args, 0, s)) != cudaSuccess) return e;
        return cudaGetLastError();
    }
    if (!schedule_ready && (e = launch_trace_schedule(p, display, s)) != cudaSuccess) return e;
    // persistent grids that take the split tiles' packets, the whole tiles in the schedule's order and the single
    // rays' packets; with the automatic choice both kernels of the whole tiles are launched and the one not
    // chosen returns at once.  All but the chain's first are programmatic: they run beside the one before.
    const void *kerns[4] = {reinterpret_cast<const void *>(&trace_forward_split_kernel<16, kSplitBlocks>), q.kern,
                            q.kern_wide,
                            reinterpret_cast<const void *>(&trace_forward_rays_kernel<kRaySlots, kRayBlocks>)};
    const int roles[4] = {0, q.kern_wide ? (int)kChoiceNarrow : 0, (int)kChoiceWide, 0};
    for (int i = 0; i < 4; i++) {
        if (!kerns[i]) continue;
        int sms = 0, per_sm = 0;
        if ((e = resident_blocks(kerns[i], kFwdThreads, 0, &sms, &per_sm)) != cudaSuccess) return e;
        const unsigned int want = (unsigned int)(sms * per_sm);
        const unsigned int items = (i == 0 ? 4u : 1u) * (unsigned int)q.a.ntiles;  // at most
        FwdArgs a = q.a;
        a.auto_role = roles[i];
        void *args[] = {&a};
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(want < items ? want : items, 1, 1);
        cfg.blockDim = dim3(kFwdThreads);
        cfg.stream = s;
        cfg.attrs = &attr;
        cfg.numAttrs = i > 0 ? 1 : 0;
        if ((e = cudaLaunchKernelExC(&cfg, kerns[i], args)) != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

size_t gray_schedule_words_for(uint32_t width, uint32_t height) {
    // estimates and order for any tile shape (tiles of at least 8x8 pixels), frontiers for tiles
    // of 8x16 or 16x8 pixels (the forward's block tiles)
    const size_t t8 = (size_t)((width + 7) / 8) * (size_t)((height + 7) / 8);
    const size_t ta = (size_t)((width + 7) / 8) * (size_t)((height + 15) / 16);
    const size_t tb = (size_t)((width + 15) / 16) * (size_t)((height + 7) / 8);
    // and the coarse frontiers of their super-tiles (kSuperTiles x kSuperTiles tiles)
    const size_t k = kSuperTiles;
    const size_t sa = (((width + 7) / 8 + k - 1) / k) * (((height + 15) / 16 + k - 1) / k);
    const size_t sb = (((width + 15) / 16 + k - 1) / k) * (((height + 7) / 8 + k - 1) / k);
    return (size_t)kSchedHeader + 2 * t8 + (ta > tb ? ta : tb) * (kOrderPerTile - 1 + kFrontierWords) +
           (sa > sb ? sa : sb) * kSuperWords;
}

cudaError_t launch_trace_batch(const gray_batch_scene *scenes, const gray_batch_view *views, int nviews,
                               uint32_t total_packets, float *out, uint32_t *counter, uint32_t *frontier,
                               uint32_t total_groups, int variant, int blocks_per_sm, int32_t *status,
                               cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const int v = variant > 0 ? variant : kDefaultTraceVariant;
    const int tile_w = (v & 4) ? 4 : 8;
    const int fcut = (v >> 3) & 3;
    const uint32_t cut = fcut == 0 ? kFrontierCutDefault : fcut == 1 ? 32u : fcut == 2 ? 128u : 0u;
    const unsigned int grid = (unsigned int)(sms * (blocks_per_sm > 0 ? blocks_per_sm : 4));
    if ((e = cudaMemsetAsync(counter, 0, sizeof(uint32_t), s)) != cudaSuccess) return e;
    if (!frontier || cut == 0 || total_groups == 0) {
        frontier = nullptr;
    } else {
        batch_frontier_kernel<<<total_groups, 32, 0, s>>>(scenes, views, nviews, frontier, tile_w, cut);
        // (with a few groups per block the order gains less than its launch takes: 3 views of 320x240 over 50k
        // Gaussians, 1800 groups, 167 us without and 178 with)
        if (total_groups > kBatchOrderFrom * grid)
            batch_order_kernel<<<1, kOrderThreads, 0, s>>>(views, nviews, frontier, total_groups, tile_w);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    const uint32_t *fr = frontier;
    switch (v & 3) {
        case 0: trace_batch_kernel<32, 1><<<grid, kFwdThreads, 0, s>>>(scenes, views, nviews, total_packets, out, counter, tile_w, fr, total_groups, status); break;
        case 1: trace_batch_kernel<32, 4><<<grid, kFwdThreads, 0, s>>>(scenes, views, nviews, total_packets, out, counter, tile_w, fr, total_groups, status); break;
        case 2: trace_batch_kernel<16, 1><<<grid, kFwdThreads, 0, s>>>(scenes, views, nviews, total_packets, out, counter, tile_w, fr, total_groups, status); break;
        default: trace_batch_kernel<16, 6><<<grid, kFwdThreads, 0, s>>>(scenes, views, nviews, total_packets, out, counter, tile_w, fr, total_groups, status); break;
    }
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------------------------
struct BwdArgs {
    uint32_t alloc_w, render_w, render_h;
    int n;
    const float *exp_power, *bg;
    const float4 *geom;
    const float2 *live;
    const float *channels;
    const float *pix_T, *pix_fullT, *pix_rem, *ray_o, *ray_d, *grad_out;
    const uint32_t *head, *pool;
    uint32_t pool_size;
    float *grad_acc;
    int32_t *status;
};

__device__ __forceinline__ void red_add4(float *addr, float x, float y, float z, float w) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(x), "f"(y), "f"(z), "f"(w));
}

// Adds one hit's 14 gradient sums, and its count, to the Gaussian's accumulator row.  Neighbouring pixels
// composite the same Gaussians at the same replay step (on the benchmark scene a warp's lanes form
// groups of 16 on average, often the whole warp), and vector reductions on one row serialise in L2,
// so the lanes that hold the same Gaussian first combine their values and the lowest of them issues
// the four reductions.  The combination is a tree over the group's ranks: every lane knows the next
// member of its group (`nxt`, the member `s` ranks further after the round of stride s, found by
// pointer jumping), and in the round of stride s the members whose rank is a multiple of 2s add
// the partial sum of the member s ranks further; after ceil(log2(largest group)) rounds the lowest
// member holds the group's sum (14 shuffles per round; the count is the group's size).
constexpr int kHitSums = 14;

__device__ __forceinline__ void reduce_hit(float *row, uint32_t gid, float (&v)[kHitSums]) {
    const unsigned active = __activemask();
    const unsigned grp = __match_any_sync(active, gid);
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const int rank = __popc(grp & below);
    const int gmax = (int)__reduce_max_sync(active, (unsigned)__popc(grp));
    const unsigned above = grp & ~below & ~(1u << lane);
    int nxt = above ? __ffs(above) - 1 : -1;  // the member one rank further, -1: none
    for (int s = 1; s < gmax; s <<= 1) {
        const int src = nxt >= 0 ? nxt : lane;
        const bool take = nxt >= 0 && (rank & (2 * s - 1)) == 0;
#pragma unroll
        for (int k = 0; k < kHitSums; k++) {
            const float t = __shfl_sync(active, v[k], src);
            if (take) v[k] += t;
        }
        const int jump = __shfl_sync(active, nxt, src);
        nxt = nxt >= 0 ? jump : -1;
    }
    if (rank == 0) {
        red_add4(row, v[0], v[1], v[2], v[3]);
        red_add4(row + 4, v[4], v[5], v[6], v[7]);
        red_add4(row + 8, v[8], v[9], v[10], 0.0f);
        red_add4(row + 12, v[11], v[12], v[13], (float)__popc(grp));
    }
}

// What one composited hit reads: the snapshot rows, the live opacity and scaling factor, the colour.
struct BwdHit {
    float4 g0, g1, g2;
    float2 live;
    float c0, c1, c2;
};

__device__ __forceinline__ void load_hit(const BwdArgs &a, uint32_t gid, BwdHit &h) {
    const float4 *gp = a.geom + 3 * (size_t)gid;
    const float *cp = a.channels + 3 * (size_t)gid;
    h.g0 = __ldg(gp);
    h.g1 = __ldg(gp + 1);
    h.g2 = __ldg(gp + 2);
    h.live = __ldg(a.live + gid);
    h.c0 = __ldg(cp);
    h.c1 = __ldg(cp + 1);
    h.c2 = __ldg(cp + 2);
}

// Reverse-order walk of a pixel's segment chain (newest segment first, each segment back to front).
struct HitCursor {
    uint32_t seg, prev;
    int e, guard;
};

// Next composited gaussian id; false at the end of the list or on a corrupt list (status raised).
__device__ __forceinline__ bool next_gid(const BwdArgs &a, HitCursor &c, uint32_t &gid) {
    for (;;) {
        while (c.e >= 0) {
            gid = a.pool[c.seg + 2u + (uint32_t)c.e];
            c.e--;
            if (gid < (uint32_t)a.n) return true;
        }
        if (c.prev == GRAY_NULL) return false;
        c.seg = c.prev;
        if (c.seg + 2u > a.pool_size || ++c.guard > kPassSlots * kMaxPasses + 1) {
            raise_status(a.status, GRAY_STATUS_HITLIST_OVERFLOW);
            return false;
        }
        c.prev = a.pool[c.seg];
        const uint32_t cnt = a.pool[c.seg + 1];
        if (cnt > a.pool_size - c.seg - 2u) {
            raise_status(a.status, GRAY_STATUS_HITLIST_OVERFLOW);
            return false;
        }
        c.e = (int)cnt - 1;
    }
}

// Pixel-constant inputs of the replay.
struct BwdPixel {
    f3 ro, rd, gout;
    float Tfin, fT, dbg, drem, inv_npix, pw;
};

// One step of the reverse replay (cuda/backward_pass.cu:17-137) for hit h; T and gT are the
// running transmittance and colour-gradient tail.
//
// With x the hit's scaled object-space point and q = d loss / d x (up to sign), the gradients of mean,
// scale and rotation are linear in q and in q x^T, with coefficients of the Gaussian alone, and q is
// parallel to x.  So a hit adds q (3 sums) and the symmetric q x^T (6), and the pass over the Gaussians that
// follows applies the coefficients once per Gaussian instead of once per hit.  A hit that carried them
// to the parameters itself needed a record of 24 floats per Gaussian, written by a pass of its own over all
// Gaussians.  Accumulator row: [q | opacity] [xx xy xz yy] [yz zz, pruning weight, 0] [channels | count].
// Train step at 3M / 1080p 4.15 -> 3.98 ms, at 1M / 1600x1040 1.99 -> 1.89 ms, 301k / 799x533 0.66 -> 0.64 ms.
// 54 registers instead of 72; bound by instruction issue and the reductions; fetching the next hit's id ahead changed nothing.
__device__ __forceinline__ void replay_hit(const BwdArgs &a, const BwdPixel &px, uint32_t gid, const BwdHit &h,
                                           float &T, float &gT) {
    const float o = h.live.x, sf = h.live.y;
    const f3 c = mk3(h.c0, h.c1, h.c2);
    LocalHit lh;
    local_ray(h.g0, h.g1, h.g2, px.ro, px.rd, lh);
    closest_point(lh);
    const f3 x = mk3(lh.u.x * sf, lh.u.y * sf, lh.u.z * sf);
    const float sq = fdot3(x, x);
    const float gv = eval_gaussian(sq, px.pw);
    const float alpha = maxalpha_mul(gv, o);

    // one reciprocal of (1 - alpha) instead of four divisions (the reference divides each time,
    // cuda/backward_pass.cu:51-59,141); the gradients differ from it by rounding only
    const float om = 1.0f - alpha;
    const float rom = 1.0f / om;
    const float Tr = T * rom;
    const float w = Tr * alpha;
    const float dgc = dot3(px.gout, c);
    float ga = (dgc - gT) * Tr;
    ga = ga + -(px.fT * rom) * px.dbg;
    ga = ga + -((px.Tfin - px.fT) * rom) * px.drem;
    gT = gT + (dgc - gT) * alpha;
    const float ggv = maxalpha_mul(ga, o);
    float gsq;
    if (px.pw == 1.0f) gsq = gv;
    else if (px.pw == 2.0f) gsq = gv * sq;
    else if (px.pw == 3.0f) gsq = gv * sq * sq;
    else gsq = gv * gpow(sq, px.pw - 1.0f);
    const f3 q = mk3(x.x * gsq * ggv, x.y * gsq * ggv, x.z * gsq * ggv);
    float v[kHitSums] = {q.x,       q.y,       q.z,       maxalpha_mul(ga, gv), q.x * x.x,       q.x * x.y,
                         q.x * x.z, q.y * x.y, q.y * x.z, q.z * x.z,            w * px.inv_npix, px.gout.x * w,
                         px.gout.y * w, px.gout.z * w};
    reduce_hit(a.grad_acc + 16 * (size_t)gid, gid, v);
    T = Tr;
}

// One thread per pixel walks its composited hits back to front (16x8-pixel blocks of four 8x4-pixel
// warps: neighbouring pixels composite the same Gaussians, which the lanes combine cheaply).
__global__ void __launch_bounds__(128) trace_backward_kernel(const BwdArgs a) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    const int px = blockIdx.x * 16 + (w & 1) * 8 + (l & 7);
    const int py = blockIdx.y * 8 + (w >> 1) * 4 + (l >> 3);
    if (px >= (int)a.render_w || py >= (int)a.render_h) return;
    const uint32_t pixel = (uint32_t)py * a.alloc_w + (uint32_t)px;
    HitCursor cur;
    cur.seg = a.head[pixel];
    if (cur.seg == GRAY_NULL) return;
    if (cur.seg + 2u > a.pool_size) {
        raise_status(a.status, GRAY_STATUS_HITLIST_OVERFLOW);
        return;
    }
    cur.prev = a.pool[cur.seg];
    {
        const uint32_t cnt = a.pool[cur.seg + 1];
        if (cnt > a.pool_size - cur.seg - 2u) {
            raise_status(a.status, GRAY_STATUS_HITLIST_OVERFLOW);
            return;
        }
        cur.e = (int)cnt - 1;
    }
    cur.guard = 1;
    BwdPixel P;
    P.pw = *a.exp_power;
    P.Tfin = a.pix_T[pixel];
    P.fT = a.pix_fullT[pixel];
    const f3 rem = mk3(a.pix_rem[3 * pixel], a.pix_rem[3 * pixel + 1], a.pix_rem[3 * pixel + 2]);
    P.ro = mk3(a.ray_o[3 * pixel], a.ray_o[3 * pixel + 1], a.ray_o[3 * pixel + 2]);
    P.rd = mk3(a.ray_d[3 * pixel], a.ray_d[3 * pixel + 1], a.ray_d[3 * pixel + 2]);
    P.gout = mk3(a.grad_out[3 * pixel], a.grad_out[3 * pixel + 1], a.grad_out[3 * pixel + 2]);
    const f3 bg = mk3(a.bg[0], a.bg[1], a.bg[2]);
    P.dbg = dot3(bg, P.gout);
    P.drem = dot3(rem, P.gout);
    P.inv_npix = 1.0f / (float)(a.render_w * a.render_h);
    float gT = 0.0f, T = P.Tfin;
    uint32_t gid;
    if (!next_gid(a, cur, gid)) return;
    do {
        BwdHit h;
        load_hit(a, gid, h);
        replay_hit(a, P, gid, h, T, gT);
    } while (next_gid(a, cur, gid));
}

cudaError_t launch_trace_backward(const gray_params &p, cudaStream_t s) {
    const int n = p.gaussians.count;
    BwdArgs a;
    a.alloc_w = p.image_width;
    a.render_w = p.render_width;
    a.render_h = p.render_height;
    a.n = n;
    a.exp_power = p.config.exp_power;
    a.bg = p.config.background_channels;
    a.geom = reinterpret_cast<const float4 *>(p.scene.geom);
    a.live = reinterpret_cast<const float2 *>(p.scene.live);
    a.channels = p.gaussians.channels;
    a.pix_T = p.framebuffer.transmittance;
    a.pix_fullT = p.framebuffer.full_transmittance;
    a.pix_rem = p.framebuffer.remaining_channels_estimate;
    a.ray_o = p.framebuffer.ray_origin;
    a.ray_d = p.framebuffer.ray_direction;
    a.grad_out = p.framebuffer.grad_output_channels;
    a.head = p.hitlist.head_per_pixel;
    a.pool = p.hitlist.pool;
    a.pool_size = p.hitlist.size;
    a.grad_acc = p.scene.grad_acc;
    a.status = p.status;
    dim3 grid((p.render_width + 15) / 16, (p.render_height + 7) / 8);
    trace_backward_kernel<<<grid, 128, 0, s>>>(a);
    return cudaGetLastError();
}

}  // namespace gray
