// Photoelectric system-matrix kernel for sm_100a.
//
// Computes A[d][v] = sum over the 8x16x8 sub-elements s of crystal d of
//   Omega_s * exp(-sum mu L) * (1 - exp(-mu_d L_abs,s)) * mu_pe,d / mu_d
// as the reference kernel photodetectorCudaMe defines it
// (PEGen_RayTracing_CircularHole/PESysMatGen.cu:951-1364), with a different execution plan:
//
//  * a block owns one crystal d and a brick of voxels: up to 16 in a launch of its own
//    (choose_bricks), what the plan says in a batched one (4 x 4 x 2 unless set or tuned, 512 at
//    most), 4 x 4 x 2 in a projection; work items are handed out by an atomic counter over a
//    persistent grid; one warp per matrix element;
//  * the block builds a conservative superset of the reference's cone test (:1105-1186) for
//    every voxel of the brick, from the brick's centre and radius, in the reference's object
//    order.  Each warp keeps the objects of its element that pass the reference cone test and
//    whose direction-slope rectangle (dx/dy, dz/dy seen from the voxel) overlaps the one of
//    crystal d, and 32 rays at a time take those that can meet their slopes.  A skipped object
//    has an exactly-zero chord in the reference, and adding 0 or fma(mu, 0, x) leaves a float
//    unchanged, so no filter changes any float result;
//  * the plate-bypass penalty (:1240-1254) is skipped for rays whose slope lies inside the
//    plate's "through both faces" rectangle, where the chord is >= T >= 0.2 mm;
//  * sub-elements whose plate penalty fired contribute exp(-(>=1e5)) = 0 and stop early
//    (only when every attenuation coefficient is non-negative).
//
// The element itself: pe_ref.cuh for the float modes SYSMAT_MODE_REFERENCE (one float chain in
// the reference's sub-element order, its atomicAdd sequence at :1359) and SYSMAT_MODE_PRECISE
// (the same contributions summed in FP64); pe_fp64.cuh (SYSMAT_MODE_FP64: the element program
// in double, culling in float); pe_local.cuh (SYSMAT_MODE_LOCAL); pe_element_sampled (crystal
// divisions and voxel source points as parameters); pe_adjoint.cuh (projections, gradient).
#include <type_traits>

#include "chord64.cuh"
#include "geom.cuh"
#include "pe.cuh"
#include "rounding.cuh"

namespace sysmat {

namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kSuperCap = 1024;         // block superset capacity (objects)
constexpr float kSlopeMargin = 2e-4f;   // slope units; >> FP32 position error / depth
constexpr float kMinDepth = 1.0f;       // mm; slope rectangles need objects this far behind

// Per-element constants shared by the lanes of a warp.
struct Elem {
    float xI, yI, zI;            // voxel centre (rotated)
    float xIs, yIs, zIs;         // voxel in crystal d's frame
    float xd, yd, zd, w, t, h;   // crystal d
    float cosr, sinr;
    float mu_t, mu_pe, imu_t;    // and RN(1 / mu_t)
    float ux, uy, uz, crit_self; // reference cone test (:1110-1116)
    float4 rd;                   // slope rectangle of crystal d
    bool filt;
};

// The objects that may pass the cone test for some voxel of a block's brick, in the reference's
// order, and the block's work item.
struct Superset {
    unsigned short sid[kSuperCap];       // holes, then n_holes + crystal (at most 8877 + 6666 ids)
    int warp_cnt[kWarps];
    int s_count;                         // superset size; -1 = superset overflowed, use all
    long long item;
    unsigned short slot[512];            // the brick's voxels that belong to the block
};

__device__ __forceinline__ bool in_rect(const float4& r, float a, float b)
{
    return a >= r.x && a <= r.y && b >= r.z && b <= r.w;
}

__device__ __forceinline__ bool rects_overlap(const float4& p, const float4& q)
{
    return p.x <= q.y && q.x <= p.y && p.z <= q.w && q.z <= p.w;
}

__device__ __forceinline__ float4 open_rect()
{
    return make_float4(-INFINITY, INFINITY, -INFINITY, INFINITY);
}

// Slope rectangle of a crystal box seen from (px, py, pz), widened by the margin; the open
// rectangle if any corner is closer than kMinDepth in y.
__device__ float4 crystal_rect(float4 pos, float4 size, float4 trig, float px, float py, float pz)
{
    const float hw = 0.5f * size.x, ht = 0.5f * size.y, hh = 0.5f * size.z;
    const float y0 = pos.y - ht - py, y1 = pos.y + ht - py;
    if (!(y0 >= kMinDepth)) return open_rect();
    const float r0 = 1.0f / y0, r1 = 1.0f / y1;
    float amin = INFINITY, amax = -INFINITY, bmin = INFINITY, bmax = -INFINITY;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float xs = (c & 1) ? hw : -hw;
        const float zs = (c & 2) ? hh : -hh;
        const float x = pos.x + (xs * trig.x - zs * trig.y) - px;
        const float z = pos.z + (xs * trig.y + zs * trig.x) - pz;
        amin = fminf(amin, fminf(x * r0, x * r1));
        amax = fmaxf(amax, fmaxf(x * r0, x * r1));
        bmin = fminf(bmin, fminf(z * r0, z * r1));
        bmax = fmaxf(bmax, fmaxf(z * r0, z * r1));
    }
    return make_float4(amin - kSlopeMargin, amax + kSlopeMargin, bmin - kSlopeMargin,
                       bmax + kSlopeMargin);
}

__device__ float4 hole_rect(float4 ha, float r, float px, float py, float pz)
{
    const float y0 = ha.y - py, y1 = ha.z - py;
    if (!(y0 >= kMinDepth) || !(y1 >= kMinDepth)) return open_rect();
    const float r0 = 1.0f / y0, r1 = 1.0f / y1;
    const float xa = ha.x - r - px, xb = ha.x + r - px;
    const float za = ha.w - r - pz, zb = ha.w + r - pz;
    const float amin = fminf(fminf(xa * r0, xa * r1), fminf(xb * r0, xb * r1));
    const float amax = fmaxf(fmaxf(xa * r0, xa * r1), fmaxf(xb * r0, xb * r1));
    const float bmin = fminf(fminf(za * r0, za * r1), fminf(zb * r0, zb * r1));
    const float bmax = fmaxf(fmaxf(za * r0, za * r1), fmaxf(zb * r0, zb * r1));
    return make_float4(amin - kSlopeMargin, amax + kSlopeMargin, bmin - kSlopeMargin,
                       bmax + kSlopeMargin);
}

// Object i in the reference's order: holes 0..H-1 (layer by layer), then crystals.
__device__ __forceinline__ float4 object_data(const DevGeom& g, int i)
{
    if (i < g.n_holes) {
        const float4 a = __ldg(&g.hole.a[i]);
        const float4 b = __ldg(&g.hole.b[i]);
        return make_float4(a.x, b.z, a.w, b.w);
    }
    const float4 p = __ldg(&g.cry.pos[i - g.n_holes]);
    return make_float4(p.x, p.y, p.z, __ldg(&g.cry.size[i - g.n_holes].w));
}

__device__ __forceinline__ int layer_of_hole(const DevGeom& g, int h)
{
    int m = 0;
    while (m + 1 < g.n_layers && h >= g.layer[m + 1].hole_begin) ++m;
    return m;
}

// box_chord of the segment voxel -> sub-element through a plate, out of line: few rays need it.  Its
// length decides whether a ray counts at all, so the fused products are written out; they are those of the
// one-loop kernels, and not the ones of the crystal chord (norm2 with the depth first).
static __device__ __noinline__ float plate_chord(float xi, float yi, float zi, float xo, float yo, float zo,
                                                 float x1, float y1, float z1, float x2, float y2, float z2)
{
    const float dx = xo - xi, dy = yo - yi, dz = zo - zi;
    if (fabsf(dx) < kEps || fabsf(dy) < kEps || fabsf(dz) < kEps)
        return box_chord_parallel(xi, yi, zi, xo, yo, zo, x1, y1, z1, x2, y2, z2, 0);
    const float tio = sqrtf(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx))));
    float tmin, tmax, a0, a1;
    slab_interval(xi, x1, x2, tio / dx, tmin, tmax);
    slab_interval(yi, y1, y2, tio / dy, a0, a1);
    if (tmin > a1 || a0 > tmax) return 0.0f;
    tmin = (a0 > tmin) ? a0 : tmin;
    tmax = (a1 < tmax) ? a1 : tmax;
    slab_interval(zi, z1, z2, tio / dz, a0, a1);
    if (tmin > a1 || a0 > tmax) return 0.0f;
    tmin = (a0 > tmin) ? a0 : tmin;
    tmax = (a1 < tmax) ? a1 : tmax;
    const float len = __fsub_rn(tmax, tmin);
    if (len < kEps) return 0.0f;
    if (tmin >= tio || tmax >= tio) return 0.0f;
    if (tmin <= kEps || tmax <= kEps) return 0.0f;
    return len;
}

// Plate penalty (:1240-1254); true if any layer fired.
__device__ __forceinline__ bool plate_penalty(const DevGeom& g, const float4* plate_inner, const Elem& e, float xD,
                                              float yD, float zD, float sa_a, float sa_b, float& att)
{
    bool blocked = false;
    for (int m = 0; m < g.n_layers; ++m) {
        if (in_rect(plate_inner[m], sa_a, sa_b)) continue;
        const LayerInfo& L = g.layer[m];
        const float tl = plate_chord(e.xI, e.yI, e.zI, xD, yD, zD, L.x1, L.y1, L.z1, L.x2, L.y2, L.z2);
        if (tl < 0.1f) { att = att + 100000.0f; blocked = true; }
    }
    return blocked;
}

// Per-element set-up shared by the lanes of a warp: voxel centre, crystal d, reference cone
// constants, slope rectangle and the plate "through both faces" rectangles.  False when the
// crystal's attenuation is too low for the reference to compute the element (it is 0).
__device__ __forceinline__ bool init_element(const DevGeom& g, float4* plate_inner, int d, long long v, float cr,
                                             float sr, int lane, Elem& e, float fx = 0.5f, float fy = 0.5f,
                                             float fz = 0.5f)
{
    voxel_centre(g, v, cr, sr, e.xI, e.yI, e.zI, fx, fy, fz);   // the source point in the voxel
    const float4 P = __ldg(&g.cry.pos[d]);
    const float4 S = __ldg(&g.cry.size[d]);
    const float4 M = __ldg(&g.cry.mu[d]);
    const float4 T = __ldg(&g.cry.trig[d]);
    e.xd = P.x; e.yd = P.y; e.zd = P.z;
    e.w = S.x; e.t = S.y; e.h = S.z;
    e.mu_t = M.x; e.mu_pe = M.y;
    e.cosr = T.x; e.sinr = T.y;
    if (!(e.mu_t > 0.01f)) return false;                   // :1107, :1194
    e.imu_t = rcp_rn(e.mu_t);
    const float vx = e.xI - e.xd, vz = e.zI - e.zd;        // :1066-1068, to_crystal_frame
    e.xIs = __fmaf_rn(vx, T.z, -__fmul_rn(vz, T.w));
    e.yIs = e.yI - e.yd;
    e.zIs = __fmaf_rn(vx, T.w, __fmul_rn(vz, T.z));
    const float dist = sqrtf((e.yd - e.yI) * (e.yd - e.yI) + (e.xd - e.xI) * (e.xd - e.xI) +
                             (e.zd - e.zI) * (e.zd - e.zI));
    e.crit_self = S.w / dist / 2.0f;
    e.ux = (e.xd - e.xI) / dist;
    e.uy = (e.yd - e.yI) / dist;
    e.uz = (e.zd - e.zI) / dist;
    e.rd = crystal_rect(P, S, T, e.xI, e.yI, e.zI);
    e.filt = isfinite(e.rd.x);

    if (lane < g.n_layers) {          // plate "through both faces" rectangles
        const LayerInfo& Ly = g.layer[lane];
        float4 inner = make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);   // empty
        const float f0 = Ly.y1 - e.yI, f1 = Ly.y2 - e.yI;
        const float behind = e.yd - 0.5f * e.t - Ly.y2;
        if (e.filt && f0 >= kMinDepth && behind >= kMinDepth && (Ly.y2 - Ly.y1) >= 0.2f) {
            const float r0 = 1.0f / f0, r1 = 1.0f / f1;
            inner.x = fmaxf((Ly.x1 - e.xI) * r0, (Ly.x1 - e.xI) * r1) + kSlopeMargin;
            inner.y = fminf((Ly.x2 - e.xI) * r0, (Ly.x2 - e.xI) * r1) - kSlopeMargin;
            inner.z = fmaxf((Ly.z1 - e.zI) * r0, (Ly.z1 - e.zI) * r1) + kSlopeMargin;
            inner.w = fminf((Ly.z2 - e.zI) * r0, (Ly.z2 - e.zI) * r1) - kSlopeMargin;
        }
        plate_inner[lane] = inner;
    }

    return true;
}

#include "pe_ref.cuh"

#include "pe_fp64.cuh"
#include "pe_local.cuh"

// Appends `value` of the threads with `in`, in thread order, to list[n ..] (capacity cap) and returns
// how many there were.  All threads of the block call it.
__device__ __forceinline__ int block_append(Superset& bs, bool in, unsigned short value, unsigned short* list, int n,
                                            int cap, int lane, int wid)
{
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (lane == 0) bs.warp_cnt[wid] = __popc(m);
    __syncthreads();
    int off = n, tot = 0;
    for (int k = 0; k < kWarps; ++k) {
        const int c = bs.warp_cnt[k];
        if (k < wid) off += c;
        tot += c;
    }
    const int pos = off + __popc(m & ((1u << lane) - 1u));
    if (in && pos < cap) list[pos] = value;
    __syncthreads();
    return tot;
}

// Block superset of the objects that any source point within rho of (cx, cy, cz) may keep
// (spread_z: the sources' extent along z).  An object stays when it can meet the slopes of crystal
// d's rays from some source (near_bundle), and passes the reference's cone test widened by the sources'
// extent: |u_o - u_d| <= (rho + r_o)/(L_o - rho) + (rho + r_d)/(L_d - rho) + 1e-4 at the centre (each
// direction moves by at most rho/(L - rho) in chord length, each angular radius r/L grows to at most
// r/(L - rho)).  Each warp scans its own run of objects, a lane keeping a group's ballot, so the block
// meets twice and not twice per 256 objects.  On a production plane the slope test leaves 73 of the
// 435 objects that pass the cone test, and the elements' own filters scan that much less: 128
// crystals x that plane, 77.4 -> 74.1 ms.
__device__ void build_superset(const DevGeom& g, Superset& bs, int d, float cx, float cy, float cz, float rho,
                               float spread_z)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const float4 P = __ldg(&g.cry.pos[d]);
    const float rdd = 0.5f * __ldg(&g.cry.size[d].w);
    const float Ld = sqrtf((P.x - cx) * (P.x - cx) + (P.y - cy) * (P.y - cy) + (P.z - cz) * (P.z - cz));
    const float uxd = (P.x - cx) / Ld, uyd = (P.y - cy) / Ld, uzd = (P.z - cz) / Ld;
    const bool near_d = !(Ld - rho > 0.5f);
    const float td = near_d ? 0.0f : (rho + rdd) / (Ld - rho);
    float4 rd;
    const bool slopes = bundle_rect(g, d, cx, cy, cz, rho, spread_z, rd);
    const int N = g.n_holes + g.n_det;
    const int groups = (N + 31) / 32, per = (groups + kWarps - 1) / kWarps;   // at most 61 groups per warp
    const int g0 = wid * per, g1 = min(g0 + per, groups);
    unsigned kept0 = 0u, kept1 = 0u;          // ballots of groups g0 + lane and g0 + 32 + lane
    int count = 0;
    for (int k = g0; k < g1; ++k) {
        const int i = k * 32 + lane;
        bool keep = false;
        if (i < N && i - g.n_holes != d && (!slopes || near_bundle(g, cx, cy, cz, rd, i, rho, spread_z))) {
            const float4 od = object_data(g, i);
            const float ro = (i < g.n_holes) ? od.w : 0.5f * od.w;
            const float Lo = sqrtf((od.x - cx) * (od.x - cx) + (od.y - cy) * (od.y - cy) +
                                   (od.z - cz) * (od.z - cz));
            keep = true;
            if (!near_d && Lo - rho > 0.5f) {
                const float dx = (od.x - cx) / Lo - uxd, dy = (od.y - cy) / Lo - uyd,
                            dz = (od.z - cz) / Lo - uzd;
                const float thr = (rho + ro) / (Lo - rho) + td + 1e-4f;
                keep = sqrtf(dx * dx + dy * dy + dz * dz) <= thr;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (lane == ((k - g0) & 31)) (k - g0 < 32 ? kept0 : kept1) = m;
        count += __popc(m);
    }
    if (lane == 0) bs.warp_cnt[wid] = count;
    __syncthreads();
    int pos = 0, total = 0;
    for (int k = 0; k < kWarps; ++k) {
        const int c = bs.warp_cnt[k];
        if (k < wid) pos += c;
        total += c;
    }
    if (total <= kSuperCap) {
        for (int k = g0; k < g1; ++k) {
            const unsigned m = __shfl_sync(0xffffffffu, k - g0 < 32 ? kept0 : kept1, (k - g0) & 31);
            if ((m >> lane) & 1u) bs.sid[pos + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(k * 32 + lane);
            pos += __popc(m);
        }
    }
    if (threadIdx.x == 0) bs.s_count = total <= kSuperCap ? total : -1;
    __syncthreads();
}

// Output block of one brick: rows (crystals) from det_begin, voxels vox_begin .. vlast.
struct BrickOut {
    float* out;
    long long ld, vox_begin, vlast;
    int det_begin;
    float* sub_out;           // per-sub-element contributions (local sampled form), or nullptr
    int det_count;
};

// Shared memory of each kernel instance; two blocks of kWarps warps per SM.
template <int MODE, bool ELL> struct SmemOf { using type = RefSmem; };       // float modes 0, 1
template <bool ELL> struct SmemOf<2, ELL> { using type = IdSmem<Mode64>; };
template <bool ELL> struct SmemOf<3, ELL> { using type = IdSmem<ModeLocal<ELL>>; };

// One work item: crystal det_begin + di against voxel brick b of the block's grid.  The block builds the cone
// superset of the brick, then its warps take the brick's voxels in turn.
// SAMPLED: elements of the sampled form `smp` (source points anywhere in the voxels: the
// superset radius grows by half a voxel diagonal).
template <int MODE, bool COUNT, bool ELL = false, bool SAMPLED = false>
__device__ __forceinline__ void pe_brick(const DevGeom& g, typename SmemOf<MODE, ELL>::type& sm, int lane, int wid,
                                         const BrickOut& O, int di, const BrickGrid& B, long long b, float cr,
                                         float sr,
                                         unsigned long long* counters, const Sampling* smp = nullptr,
                                         float rotation = 0.0f)
{
    Superset& sup = sm.sup;
    const int gz = (int)(b / ((long long)B.nbx * B.nby));
    const int rem = (int)(b - (long long)gz * B.nbx * B.nby);
    const int gy = rem / B.nbx, gx = rem - gy * B.nbx;
    const int bx = B.bx, by = B.by, bz = B.bz;
    const int x0 = B.x0 + gx * bx, y0 = B.y0 + gy * by, z0 = B.z0 + gz * bz;
    const int x1 = min(x0 + bx - 1, B.x1), y1 = min(y0 + by - 1, B.y1), z1 = min(z0 + bz - 1, B.z1);
    const int d = O.det_begin + di;
    // the brick's voxels inside the block, so that a ragged block's warps share them evenly (and a
    // brick without any builds no superset)
    const int n_slots = bx * by * bz;
    auto active = [&](int slot) {
        const int ix = x0 + slot % bx, iy = y0 + (slot / bx) % by, iz = z0 + slot / (bx * by);
        const long long v = ix + g.nx * ((long long)iy + (long long)g.ny * iz);
        return slot < n_slots && ix <= x1 && iy <= y1 && iz <= z1 && v >= O.vox_begin && v <= O.vlast;
    };
    int n_active = 0;
    if (SAMPLED && n_slots <= 32) {        // every warp counts them; build_superset's barriers publish the list
        const bool in = active(lane);
        const unsigned m = __ballot_sync(0xffffffffu, in);
        n_active = __popc(m);
        if (wid == 0 && in) sup.slot[__popc(m & ((1u << lane) - 1u))] = (unsigned short)lane;
    } else {
        for (int base = 0; base < n_slots; base += kThreads) {
            const int slot = base + threadIdx.x;
            n_active += block_append(sup, active(slot), (unsigned short)slot, sup.slot, n_active, 512, lane, wid);
        }
    }
    if (n_active == 0) return;
    // brick centre and radius from its extreme voxel centres (rotation about z keeps lengths)
    float ax, ay, az, bxx, byy, bzz;
    voxel_centre(g, x0 + g.nx * ((long long)y0 + g.ny * z0), 1.0f, 0.0f, ax, ay, az);
    voxel_centre(g, x1 + g.nx * ((long long)y1 + g.ny * z1), 1.0f, 0.0f, bxx, byy, bzz);
    const float mx = 0.5f * (ax + bxx), my = 0.5f * (ay + byy), mz = 0.5f * (az + bzz);
    float rho = 0.5f * sqrtf((bxx - ax) * (bxx - ax) + (byy - ay) * (byy - ay) +
                             (bzz - az) * (bzz - az)) + 1e-3f;
    float spread_z = 0.5f * fabsf(bzz - az) + 1e-3f;
    if constexpr (SAMPLED) {
        rho += 0.5f * sqrtf(g.wx * g.wx + g.wy * g.wy + g.wz * g.wz);
        spread_z += 0.5f * fabsf(g.wz);
    }
    build_superset(g, sup, d, mx * cr - my * sr, mx * sr + my * cr, mz, rho, spread_z);
    // the block's warps start each element together: they then run the same phase's loop, which the
    // schedulers' instruction caches hold, most of the time
    for (int base = 0; base < n_active; base += kWarps) {
        if (base + wid < n_active) {
            const int slot = sup.slot[base + wid];
            const int ix = x0 + slot % bx, iy = y0 + (slot / bx) % by, iz = z0 + slot / (bx * by);
            const long long v = ix + g.nx * ((long long)iy + (long long)g.ny * iz);
            float val;
            if constexpr (MODE <= 1 && SAMPLED) {
                val = (float)pe_element_sampled<ELL>(g, sup, sm.w[wid], d, v, cr, sr, lane, *smp);
            } else if constexpr (MODE <= 1) {
                val = (float)pe_element_ref<MODE, COUNT, ELL>(g, sup, sm.w[wid], d, v, cr, sr, lane, counters);
            } else if constexpr (MODE == 3) {
                float* so = nullptr;
                if (SAMPLED && O.sub_out)
                    so = O.sub_out + ((v - O.vox_begin) * O.det_count + di) * (long long)(smp->nx * smp->ny * smp->nz);
                val = (float)pe_element_local<ELL, SAMPLED>(g, sup, sm.w[wid], d, v, cr, sr, rotation, lane, smp, so);
            } else {
                val = (float)pe_element64(g, sup, sm.w[wid], d, v, cr, sr, rotation, lane);
            }
            if (lane == 0) O.out[(long long)di * O.ld + (v - O.vox_begin)] = val;
        }
        __syncthreads();
    }
}

template <int MODE, bool COUNT, bool ELL, bool SAMPLED = false>
__global__ void __launch_bounds__(kThreads, 2)
pe_kernel(DevGeom g, PeLaunch L, BrickGrid B)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& sm = *reinterpret_cast<typename SmemOf<MODE, ELL>::type*>(smem_raw);
    Superset& bs = sm.sup;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const float ang = L.rotation * g.angle_step;           // :1006
    const float cr = cosf(ang), sr = sinf(ang);
    const long long vlast = L.vox_begin + L.vox_count - 1;
    const long long n_bricks = (long long)B.nbx * B.nby * B.nbz;
    const long long total = n_bricks * L.det_count;
    const BrickOut O{L.out, L.ld, L.vox_begin, vlast, L.det_begin, L.sub_out, L.det_count};
    for (;;) {
        if (threadIdx.x == 0) bs.item = (long long)atomicAdd(L.work_counter, 1ull);
        __syncthreads();
        const long long item = bs.item;
        __syncthreads();
        if (item >= total) break;
        const int di = (int)(item / n_bricks);
        const long long b = item - (long long)di * n_bricks;
        pe_brick<MODE, COUNT, ELL, SAMPLED>(g, sm, lane, wid, O, di, B, b, cr, sr, L.counters, &L.smp, L.rotation);
    }
}

// Shared memory of the batched kernel: the block's working set plus the geometry of the
// task in hand (copied in when the block moves to a task of another geometry).
template <int MODE, bool ELL>
struct BatchSmem {
    typename SmemOf<MODE, ELL>::type bs;
    DevGeom g;
    int task;
};

// Batched launch: one persistent grid over the items of many (geometry, rotation, block)
// tasks, taken from one work counter; a block finds its item's task by binary search over
// the tasks' first item numbers.
template <int MODE, bool ELL>
__global__ void __launch_bounds__(kThreads, 2) pe_batch_kernel(BatchLaunch B)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BatchSmem<MODE, ELL>& sm = *reinterpret_cast<BatchSmem<MODE, ELL>*>(smem_raw);
    Superset& bs = sm.bs.sup;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int cur_geom = -1;
    for (;;) {
        if (threadIdx.x == 0) {
            const long long item = (long long)atomicAdd(B.work_counter, 1ull);
            int lo = 0, hi = B.n_tasks - 1;
            while (lo < hi) {                       // last task with item_begin <= item
                const int mid = (lo + hi + 1) >> 1;
                if (B.tasks[mid].item_begin <= item) lo = mid; else hi = mid - 1;
            }
            bs.item = item;
            sm.task = lo;
        }
        __syncthreads();
        const long long item = bs.item;
        const BatchTask T = B.tasks[sm.task];
        __syncthreads();
        if (item >= B.total_items) break;
        if (T.geom != cur_geom) {                   // block-uniform
            const int* src = reinterpret_cast<const int*>(B.geoms + T.geom);
            int* dst = reinterpret_cast<int*>(&sm.g);
            for (int i = threadIdx.x; i < (int)(sizeof(DevGeom) / sizeof(int)); i += kThreads) dst[i] = src[i];
            cur_geom = T.geom;
            __syncthreads();
        }
        const DevGeom& g = sm.g;
        const float ang = T.rotation * g.angle_step;       // :1006
        const float cr = cosf(ang), sr = sinf(ang);
        const long long n_bricks = (long long)T.bricks.nbx * T.bricks.nby * T.bricks.nbz;
        const long long local = item - T.item_begin;
        const int di = (int)(local / n_bricks);
        const long long b = local - (long long)di * n_bricks;
        const BrickOut O{T.out, T.ld, T.vox_begin, T.vox_begin + T.vox_count - 1, T.det_begin, nullptr, T.det_count};
        pe_brick<MODE, false, ELL>(g, sm.bs, lane, wid, O, di, T.bricks, b, cr, sr, nullptr, nullptr, T.rotation);
    }
}

#include "pe_adjoint.cuh"

}  // namespace

// Brick of a block's work items: 16 voxels (two elements per warp share one superset; the superset of
// a 32- or 64-voxel brick is larger and measured 2-11 % slower per element), 4 x 4 in a plane, or
// as many rows as the block has.  Blocks of few elements take 8 or 4 voxels, so that every block of
// the grid gets an item: a 36 x 128 matrix took 582 us in 32-voxel bricks, 328 in 16, 299 in 8.
static BrickGrid choose_bricks(const DevGeom& g, const PeLaunch& L, int blocks)
{
    const BrickGrid all = brick_grid(g, L.vox_begin, L.vox_count, 1, 1, 1);
    const int rows = all.y1 - all.y0 + 1;
    const double elements = (double)L.det_count * (double)L.vox_count;
    const int voxels = elements >= 32.0 * blocks ? 16 : (elements >= 4.0 * blocks ? 8 : 4);
    const int by = rows >= 4 && voxels == 16 ? 4 : (rows >= 2 ? 2 : 1);
    return brick_grid(g, L.vox_begin, L.vox_count, voxels / by, by, 1);
}

template <int MODE, bool COUNT, bool ELL, bool SAMPLED = false>
static int launch_mode(const DevGeom& g, const PeLaunch& L, int num_sms, cudaStream_t stream)
{
    const int smem = (int)sizeof(typename SmemOf<MODE, ELL>::type);
    static unsigned long long configured = 0;   // one bit per device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(__atomic_load_n(&configured, __ATOMIC_ACQUIRE) & bit)) {
        if (cudaFuncSetAttribute(pe_kernel<MODE, COUNT, ELL, SAMPLED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 smem) !=
            cudaSuccess)
            return -1;
        __atomic_fetch_or(&configured, bit, __ATOMIC_RELEASE);
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pe_kernel<MODE, COUNT, ELL, SAMPLED>, kThreads, smem);
    if (per_sm < 1) per_sm = 1;
    pe_kernel<MODE, COUNT, ELL, SAMPLED><<<num_sms * per_sm, kThreads, smem, stream>>>(g, L, choose_bricks(g, L, num_sms * per_sm));
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <int KIND, bool ELL>
static int launch_adjoint_kind(const DevGeom& g, const AdjLaunch& L, int num_sms, cudaStream_t stream)
{
    const int smem = (int)sizeof(AdjSmem<KIND>);
    static unsigned long long configured = 0;   // one bit per device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(__atomic_load_n(&configured, __ATOMIC_ACQUIRE) & bit)) {
        if (cudaFuncSetAttribute(pe_adjoint_kernel<KIND, ELL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
            cudaSuccess)
            return -1;
        __atomic_fetch_or(&configured, bit, __ATOMIC_RELEASE);
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pe_adjoint_kernel<KIND, ELL>, kThreads, smem);
    if (per_sm < 1) per_sm = 1;
    pe_adjoint_kernel<KIND, ELL><<<num_sms * per_sm, kThreads, smem, stream>>>(g, L);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Systems with elliptical holes (sysmat_set_hole_shapes) run the elliptical instances.
int launch_pe_adjoint(const DevGeom& g, const AdjLaunch& L, int kind, int num_sms, cudaStream_t stream)
{
    if (g.hole_shape) {
        if (kind == 0) return launch_adjoint_kind<0, true>(g, L, num_sms, stream);
        if (kind == 1) return launch_adjoint_kind<1, true>(g, L, num_sms, stream);
        return launch_adjoint_kind<2, true>(g, L, num_sms, stream);
    }
    if (kind == 0) return launch_adjoint_kind<0, false>(g, L, num_sms, stream);
    if (kind == 1) return launch_adjoint_kind<1, false>(g, L, num_sms, stream);
    return launch_adjoint_kind<2, false>(g, L, num_sms, stream);
}

template <int MODE, bool ELL>
static int configure_batch_mode(int* per_sm)
{
    const int smem = (int)sizeof(BatchSmem<MODE, ELL>);
    static unsigned long long configured = 0;   // one bit per device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(__atomic_load_n(&configured, __ATOMIC_ACQUIRE) & bit)) {
        if (cudaFuncSetAttribute(pe_batch_kernel<MODE, ELL>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
            cudaSuccess)
            return -1;
        __atomic_fetch_or(&configured, bit, __ATOMIC_RELEASE);
    }
    *per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, pe_batch_kernel<MODE, ELL>, kThreads, smem) !=
        cudaSuccess)
        return -1;
    if (*per_sm < 1) *per_sm = 1;
    return 0;
}

int configure_pe_batch(int mode, bool ell, int* blocks_per_sm)
{
    if (mode == 2) return configure_batch_mode<2, false>(blocks_per_sm);   // shapes read at run time
    if (mode == 3) return ell ? configure_batch_mode<3, true>(blocks_per_sm) : configure_batch_mode<3, false>(blocks_per_sm);
    if (ell) {
        return mode == 0 ? configure_batch_mode<0, true>(blocks_per_sm)
                         : configure_batch_mode<1, true>(blocks_per_sm);
    }
    return mode == 0 ? configure_batch_mode<0, false>(blocks_per_sm) : configure_batch_mode<1, false>(blocks_per_sm);
}

template <int MODE, bool ELL>
static void launch_batch_mode(const BatchLaunch& B, int grid, cudaStream_t stream)
{
    pe_batch_kernel<MODE, ELL><<<grid, kThreads, (int)sizeof(BatchSmem<MODE, ELL>), stream>>>(B);
}

int launch_pe_batch(const BatchLaunch& B, int mode, bool ell, int grid, cudaStream_t stream)
{
    if (B.n_tasks < 1 || B.total_items < 1) return 0;
    if (mode == 2) launch_batch_mode<2, false>(B, grid, stream);   // FP64: shapes read at run time
    else if (mode == 3) ell ? launch_batch_mode<3, true>(B, grid, stream) : launch_batch_mode<3, false>(B, grid, stream);
    else if (mode == 0) ell ? launch_batch_mode<0, true>(B, grid, stream) : launch_batch_mode<0, false>(B, grid, stream);
    else ell ? launch_batch_mode<1, true>(B, grid, stream) : launch_batch_mode<1, false>(B, grid, stream);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_pe(const DevGeom& g, const PeLaunch& L, int mode, int num_sms, cudaStream_t stream)
{
    if (mode == 2) return g.t64.cry_pos ? launch_mode<2, false, false>(g, L, num_sms, stream) : -1;
    if (mode == 3) {
        if (!g.t64.cry_pos) return -1;
        return g.hole_shape ? launch_mode<3, false, true>(g, L, num_sms, stream)
                            : launch_mode<3, false, false>(g, L, num_sms, stream);
    }
    if (g.hole_shape) {                   // systems with elliptical holes
        if (L.counters) return launch_mode<0, true, true>(g, L, num_sms, stream);
        return mode == 0 ? launch_mode<0, false, true>(g, L, num_sms, stream)
                         : launch_mode<1, false, true>(g, L, num_sms, stream);
    }
    if (L.counters) return launch_mode<0, true, false>(g, L, num_sms, stream);
    return mode == 0 ? launch_mode<0, false, false>(g, L, num_sms, stream)
                     : launch_mode<1, false, false>(g, L, num_sms, stream);
}

int launch_pe_local_sampled(const DevGeom& g, const PeLaunch& L, int num_sms, cudaStream_t stream)
{
    if (!g.t64.cry_pos) return -1;
    return g.hole_shape ? launch_mode<3, false, true, true>(g, L, num_sms, stream)
                        : launch_mode<3, false, false, true>(g, L, num_sms, stream);
}

int launch_pe_sampled(const DevGeom& g, const PeLaunch& L, int num_sms, cudaStream_t stream)
{
    if (g.hole_shape) return launch_mode<1, false, true, true>(g, L, num_sms, stream);
    return launch_mode<1, false, false, true>(g, L, num_sms, stream);
}

}  // namespace sysmat
