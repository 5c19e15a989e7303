// Primary-Compton scatter kernels and geometry-relationship bitmaps for sm_100a.
//
// Physics follows the reference kernels crystalScatterSysMatCuda
// (ScatterGen_RayTracing_CircularHole/scatter.cu:1077-1437) and collimatorScatterSysMatCuda
// (:1544-1936; hole solid angle of the collimator-only program at
// ScatterGen_Collimator/scatter.cu:1212-1215).  Execution plan:
//
//  * everything that depends only on the (scatterer s, detector d) pair is computed once
//    per pair instead of once per (d, v, s) item: the scatter point in d's frame, the
//    scatter-to-detector distance, the absorption chord in d, and the list of attenuating
//    crystals flagged by the relationship bitmap with a non-zero chord (the reference scans
//    all D crystals of the bitmap for every item, :1343-1401);
//  * the self-attenuation term (:1404-1417) is exactly 0 with the reference's 1x1x1
//    detector sub-division (the crystal box and the sub-element box are the same floats), so
//    it is not evaluated;
//  * the Klein-Nishina angular ratio is the reference's left Riemann sum with
//    n = (int)((theta_max - theta_min) / 0.01f) + 1 terms (:980-993, :1338), evaluated through the
//    Euler-Maclaurin identity
//      sum_{i=0..n} F(a + i h) h = int_a^b F + h/2 (F(a) + F(b)) + h^2/12 (F'(b) - F'(a)) + O(h^4)
//    from two FP64 tables of cubics (scatter.cuh), instead of n+1 cos/sin evaluations; theta_min,
//    theta_max and n are computed with the reference's float formulas, so the step count
//    matches.  The normalisation over [0, pi] is a host FP64 sum;
//  * per item, the corner cosines of the theta range are formed only for the corners that can be
//    extreme, the theta_min chord only for rays that pass near the crystal, and divisions share
//    correctly rounded reciprocals.  Configuration 3, 768 voxels: 39.5 -> 27.6 ms (all eight
//    corners, every chord and three table interpolations per end before; bound by issue, 62 % of
//    the slots, 465 warp instructions per item);
//  * one thread per matrix element (d, v); a block shares d, so pair records are staged in
//    shared memory and attenuator lists are broadcast loads; each element sums its items in
//    FP64 (the reference adds float items with atomicAdd in an unspecified order).
#include <algorithm>
#include <cmath>

#include <cub/cub.cuh>

#include "rounding.cuh"
#include "scatter.cuh"

namespace sysmat {

namespace {

constexpr int kItemThreads = kScatterBlockVoxels;
constexpr int kPairChunk = 256;

// ---- reference helper formulas (scatter.cu:961-1038) ----

// Scattering angle at the point a between the directions s -> a and a -> d; mb = |a -> d|, the
// pair's distance (within an ulp of what the three differences here give: another product is fused).
__device__ __forceinline__ float cone_angle(float xs, float ys, float zs, float xa, float ya, float za,
                                            float xd, float yd, float zd, float mb)
{
    const float a0 = xa - xs, a1 = ya - ys, a2 = za - zs;
    const float b0 = xd - xa, b1 = yd - ya, b2 = zd - za;
    const float dot = b0 * a0 + b1 * a1 + b2 * a2;
    const float ma = sqrt_mid(a0 * a0 + a1 * a1 + a2 * a2);
    float c = div_rn(dot, ma * mb);
    if (c > 1.0f) c = 1.0f;
    if (c < -1.0f) c = -1.0f;
    return acosf(c);
}

__device__ __forceinline__ float dist3(float x1, float y1, float z1, float x2, float y2, float z2)
{
    return sqrtf((x1 - x2) * (x1 - x2) + (y1 - y2) * (y1 - y2) + (z1 - z2) * (z1 - z2));
}

// Crystal d's single sub-element centre (1x1x1 division, :1242-1252) in its own frame and
// in world coordinates.
struct DetPoint {
    float xDs, yDs, zDs, xD, yD, zD;
};

__device__ __forceinline__ DetPoint det_point(float4 P, float4 S, float4 T)
{
    DetPoint q;
    const float w = S.x, t = S.y, h = S.z;
    q.xDs = -w / 2.0f + ((float)0 + 0.5f) / 1.0f * w;
    q.zDs = -h / 2.0f + ((float)0 + 0.5f) / 1.0f * h;
    q.yDs = -t / 2.0f + ((float)0 + 0.5f) / 1.0f * t;
    q.xD = P.x + (q.xDs * T.x - q.zDs * T.y);
    q.zD = P.z + (q.xDs * T.y + q.zDs * T.x);
    q.yD = P.y + q.yDs;
    return q;
}

// ---- relationship bitmaps (no atomics) ----
//
// A bit asks whether crystal k lies in the angular cone of a segment i-j, seen from one end: that
// |u_k - u_j| <= c_k + c_j for the unit directions u and angular radii c of k and j seen from i.
// Directions and radii belong to (i, k) alone, so a block takes one i, forms them for every
// crystal once in shared memory (Seen), and each bit costs two shared loads, a distance and a
// compare; a warp's ballot is the output word.  Per bit the former kernels recomputed both
// directions with six divisions and four roots: the two bitmaps of configuration 3 (1.6e9 bits)
// took 36.6 ms, and take 4.2 ms (bound by issue; the 201 MB written take 0.03 ms).

constexpr int kBitmapThreads = 256;

// Angular radius of a crystal at distance l, at least 2^-51.
__device__ __forceinline__ float angular_radius(float r, float l) { return fmaxf(r / l, 0x1p-51f); }

// A crystal seen from a point: unit direction and angular radius (scatter.cu:1476-1500, :1975-1996).
__device__ __forceinline__ float4 seen_from(float xi, float yi, float zi, const float* __restrict__ pk, float rk)
{
    const float l = dist3(pk[1], pk[2], pk[3], xi, yi, zi);
    return make_float4((pk[1] - xi) / l, (pk[2] - yi) / l, (pk[3] - zi) / l, angular_radius(rk, l));
}

__device__ __forceinline__ float crystal_radius(const float* __restrict__ p)
{
    return sqrtf(p[4] * p[4] + p[6] * p[6] + p[5] * p[5]) / 2.0f;
}

// |u_k - u_j| <= c_k + c_j.  The root is the IEEE one from 2^-50 on; crystals that lie behind one another
// but for offsets below 1e-15 of their distance count as that far apart, which angular_radius's least value
// always covers.
__device__ __forceinline__ bool cone_meets(const float4& k, const float4& j)
{
    const float dx = k.x - j.x, dy = k.y - j.y, dz = k.z - j.z;
    const float d2 = dx * dx + dy * dy + dz * dz;
    return sqrt_mid(d2 < kMinRoot ? kMinRoot : d2) <= k.w + j.w;   // false for a NaN (no direction)
}

// cone_meets of crystals k and i (centres, radii) seen from (x, y, z).  Approximate directions decide
// unless the distance and the radii's sum are within the error of both forms: reciprocal roots to
// 2^-22 put a unit vector's components within 4e-7, a distance of two within 3e-6 with the reference
// form's own rounding, and the radii's sum within 1e-6 of itself.  Configuration 3, the crystal bitmap:
// 4.04 -> 2.18 ms.
__device__ __forceinline__ bool cone_meets_from(float x, float y, float z, float xk, float yk, float zk, float rk,
                                                float xi, float yi, float zi, float ri)
{
    const float kx = xk - x, ky = yk - y, kz = zk - z, jx = xi - x, jy = yi - y, jz = zi - z;
    const float a = rsqrtf(kx * kx + ky * ky + kz * kz), b = rsqrtf(jx * jx + jy * jy + jz * jz);
    const float ux = kx * a - jx * b, uy = ky * a - jy * b, uz = kz * a - jz * b;
    const float d2 = ux * ux + uy * uy + uz * uz, c = rk * a + ri * b;
    const float m = 4e-6f + 2e-6f * c, low = fmaxf(c - m, 0.0f), top = c + m;
    if (d2 < low * low) return true;
    if (d2 > top * top) return false;
    const float lk = dist3(xk, yk, zk, x, y, z), li = dist3(xi, yi, zi, x, y, z);
    return cone_meets(make_float4(kx / lk, ky / lk, kz / lk, angular_radius(rk, lk)),
                      make_float4(jx / li, jy / li, jz / li, angular_radius(ri, li)));
}

// Whether crystal k may attenuate the path between crystals i and j, i < j (:1465-1534).
__device__ __forceinline__ bool crystal_related(const float* __restrict__ det, int i, int j, int k)
{
    const float *pi = det + 12 * i, *pj = det + 12 * j, *pk = det + 12 * k;
    const float ri = crystal_radius(pi), rj = crystal_radius(pj), rk = crystal_radius(pk);
    return cone_meets(seen_from(pi[1], pi[2], pi[3], pk, rk), seen_from(pi[1], pi[2], pi[3], pj, rj)) ||
           cone_meets(seen_from(pj[1], pj[2], pj[3], pk, rk), seen_from(pj[1], pj[2], pj[3], pi, ri));
}

// Whether crystal k may attenuate the path from hole i (raw parameters hr) to crystal j:
// k's bounding sphere within the angular cone of the hole-to-j segment, seen from the hole
// (scatter.cu:1963-2006; raw y, no FOV offset).
__device__ __forceinline__ bool collimator_related(const float* __restrict__ det, float4 hr, int j, int k)
{
    const float xi = hr.x, yi = (hr.y + hr.z) / 2.0f, zi = hr.w;
    const float *pj = det + 12 * j, *pk = det + 12 * k;
    return cone_meets(seen_from(xi, yi, zi, pk, crystal_radius(pk)), seen_from(xi, yi, zi, pj, crystal_radius(pj)));
}

// First pair of row i (pairs (i, j), i <= j < n).
__host__ __device__ __forceinline__ long long pair_row(long long n, long long i) { return i * n - i * (i - 1) / 2; }

// The bit of the crystal bitmap at flat index `bit` (pair index (i n - i (i+1) / 2 + j), then k).
__device__ bool crystal_bit(const float* __restrict__ det, int n, long long bit)
{
    const long long pair = bit / n;
    const int k = (int)(bit - pair * n);
    const double disc = (2.0 * n + 1.0) * (2.0 * n + 1.0) - 8.0 * (double)pair;
    long long i = (long long)floor(((2.0 * n + 1.0) - sqrt(disc > 0 ? disc : 0)) / 2.0);
    if (i < 0) i = 0;
    while (i > 0 && pair_row(n, i) > pair) --i;
    while (pair_row(n, i + 1) <= pair) ++i;
    const int ii = (int)i, jj = (int)(pair - pair_row(n, i) + i);
    return ii < jj && k != ii && k != jj && crystal_related(det, ii, jj, k);
}

// Block (i, part of row i): the words whose first bit belongs to pairs (i, i .. n-1).
__global__ void __launch_bounds__(kBitmapThreads) bitmap_crystal_kernel(const float* __restrict__ det, int n,
                                                                        long long bits, uint32_t* __restrict__ out)
{
    extern __shared__ float4 seen[];                       // every crystal seen from crystal i, then radii
    float* radius = reinterpret_cast<float*>(seen + n);
    const int i = blockIdx.x, lane = threadIdx.x & 31;
    const float* pi = det + 12 * i;
    const float xi = pi[1], yi = pi[2], zi = pi[3];
    for (int k = threadIdx.x; k < n; k += kBitmapThreads) {
        const float rk = crystal_radius(det + 12 * k);
        radius[k] = rk;
        seen[k] = seen_from(xi, yi, zi, det + 12 * k, rk);
    }
    __syncthreads();
    const float ri = radius[i];
    const long long b0 = pair_row(n, i) * n, b1 = pair_row(n, i + 1) * n;
    const int step = 32 * (kBitmapThreads / 32) * gridDim.y;
    const int step_j = step / n, step_k = step - step_j * n;
    long long w = (b0 + 31) / 32 + blockIdx.y * (kBitmapThreads / 32) + (threadIdx.x >> 5);
    const int off = (int)(w * 32 + lane - b0);             // a row holds at most n^2 < 2^31 bits
    int j = off / n, k = off - j * n;
    for (; w * 32 < b1; w += step / 32) {
        const long long bit = w * 32 + lane;
        bool hit = false;
        if (bit < b1) {
            const int jj = i + j;
            if (j > 0 && k != i && k != jj) {
                hit = cone_meets(seen[k], seen[jj]);
                if (!hit) {                                 // seen from the other end
                    const float* pj = det + 12 * jj;
                    const float* pk = det + 12 * k;
                    const float xj = __ldg(&pj[1]), yj = __ldg(&pj[2]), zj = __ldg(&pj[3]);
                    hit = cone_meets_from(xj, yj, zj, __ldg(&pk[1]), __ldg(&pk[2]), __ldg(&pk[3]), radius[k], xi, yi,
                                          zi, ri);
                }
            }
        } else if (bit < bits) {                            // the word's tail in the next rows
            hit = crystal_bit(det, n, bit);
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) out[w] = m;
        k += step_k;
        j += step_j;
        if (k >= n) {
            k -= n;
            ++j;
        }
    }
}

// Block (hole i, part of its bits): the words whose first bit belongs to hole i (bit
// (i n + j) n + k).
__global__ void __launch_bounds__(kBitmapThreads) bitmap_collimator_kernel(const float* __restrict__ det,
                                                                           const float4* __restrict__ hraw, int n,
                                                                           long long bits, uint32_t* __restrict__ out)
{
    extern __shared__ float4 seen[];                       // every crystal seen from the hole
    const int i = blockIdx.x, lane = threadIdx.x & 31;
    const float4 hr = __ldg(&hraw[i]);
    const float xi = hr.x, yi = (hr.y + hr.z) / 2.0f, zi = hr.w;
    for (int k = threadIdx.x; k < n; k += kBitmapThreads)
        seen[k] = seen_from(xi, yi, zi, det + 12 * k, crystal_radius(det + 12 * k));
    __syncthreads();
    const long long nn = (long long)n * n, b0 = i * nn, b1 = b0 + nn;
    const int step = 32 * (kBitmapThreads / 32) * gridDim.y;
    const int step_j = step / n, step_k = step - step_j * n;
    long long w = (b0 + 31) / 32 + blockIdx.y * (kBitmapThreads / 32) + (threadIdx.x >> 5);
    const int off = (int)(w * 32 + lane - b0);
    int j = off / n, k = off - j * n;
    for (; w * 32 < b1; w += step / 32) {
        const long long bit = w * 32 + lane;
        bool hit = false;
        if (bit < b1) {
            hit = cone_meets(seen[k], seen[j]);
        } else if (bit < bits) {                            // the word's tail in the next holes
            const long long ij = bit / n;
            hit = collimator_related(det, __ldg(&hraw[ij / n]), (int)(ij % n), (int)(bit - ij * n));
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) out[w] = m;
        k += step_k;
        j += step_j;
        if (k >= n) {
            k -= n;
            ++j;
        }
    }
}

// ---- pair tables ----

// Scatter point of scatterer s: crystal centre (y + FOV) or hole centre
// ((y1 + y2) / 2 + FOV), scatter.cu:1221-1223, :1707-1709.
__device__ __forceinline__ void scatter_point(const DevGeom& g, int s, float& xs, float& ys, float& zs)
{
    if (s < g.n_det) {
        const float4 p = __ldg(&g.cry.pos[s]);
        xs = p.x; ys = p.y; zs = p.z;
    } else {
        const float4 r = __ldg(&g.hole.raw[s - g.n_det]);
        xs = r.x;
        ys = (r.y + r.z) / 2.0f + g.fov;
        zs = r.w;
    }
}

// Pair-table kernels: one warp per (detector d, scatterer s) pair.  The pair's candidate
// attenuators (its bitmap row, or the relationship predicate) are compacted into a per-warp
// list in ascending crystal order, so every lane tests one; those whose box the path may meet
// (a few of a hundred) move on to a queue, and the reference's chord is formed for 32 of them at
// a time.  Both kernels on configuration 3: 7.2 -> 5.2 ms against a chord for every candidate.  The
// lists have a buffer of their own, so a context's first tables keep the counts they were sized
// from (3 ms).
constexpr int kPairWarps = 8;          // warps per block
constexpr int kPairSpan = 1024;        // candidates compacted per pass (32 per lane)

struct PairLists {
    uint16_t list[kPairSpan];          // candidates, from the pass's first crystal
    int queue[64];                     // crystals whose chord is formed
};

// Bit start of the n-bit row of pair (s, d): crystal pairs in the upper triangle (i < j),
// hole pairs by (hole, detector).
__device__ __forceinline__ long long pair_row_bit(int n, int s, int d)
{
    if (s < n) {
        const long long i = s < d ? s : d, j = s < d ? d : s;
        return (i * n - (i * (i + 1)) / 2 + j) * n;
    }
    return ((long long)(s - n) * n + d) * n;
}

// Candidates a0 .. a0+31 of pair (s, d) as a bit mask (bit k: crystal a0 + k), without
// crystal d and scatter crystal s.  NATIVE hole scatterers evaluate the predicate instead of
// reading a bitmap.
template <bool NATIVE>
__device__ __forceinline__ uint32_t candidate_mask(const DevGeom& g, const uint32_t* bm, long long base,
                                                   float4 hr, int s, int d, int a0)
{
    const int n = g.n_det;
    if (a0 >= n) return 0u;
    const int span = n - a0 < 32 ? n - a0 : 32;
    uint32_t m = 0u;
    if (NATIVE && s >= n) {
        for (int k = 0; k < span; ++k)
            if (collimator_related(g.raw_det, hr, d, a0 + k)) m |= 1u << k;
    } else {
        const long long b = base + a0, w = b >> 5;
        const int sh = (int)(b & 31);
        const uint32_t lo = __ldg(&bm[w]);
        // the next word only when the row continues into it
        const uint32_t hi = (sh != 0 && w + 1 <= ((base + n - 1) >> 5)) ? __ldg(&bm[w + 1]) : 0u;
        m = __funnelshift_r(lo, hi, sh);
        if (span < 32) m &= (1u << span) - 1u;
    }
    if (d >= a0 && d - a0 < 32) m &= ~(1u << (d - a0));
    if (s < n && s >= a0 && s - a0 < 32) m &= ~(1u << (s - a0));
    return m;
}

// Whether the segment may meet crystal a's box: no face normal and no edge cross product of the
// segment separates them by more than the chord's rounding can bridge (the axes that do are
// exact rejects: the reference's chord is 0 beyond them).  Rounding moves the chord's faces by
// some 1e-6 of the coordinates, and directions below kEps count as parallel there.
__device__ __forceinline__ bool may_meet(const DevGeom& g, int a, float xs, float ys, float zs, const DetPoint& q)
{
    const float4 pa = __ldg(&g.cry.pos[a]);
    const float4 sa = __ldg(&g.cry.size[a]);
    const float4 ta = __ldg(&g.cry.trig[a]);
    float mx, my, mz, vx, vy, vz;                        // middle and half of the segment, a's frame
    to_crystal_frame(pa.x, pa.y, pa.z, ta.z, ta.w, 0.5f * (xs + q.xD), 0.5f * (ys + q.yD), 0.5f * (zs + q.zD), mx, my, mz);
    to_crystal_frame(0.0f, 0.0f, 0.0f, ta.z, ta.w, 0.5f * (q.xD - xs), 0.5f * (q.yD - ys), 0.5f * (q.zD - zs), vx, vy, vz);
    const float ax = fabsf(vx), ay = fabsf(vy), az = fabsf(vz);
    const float slack = 2.0f * kEps + 1e-5f * (fabsf(mx) + fabsf(my) + fabsf(mz) + ax + ay + az + fabsf(pa.x) +
                                               fabsf(pa.y) + fabsf(pa.z));
    const float hx = 0.5f * sa.x + slack, hy = 0.5f * sa.y + slack, hz = 0.5f * sa.z + slack;
    return !(fabsf(mx) > hx + ax || fabsf(my) > hy + ay || fabsf(mz) > hz + az ||
             fabsf(mx * vy - my * vx) > hx * ay + hy * ax || fabsf(my * vz - mz * vy) > hy * az + hz * ay ||
             fabsf(mx * vz - mz * vx) > hx * az + hz * ax);
}

// Chord of the scatter point -> detector point segment inside an attenuating crystal (tables pa, sa,
// ta; scatter.cu:1377-1394).  Out of line: the kernel that counts a pair's chords and the one that
// stores them then run the same instructions.  Inlined in each, the compiler may contract a sum of
// products one way here and another way there, and a chord at a threshold is 0 in one of them only.
static __device__ __noinline__ float attenuator_chord(float4 pa, float4 sa, float4 ta, float xs, float ys, float zs,
                                                      float xD, float yD, float zD)
{
    float xa, ya, za, xb, yb, zb;
    to_crystal_frame(pa.x, pa.y, pa.z, ta.z, ta.w, xs, ys, zs, xa, ya, za);
    to_crystal_frame(pa.x, pa.y, pa.z, ta.z, ta.w, xD, yD, zD, xb, yb, zb);
    return box_chord(xa, ya, za, xb, yb, zb, -0.5f * sa.x, -0.5f * sa.y, -0.5f * sa.z, 0.5f * sa.x,
                     0.5f * sa.y, 0.5f * sa.z);
}

// Warp-collective walk over the attenuators of pair (s, d) in ascending crystal order: f(a,
// len, ok) is called by every lane for each group of 32 queued candidates (ok false on lanes past
// the group's end).  lists: the warp's shared buffers.
template <bool NATIVE, typename F>
__device__ __forceinline__ void warp_attenuators(const DevGeom& g, const uint32_t* bm_cry, const uint32_t* bm_col,
                                                 int s, int d, float xs, float ys, float zs, const DetPoint& q,
                                                 int lane, PairLists& lists, F&& f)
{
    const int n = g.n_det;
    const long long base = (NATIVE && s >= n) ? 0 : pair_row_bit(n, s, d);
    const uint32_t* bm = s < n ? bm_cry : bm_col;
    const float4 hr = (NATIVE && s >= n) ? __ldg(&g.hole.raw[s - n]) : make_float4(0.f, 0.f, 0.f, 0.f);
    int queued = 0;
    auto flush = [&](int cnt) {                            // the first cnt <= 32 of the queue
        const bool ok = lane < cnt;
        const int a = ok ? lists.queue[lane] : 0;
        const float len = ok ? attenuator_chord(__ldg(&g.cry.pos[a]), __ldg(&g.cry.size[a]), __ldg(&g.cry.trig[a]), xs,
                                                ys, zs, q.xD, q.yD, q.zD)
                             : 0.0f;
        f(a, len, ok);
    };
    for (int c0 = 0; c0 < n; c0 += kPairSpan) {
        const int a0 = c0 + 32 * lane;
        uint32_t m = candidate_mask<NATIVE>(g, bm, base, hr, s, d, a0);
        const int cnt = __popc(m);
        int incl = cnt;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += v;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        int pos = incl - cnt;
        while (m) {
            lists.list[pos++] = (uint16_t)(a0 - c0 + __ffs(m) - 1);
            m &= m - 1u;
        }
        __syncwarp();
        for (int b = 0; b < total; b += 32) {
            const int a = b + lane < total ? c0 + lists.list[b + lane] : 0;
            const bool hit = b + lane < total && may_meet(g, a, xs, ys, zs, q);
            const unsigned hits = __ballot_sync(0xffffffffu, hit);
            if (hit) lists.queue[queued + __popc(hits & ((1u << lane) - 1u))] = a;
            queued += __popc(hits);
            __syncwarp();
            if (queued >= 32) {
                flush(32);
                __syncwarp();
                if (lane < queued - 32) lists.queue[lane] = lists.queue[32 + lane];
                __syncwarp();
                queued -= 32;
            }
        }
    }
    if (queued > 0) flush(queued);
    __syncwarp();
}

__device__ __forceinline__ bool pair_enabled(const DevGeom& g, int parts, int s, int d)
{
    if (s < g.n_det) return (parts & 1) && s != d;
    return (parts & 2) != 0;
}

// Layer of hole h (global numbering, layer by layer).
__device__ __forceinline__ int hole_layer(const DevGeom& g, int h)
{
    int m = 0;
    while (m + 1 < g.n_layers && h >= g.layer[m + 1].hole_begin) ++m;
    return m;
}

// Distance from the centre (x, ym, z) of hole h along the unit direction k to where the
// path leaves the hole (side wall or cap), capped at len.
__device__ __forceinline__ float hole_exit(float4 a, float r, float ym, float kx, float ky, float kz, float len)
{
    const float kk = kx * kx + kz * kz;
    float t = len;
    if (kk > 0.0f) t = fminf(t, r / sqrtf(kk));
    if (ky > 0.0f) t = fminf(t, (a.z - ym) / ky);
    else if (ky < 0.0f) t = fminf(t, (a.y - ym) / ky);
    return t;
}

// Native model: tungsten crossed by the scattered photon from the centre S of hole h to the
// detector point D, as sum_m mu_pe,m L_m and sum_m mu_C,m L_m, L_m = plate chord of layer m
// minus the hole chords of layer m (the reference chords; the scatter hole's own part is its
// exit distance from S, and in its own layer the plate chord runs from the plate entry seen
// from D to S).
__device__ void tungsten_path(const DevGeom& g, int h, float sx, float sy, float sz, float dx, float dy, float dz,
                              float& w_pe, float& w_c)
{
    w_pe = 0.0f;
    w_c = 0.0f;
    const int mh = hole_layer(g, h);
    const float ex = dx - sx, ey = dy - sy, ez = dz - sz;
    const float len = sqrtf(ex * ex + ey * ey + ez * ez);
    const float kx = ex / len, ky = ey / len, kz = ez / len;
    const float n2 = ex * ex + ez * ez;
    for (int m = 0; m < g.n_layers; ++m) {
        const LayerInfo& Ly = g.layer[m];
        const float box = (m == mh) ? box_chord_inside(dx, dy, dz, sx, sy, sz, Ly.x1, Ly.y1, Ly.z1, Ly.x2, Ly.y2, Ly.z2)
                                    : box_chord(sx, sy, sz, dx, dy, dz, Ly.x1, Ly.y1, Ly.z1, Ly.x2, Ly.y2, Ly.z2);
        if (box == 0.0f) continue;
        float holes = 0.0f;
        for (int j = Ly.hole_begin; j < Ly.hole_begin + Ly.hole_count; ++j) {
            const float4 a = __ldg(&g.hole.a[j]);
            const float r = __ldg(&g.hole.b[j].x);
            if (j == h) {
                holes = holes + hole_exit(a, r, sy, kx, ky, kz, len);
                continue;
            }
            // the line keeps further than r from the axis: the chord is 0 (exact-safe reject)
            const float cr = ex * (a.w - sz) - ez * (a.x - sx);
            if (cr * cr > r * r * n2 * 1.001f + 1e-12f) continue;
            holes = holes + cyl_chord(sx, sy, sz, dx, dy, dz, a.x, a.y, a.z, a.w, r);
        }
        const float L = box - holes;
        if (L > 0.0f) {
            w_pe = w_pe + Ly.mu_pe * L;
            w_c = w_c + Ly.mu_c * L;
        }
    }
}

template <bool NATIVE>
__global__ void __launch_bounds__(32 * kPairWarps) pair_count_kernel(DevGeom g, int parts, const uint32_t* bm_cry,
                                                                     const uint32_t* bm_col, long long* counts)
{
    __shared__ PairLists lists[kPairWarps];
    const int ns = g.n_det + (NATIVE ? g.n_holes : g.n_holes0);
    const long long np = (long long)g.n_det * ns;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (long long p = (long long)blockIdx.x * kPairWarps + wid; p < np; p += (long long)gridDim.x * kPairWarps) {
        const int d = (int)(p / ns), s = (int)(p - (long long)d * ns);
        int c = 0;
        if (pair_enabled(g, parts, s, d)) {
            float xs, ys, zs;
            scatter_point(g, s, xs, ys, zs);
            const DetPoint q = det_point(__ldg(&g.cry.pos[d]), __ldg(&g.cry.size[d]), __ldg(&g.cry.trig[d]));
            warp_attenuators<NATIVE>(g, bm_cry, bm_col, s, d, xs, ys, zs, q, lane, lists[wid],
                                     [&](int, float len, bool ok) {
                                         c += __popc(__ballot_sync(0xffffffffu, ok && len != 0.0f));
                                     });
        }
        if (lane == 0) counts[p] = c;
    }
}

template <bool NATIVE>
__global__ void __launch_bounds__(32 * kPairWarps) pair_fill_kernel(DevGeom g, int parts, const uint32_t* bm_cry,
                                                                    const uint32_t* bm_col, const long long* offsets,
                                                                    PairRec* pairs, AttEntry* att)
{
    __shared__ PairLists lists[kPairWarps];
    const int ns = g.n_det + (NATIVE ? g.n_holes : g.n_holes0);
    const long long np = (long long)g.n_det * ns;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (long long p = (long long)blockIdx.x * kPairWarps + wid; p < np; p += (long long)gridDim.x * kPairWarps) {
        const int d = (int)(p / ns), s = (int)(p - (long long)d * ns);
        PairRec r{};
        r.valid = pair_enabled(g, parts, s, d);
        if (r.valid) {
            float xs, ys, zs;
            scatter_point(g, s, xs, ys, zs);
            const float4 P = __ldg(&g.cry.pos[d]), S = __ldg(&g.cry.size[d]), T = __ldg(&g.cry.trig[d]);
            const DetPoint q = det_point(P, S, T);
            to_crystal_frame(P.x, P.y, P.z, T.z, T.w, xs, ys, zs, r.xss, r.yss, r.zss);   // :1290-1292
            r.lsd = dist3(xs, ys, zs, q.xD, q.yD, q.zD);                                   // :1275
            // absorption chord along the extended scatter->detector ray (:1420-1424)
            const float ux1 = ((float)0 / (float)1 - 0.5f) * S.x, ux2 = (((float)0 + 1.0f) / (float)1 - 0.5f) * S.x;
            const float uy1 = ((float)0 / (float)1 - 0.5f) * S.y, uy2 = (((float)0 + 1.0f) / (float)1 - 0.5f) * S.y;
            const float uz1 = ((float)0 / (float)1 - 0.5f) * S.z, uz2 = (((float)0 + 1.0f) / (float)1 - 0.5f) * S.z;
            const float xt = q.xDs + 1000.0f * (q.xDs - r.xss) / r.lsd;
            const float yt = q.yDs + 1000.0f * (q.yDs - r.yss) / r.lsd;
            const float zt = q.zDs + 1000.0f * (q.zDs - r.zss) / r.lsd;
            r.labs = box_chord(r.xss, r.yss, r.zss, xt, yt, zt, ux1, uy1, uz1, ux2, uy2, uz2);
            // row-relative start: a row holds at most ns * D entries, which fits an int
            r.att_begin = (int)(offsets[p] - offsets[(long long)d * ns]);
            // never past the pair's own part of the list, whatever the bitmaps hold by now
            AttEntry* dst = att + offsets[p];
            const int room = (int)(offsets[p + 1] - offsets[p]);
            int k = 0;
            warp_attenuators<NATIVE>(g, bm_cry, bm_col, s, d, xs, ys, zs, q, lane, lists[wid],
                                     [&](int a, float len, bool ok) {
                                         const bool nz = ok && len != 0.0f;
                                         const unsigned m = __ballot_sync(0xffffffffu, nz);
                                         const int at = k + __popc(m & ((1u << lane) - 1u));
                                         if (nz && at < room) {
                                             const float4 mu = __ldg(&g.cry.mu[a]);
                                             dst[at] = AttEntry{len, mu.y, mu.z};
                                         }
                                         k += __popc(m);
                                     });
            r.att_count = min(k, room);
        }
        if (lane == 0) pairs[p] = r;
    }
}

// Native model: the tungsten terms of each pair, one thread per pair.
__global__ void pair_native_kernel(DevGeom g, int parts, PairNative* nat)
{
    const int ns = g.n_det + g.n_holes;
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (long long)g.n_det * ns) return;
    const int d = (int)(p / ns), s = (int)(p - (long long)d * ns);
    PairNative n{};
    if (s >= g.n_det && pair_enabled(g, parts, s, d)) {
        float xs, ys, zs;
        scatter_point(g, s, xs, ys, zs);
        const DetPoint q = det_point(__ldg(&g.cry.pos[d]), __ldg(&g.cry.size[d]), __ldg(&g.cry.trig[d]));
        const int h = s - g.n_det;
        tungsten_path(g, h, xs, ys, zs, q.xD, q.yD, q.zD, n.w_pe, n.w_c);
        const LayerInfo& Ly = g.layer[hole_layer(g, h)];
        n.mu_tot_h = Ly.mu_total;
        n.mu_c_h = Ly.mu_c;
    }
    nat[p] = n;
}

// ---- scatter items ----

struct ElemConst {
    float xI, yI, zI, xIs, yIs, zIs;
    DetPoint q;
    float w, t, h;
    float mu_pe, mu_c, eres;
    float lo, hi;
    bool bounded;               // both bounds small enough for div_by
    float rdet, near2;          // circumscribed radius; its square with a margin
};

// A staged pair: its record and what else belongs to the pair alone, formed once per block: the
// angular half width of d seen from the scatter point, and 1 / |corner - scatter point| for d's
// eight corners (approximate: they only select corners).
struct StagedPair {
    PairRec r;
    float half_width;
    float rcorner[8];
    float slack;                // bound of the selection's error per unit of the summed terms
};

// Corner c of d (bit 0: x, bit 1: y, bit 2: z) minus the scatter point, in d's frame
// (the faces of the single detector unit, (0 / 1 - 0.5) w and (1 / 1 - 0.5) w, :1305-1320).
__device__ __forceinline__ void corner_offset(const ElemConst& e, const PairRec& pr, int c, float& bx, float& by, float& bz)
{
    bx = ((c & 1) ? 0.5f * e.w : -0.5f * e.w) - pr.xss;
    by = ((c & 2) ? 0.5f * e.t : -0.5f * e.t) - pr.yss;
    bz = ((c & 4) ? 0.5f * e.h : -0.5f * e.h) - pr.zss;
}

__device__ __forceinline__ StagedPair stage_pair(const ElemConst& e, const PairRec& pr)
{
    StagedPair p;
    p.r = pr;
    p.half_width = e.rdet / 2.0f / pr.lsd;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        float bx, by, bz;
        corner_offset(e, pr, c, bx, by, bz);
        p.rcorner[c] = rsqrtf(bx * bx + by * by + bz * bz);
    }
    float far = 0.0f;
#pragma unroll
    for (int c = 0; c < 8; ++c) far = fmaxf(far, p.rcorner[c]);
    p.slack = 2e-6f * far;
    return p;
}

// One (d, v, s) item; (xs, ys, zs) the scatter point, w_s the interaction weight (PE * muC/muPE
// or hole solid angle * muC/mu of layer 0).  Returns the float the reference would atomically add.
template <bool NATIVE>
__device__ float scatter_item(const ElemConst& e, const StagedPair& sp, const PairNative& pn,
                              const AttEntry* __restrict__ att, float xs, float ys, float zs, float w_s, float e0,
                              float re0, float integ, const double* __restrict__ kn_tab)
{
    const PairRec& pr = sp.r;
    const float cone = cone_angle(e.xI, e.yI, e.zI, xs, ys, zs, e.q.xD, e.q.yD, e.q.zD, pr.lsd);
    const float es = e0 / (1.0f + (e0 / 511.0f) * (1.0f - cosf(cone)));     // :1016-1023
    const float res = e.eres * sqrt_mid(div_by(es, e0, re0));
    constexpr float kFwhm = 2.35482f, kRFwhm = 1.0f / 2.35482f;
    const float fw = div_by(res, kFwhm, kRFwhm);           // 2 * res / 2.35482f is its double
    if ((es * (1 + 2 * fw)) <= e.lo || (es * (1 - 2 * fw)) >= e.hi) return 0.0f;   // :1263-1269
    const float rs = rcp_rn(es);
    // energy-window probability (calculategaussianIntegral, :1025-1038)
    const float s2 = (float)((double)(fw * es) * 1.4142135623730951), rs2 = rcp_rn(s2);
    float z1 = div_by(e.lo - es, s2, rs2), z2 = div_by(e.hi - es, s2, rs2);
    if (!(s2 >= kMinDivisor && e.bounded)) {               // no energy spread, or an open window
        z1 = (e.lo - es) / s2;
        z2 = (e.hi - es) / s2;
    }
    const float pwin = 0.5f * (erff(z2) - erff(z1));
    const float sc = sinf(cone);
    float phi;
    if (pr.lsd * sc * 2.0f <= e.rdet) phi = (float)(2.0f * 3.14159265358979323846);
    else {
        const float arg = div_rn(sp.half_width, sc);
        phi = 4.0f * asinf((arg <= 1.0f) ? arg : 1.0f);
    }
    // theta range over the 8 corners of the (single) detector unit (:1305-1335).  The reference
    // takes the extremes of the 8 corner angles acos(c_k); acos decreases, so they are
    // acos(max c_k) and acos(min c_k).  c_k = dot_k / (|a| |b_k|) rounds each quotient; approximate
    // cosines (error below a quarter of the slack) select the corners that can be extreme, usually
    // two or three, and only those quotients are formed.
    const float ax = pr.xss - e.xIs, ay = pr.yss - e.yIs, az = pr.zss - e.zIs;
    const float ma = sqrt_mid(ax * ax + ay * ay + az * az);
    float tmin, tmax;
    {
        const float hw = 0.5f * e.w, ht = 0.5f * e.t, hh = 0.5f * e.h;
        const float x0 = ax * (-hw - pr.xss), x1 = ax * (hw - pr.xss);
        const float y0 = ay * (-ht - pr.yss), y1 = ay * (ht - pr.yss);
        const float z0 = az * (-hh - pr.zss), z1 = az * (hh - pr.zss);
        float c[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            c[k] = (((k & 1) ? x1 : x0) + ((k & 2) ? y1 : y0) + ((k & 4) ? z1 : z0)) * sp.rcorner[k];
        float top = c[0], low = c[0];
#pragma unroll
        for (int k = 1; k < 8; ++k) {
            top = fmaxf(top, c[k]);
            low = fminf(low, c[k]);
        }
        const float slack = (fabsf(x0) + fabsf(x1) + fabsf(y0) + fabsf(y1) + fabsf(z0) + fabsf(z1)) * sp.slack;
        unsigned can = 0u;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (c[k] >= top - slack || c[k] <= low + slack) can |= 1u << k;
        float cmin = 2.0f, cmax = -2.0f;
        while (can) {
            const int k = __ffs(can) - 1;
            can &= can - 1u;
            float bx, by, bz;
            corner_offset(e, pr, k, bx, by, bz);
            const float dot = bx * ax + by * ay + bz * az;
            const float mb = sqrt_mid(bx * bx + by * by + bz * bz);
            float ck = div_rn(dot, ma * mb);
            if (ck > 1.0f) ck = 1.0f;
            if (ck < -1.0f) ck = -1.0f;
            cmin = fminf(cmin, ck);
            cmax = fmaxf(cmax, ck);
        }
        tmin = acosf(cmax);
        tmax = acosf(cmin);
    }
    // a ray from the voxel through the scatter point that crosses d has theta_min = 0.  It passes
    // d's centre at lsd sin(cone), so beyond d's circumscribed radius there is no chord to form.  A float
    // cosine of the cone is within nine units of 2^-24 of the exact one, and cosines that far apart have
    // squared sines within 1.1e-6 of each other, whatever the angle: a tenth of a millimetre at 1 m.
    const float pass = pr.lsd * sc;
    if (pass * pass <= __fmaf_rn(1.2e-6f * pr.lsd, pr.lsd, e.near2)) {
        const float rdis = rcp_rn(ma);                     // |voxel - point| in d's frame (:1314)
        const float xt = pr.xss + div_by(1000.0f * ax, ma, rdis);
        const float yt = pr.yss + div_by(1000.0f * ay, ma, rdis);
        const float zt = pr.zss + div_by(1000.0f * az, ma, rdis);
        const float lthr = box_chord(e.xIs, e.yIs, e.zIs, xt, yt, zt, -0.5f * e.w, -0.5f * e.t, -0.5f * e.h, 0.5f * e.w,
                                     0.5f * e.t, 0.5f * e.h);
        if (lthr > 0.001f) tmin = 0.0f;
    }
    const int n = (int)((tmax - tmin) / 0.01f);
    const double ta = (double)tmin, tb = ta + (double)n * (double)0.01f;
    const float ratio = (float)(kn_tab_eval(kn_tab, kKnU, tb) - kn_tab_eval(kn_tab, kKnV, ta)) / integ;
    // attenuation by the flagged crystals at the scattered energy (:1369-1396): the scaled
    // coefficient depends only on (mu_pe, mu_c) and E', so it is formed again only when they differ
    // from the last ones used, starting from d's own (same operands, same float)
    auto scaled_pe = [&](float mu) {                       // mu e0 e0 e0 / es / es / es
        return div_by(div_by(div_by(mu * e0 * e0 * e0, es, rs), es, rs), es, rs);
    };
    const float mpe_s = scaled_pe(e.mu_pe);                // :1411-1417
    const float mt_s = mpe_s + div_by(e.mu_c * e0, es, rs);
    float a_sum = 0.0f;
    float c_pe = e.mu_pe, c_c = e.mu_c, mt = mt_s;
    for (int k = 0; k < pr.att_count; ++k) {
        const AttEntry ae = att[pr.att_begin + k];
        if (!(ae.mu_pe == c_pe && ae.mu_c == c_c)) {
            c_pe = ae.mu_pe;
            c_c = ae.mu_c;
            mt = scaled_pe(ae.mu_pe) + div_by(ae.mu_c * e0, es, rs);
        }
        a_sum = a_sum + ae.len * mt;
    }
    if (NATIVE && (pn.w_pe != 0.0f || pn.w_c != 0.0f))     // native model: tungsten at E'
        a_sum = a_sum + (scaled_pe(pn.w_pe) + div_by(pn.w_c * e0, es, rs));
    const double c = (double)(w_s * phi / 2.0f) * (1.0 / 3.14159265358979323846) * (double)ratio *
                     (double)pwin * (double)expf(-a_sum) *
                     (double)(1.0f - expf(-pr.labs * mt_s)) * (double)mpe_s / (double)mt_s;
    return (float)c;
}

// One block's share of a scatter launch: detector row di, voxels vblock * kItemThreads + t
// (t = threadIdx.x).  sp, spn: the block's pair staging buffers in shared memory.
template <bool NATIVE>
__device__ __forceinline__ void scatter_rows(const DevGeom& g, const ScatterPhysics& ph, const ScatterLaunch& L,
                                             int di, long long vblock, StagedPair* sp, PairNative* spn)
{
    const int d = L.det_begin + di;
    const long long vi = vblock * kItemThreads + threadIdx.x;
    const bool active = vi < L.vox_count;
    const long long v = L.vox_begin + (active ? vi : 0);
    const int ns = g.n_det + (NATIVE ? g.n_holes : g.n_holes0);

    const float4 P = __ldg(&g.cry.pos[d]), S = __ldg(&g.cry.size[d]);
    const float4 M = __ldg(&g.cry.mu[d]), T = __ldg(&g.cry.trig[d]);
    const bool run = ph.use_compton && (M.x > 0.01f);                       // :1226-1228

    ElemConst e;
    const float ang = L.rotation * g.angle_step;
    voxel_centre(g, v, cosf(ang), sinf(ang), e.xI, e.yI, e.zI);
    to_crystal_frame(P.x, P.y, P.z, T.z, T.w, e.xI, e.yI, e.zI, e.xIs, e.yIs, e.zIs);
    e.q = det_point(P, S, T);
    e.w = S.x; e.t = S.y; e.h = S.z;
    e.mu_pe = M.y; e.mu_c = M.z; e.eres = M.w;
    if (ph.same_window) { e.lo = ph.lo; e.hi = ph.hi; }
    else {
        e.lo = (1 - e.eres / 2.0f) * ph.e0;                                  // :1161-1162
        e.hi = (1 + e.eres / 2.0f) * ph.e0;
    }
    e.bounded = fabsf(e.lo) <= 1e15f && fabsf(e.hi) <= 1e15f;
    e.rdet = sqrtf(e.w * e.w / (float)1 / (float)1 + e.h * e.h / (float)1 / (float)1 +
                   e.t * e.t / (float)1 / (float)1) / 2.0f;
    e.near2 = (1.001f * e.rdet + 0.01f) * (1.001f * e.rdet + 0.01f);
    const float re0 = rcp_rn(ph.e0);

    double acc_c = 0.0, acc_h = 0.0;
    const int s_begin = (L.parts & 1) ? 0 : g.n_det;
    const int s_end = (L.parts & 2) ? ns : g.n_det;
    const PairRec* prow = L.pairs + (long long)d * ns;
    const AttEntry* att_row = L.att + L.att_offsets[(long long)d * ns];
    for (int s0 = s_begin; s0 < s_end; s0 += kPairChunk) {
        const int cnt = min(kPairChunk, s_end - s0);
        __syncthreads();
        for (int k = threadIdx.x; k < cnt; k += kItemThreads) {
            sp[k] = stage_pair(e, prow[s0 + k]);
            if constexpr (NATIVE) spn[k] = L.native[(long long)d * ns + s0 + k];
        }
        __syncthreads();
        if (!run || !active) continue;
        for (int k = 0; k < cnt; ++k) {
            const int s = s0 + k;
            const StagedPair& pr = sp[k];
            if (!pr.r.valid) continue;
            float xs, ys, zs, w_s;
            const bool crystal = s < g.n_det;
            if (crystal) {
                w_s = __ldg(&L.pe[(long long)s * g.nvox + v]) * e.mu_c / e.mu_pe;   // :1218-1219
                if (w_s == 0.0f) continue;          // the item is exactly 0
                const float4 ps = __ldg(&g.cry.pos[s]);
                xs = ps.x; ys = ps.y; zs = ps.z;
            } else {
                const float4 hr = __ldg(&g.hole.raw[s - g.n_det]);
                xs = hr.x;
                ys = (hr.y + hr.z) / 2.0f + g.fov;
                zs = hr.w;
                const float lih = dist3(e.xI, e.yI, e.zI, xs, ys, zs);
                float sa;
                if (L.hole_model != 1) {                                  // :1711-1715
                    const float vr = 0.1f;
                    // (pi vr^2 + h vr) / (4 pi lih^2) * |dy| / lih, with one double reciprocal
                    const double rl = 1.0 / (double)lih;
                    sa = (float)(((double)(vr * vr) * 3.14159265358979323846 + (double)((hr.z - hr.y) * vr)) *
                                 (1.0 / (4.0 * 3.14159265358979323846)) * rl * rl * (double)fabsf(ys - e.yI) * rl);
                } else {                                                  // ScatterGen_Collimator :1212-1215
                    const float vr = 0.2f;
                    sa = (vr * vr + (hr.z - hr.y) * vr) / (4.0f * lih * lih);
                }
                if (NATIVE) w_s = sa / spn[k].mu_tot_h * spn[k].mu_c_h;        // the hole's own layer
                else w_s = sa / ph.col_mu_tot0 * ph.col_mu_c0;            // :1716
            }
            // one call site keeps a single copy of the item code
            const double c = (double)scatter_item<NATIVE>(e, pr, spn[NATIVE ? k : 0], att_row, xs, ys, zs, w_s,
                                                          ph.e0, re0, ph.integ, L.kn_tab);
            if (crystal) acc_c += c;
            else acc_h += c;
        }
    }
    if (!active) return;
    float outv;
    if ((L.parts & 3) == 3) outv = (float)acc_h + (float)acc_c;              // :2354-2357
    else if (L.parts & 1) outv = (float)acc_c;
    else outv = (float)acc_h;
    L.out[(long long)di * L.ld + vi] = outv;
}

template <bool NATIVE>
__global__ void __launch_bounds__(kItemThreads)
scatter_kernel(DevGeom g, ScatterPhysics ph, ScatterLaunch L)
{
    __shared__ StagedPair sp[kPairChunk];
    __shared__ PairNative spn[NATIVE ? kPairChunk : 1];
    scatter_rows<NATIVE>(g, ph, L, blockIdx.y, blockIdx.x, sp, spn);
}

// Batched scatter: one persistent grid over the (row, voxel block) items of many tasks, taken
// from one counter; a block finds its item's task by binary search over the tasks' first item
// numbers and copies the task (and its geometry, when it changes) into shared memory.  Each
// item runs scatter_rows, so every element equals the single launch's bit for bit.
__global__ void __launch_bounds__(kItemThreads) scatter_batch_kernel(ScatterBatchLaunch B)
{
    __shared__ StagedPair sp[kPairChunk];
    __shared__ PairNative spn[kPairChunk];
    __shared__ DevGeom sg;
    __shared__ ScatterTask st;
    __shared__ long long s_item;
    __shared__ int s_task;
    int cur_task = -1, cur_geom = -1;
    for (;;) {
        if (threadIdx.x == 0) {
            const long long item = (long long)atomicAdd(B.work_counter, 1ull);
            int lo = 0, hi = B.n_tasks - 1;
            while (lo < hi) {                       // last task with item_begin <= item
                const int mid = (lo + hi + 1) >> 1;
                if (B.tasks[mid].item_begin <= item) lo = mid; else hi = mid - 1;
            }
            s_item = item;
            s_task = lo;
        }
        __syncthreads();
        const long long item = s_item;
        const int task = s_task;
        __syncthreads();
        if (item >= B.total_items) break;
        if (task != cur_task) {                     // block-uniform
            const int* src = reinterpret_cast<const int*>(B.tasks + task);
            int* dst = reinterpret_cast<int*>(&st);
            for (int i = threadIdx.x; i < (int)(sizeof(ScatterTask) / sizeof(int)); i += kItemThreads) dst[i] = src[i];
            __syncthreads();
            if (st.geom != cur_geom) {
                const int* gs = reinterpret_cast<const int*>(B.geoms + st.geom);
                int* gd = reinterpret_cast<int*>(&sg);
                for (int i = threadIdx.x; i < (int)(sizeof(DevGeom) / sizeof(int)); i += kItemThreads) gd[i] = gs[i];
                cur_geom = st.geom;
            }
            cur_task = task;
            __syncthreads();
        }
        const long long local = item - st.item_begin;
        const int di = (int)(local / st.n_vblocks);
        const long long vb = local - (long long)di * st.n_vblocks;
        if (st.L.hole_model == 2) scatter_rows<true>(sg, st.ph, st.L, di, vb, sp, spn);
        else scatter_rows<false>(sg, st.ph, st.L, di, vb, sp, spn);
    }
}

}  // namespace

long long bitmap_crystal_words(int n)
{
    const long long pairs = (long long)n * (n + 1) / 2;
    return (pairs * n + 31) / 32;
}

long long bitmap_collimator_words(int n, int nh0)
{
    return ((long long)n * n * nh0 + 31) / 32;
}

// Blocks per row or hole: enough for several waves over the SMs, no more than there are words.
static unsigned bitmap_parts(long long rows, long long words)
{
    const long long want = (8 * 148 + rows - 1) / rows, most = words / rows / (kBitmapThreads / 32) + 1;
    return (unsigned)std::max(1LL, std::min(want, most));
}

// Opt-in above 48 KB of dynamic shared memory: the most crystals that a system can have, not this call's
// number, since the limit belongs to the kernel and calls from several threads may set it in turn.
constexpr int kMostCrystals = (kNDetector - 1) / 12;

template <class K>
static int bitmap_smem(K kernel, size_t per_crystal, int n)
{
    if (per_crystal * n <= 48 * 1024) return 0;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(per_crystal * kMostCrystals)) ==
                   cudaSuccess
               ? 0
               : -1;
}

int launch_bitmap_crystal(const DevGeom& g, uint32_t* words, cudaStream_t s)
{
    const long long nw = bitmap_crystal_words(g.n_det), n = g.n_det;
    if (nw == 0) return 0;
    constexpr size_t per_crystal = sizeof(float4) + sizeof(float);   // at most 6666 crystals: 133 KB
    if (bitmap_smem(bitmap_crystal_kernel, per_crystal, g.n_det)) return -1;
    const dim3 grid((unsigned)n, bitmap_parts(n, nw));
    bitmap_crystal_kernel<<<grid, kBitmapThreads, per_crystal * n, s>>>(g.raw_det, g.n_det, n * (n + 1) / 2 * n, words);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_bitmap_collimator(const DevGeom& g, uint32_t* words, cudaStream_t s)
{
    const long long nw = bitmap_collimator_words(g.n_det, g.n_holes0), n = g.n_det;
    if (nw == 0) return 0;
    constexpr size_t per_crystal = sizeof(float4);
    if (bitmap_smem(bitmap_collimator_kernel, per_crystal, g.n_det)) return -1;
    const dim3 grid((unsigned)g.n_holes0, bitmap_parts(g.n_holes0, nw));
    bitmap_collimator_kernel<<<grid, kBitmapThreads, per_crystal * n, s>>>(g.raw_det, g.hole.raw, g.n_det, n * n * g.n_holes0,
                                                                words);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <bool NATIVE>
static int build_pairs(const DevGeom& g, int parts, const uint32_t* bm_cry, const uint32_t* bm_col,
                       ScatterScratch& scratch, PairRec** pairs, PairNative** native, AttEntry** att,
                       long long** att_offsets, cudaStream_t s)
{
    const int ns = g.n_det + (NATIVE ? g.n_holes : g.n_holes0);
    const long long np = (long long)g.n_det * ns;
    // layout: [counts (np+1)][64-bit offsets (np+1)][cub temp][pairs][native]; the lists have a buffer of
    // their own, sized once they are counted
    size_t temp_bytes = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, temp_bytes, (long long*)nullptr, (long long*)nullptr, np + 1, s);
    auto align = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t off_counts = 0;
    const size_t off_offsets = align(off_counts + sizeof(long long) * (np + 1));
    const size_t off_temp = align(off_offsets + sizeof(long long) * (np + 1));
    const size_t off_pairs = align(off_temp + temp_bytes);
    const size_t off_native = align(off_pairs + sizeof(PairRec) * np);
    const size_t fixed = align(off_native + (NATIVE ? sizeof(PairNative) * np : 0));
    if (scratch.bytes < fixed) {
        scatter_scratch_free(scratch);
        if (cudaMalloc(&scratch.base, fixed) != cudaSuccess) { scratch.base = nullptr; return -2; }
        scratch.bytes = fixed;
    }
    char* base = (char*)scratch.base;
    long long* counts = (long long*)(base + off_counts);
    long long* offsets = (long long*)(base + off_offsets);
    const unsigned blocks = (unsigned)((np + 255) / 256);
    // one warp per pair, grid-stride beyond 148 x 64 blocks (64 per SM of a B200)
    const unsigned warp_blocks = (unsigned)std::min<long long>((np + kPairWarps - 1) / kPairWarps, 148LL * 64);
    pair_count_kernel<NATIVE><<<warp_blocks, 32 * kPairWarps, 0, s>>>(g, parts, bm_cry, bm_col, counts);
    if (cudaMemsetAsync(counts + np, 0, sizeof(long long), s) != cudaSuccess) return -1;
    cub::DeviceScan::ExclusiveSum(base + off_temp, temp_bytes, counts, offsets, np + 1, s);
    long long total = 0;
    if (cudaMemcpyAsync(&total, offsets + np, sizeof(long long), cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
    if (total < 0) return -1;
    const size_t need = sizeof(AttEntry) * (size_t)(total > 0 ? total : 1);
    if (scratch.att_bytes < need) {                       // its own buffer: the counts above stay
        cudaFree(scratch.att);
        scratch.att = nullptr;
        scratch.att_bytes = 0;
        if (cudaMalloc(&scratch.att, need) != cudaSuccess) { scratch.att = nullptr; return -2; }
        scratch.att_bytes = need;
    }
    *pairs = (PairRec*)(base + off_pairs);
    PairNative* nat = NATIVE ? (PairNative*)(base + off_native) : nullptr;
    if (native) *native = nat;
    *att = (AttEntry*)scratch.att;
    *att_offsets = offsets;
    pair_fill_kernel<NATIVE><<<warp_blocks, 32 * kPairWarps, 0, s>>>(g, parts, bm_cry, bm_col, offsets, *pairs, *att);
    if (NATIVE) pair_native_kernel<<<blocks, 256, 0, s>>>(g, parts, nat);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int build_scatter_pairs(const DevGeom& g, int parts, const uint32_t* bm_cry, const uint32_t* bm_col,
                        ScatterScratch& scratch, PairRec** pairs, AttEntry** att, long long** att_offsets,
                        cudaStream_t s)
{
    return build_pairs<false>(g, parts, bm_cry, bm_col, scratch, pairs, nullptr, att, att_offsets, s);
}

int build_scatter_pairs_native(const DevGeom& g, int parts, const uint32_t* bm_cry, ScatterScratch& scratch,
                               PairRec** pairs, PairNative** native, AttEntry** att, long long** att_offsets,
                               cudaStream_t s)
{
    return build_pairs<true>(g, parts, bm_cry, nullptr, scratch, pairs, native, att, att_offsets, s);
}

int scatter_batch_blocks_per_sm()
{
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, scatter_batch_kernel, kItemThreads, 0) != cudaSuccess)
        return 1;
    return per_sm < 1 ? 1 : per_sm;
}

int launch_scatter_batch(const ScatterBatchLaunch& B, int grid, cudaStream_t s)
{
    if (B.n_tasks < 1 || B.total_items < 1) return 0;
    scatter_batch_kernel<<<grid, kItemThreads, 0, s>>>(B);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_scatter(const DevGeom& g, const ScatterPhysics& ph, const ScatterLaunch& L, cudaStream_t s)
{
    if (L.det_count == 0 || L.vox_count == 0) return 0;
    dim3 grid((unsigned)((L.vox_count + kItemThreads - 1) / kItemThreads), (unsigned)L.det_count);
    if (L.hole_model == 2) scatter_kernel<true><<<grid, kItemThreads, 0, s>>>(g, ph, L);
    else scatter_kernel<false><<<grid, kItemThreads, 0, s>>>(g, ph, L);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

static double kn_shape_sin(double th, double alpha)
{
    const double c = std::cos(th), sn = std::sin(th);
    const double f1 = alpha * (1.0 - c), f2 = 1.0 + c * c, p = 1.0 + f1;
    return f2 / p / p * (1.0 + f1 * f1 / f2 / p) * sn;
}

static double kn_shape_sin_prime(double th, double alpha)
{
    const double c = std::cos(th), s = std::sin(th), om = 1.0 - c, p = 1.0 + alpha * om;
    const double g = (1.0 + c * c) / (p * p) + alpha * alpha * om * om / (p * p * p);
    const double gp = 2.0 * c / (p * p) + 2.0 * alpha * (1.0 + c * c) / (p * p * p) -
                      2.0 * alpha * alpha * om / (p * p * p) + 3.0 * alpha * alpha * alpha * om * om / (p * p * p * p);
    return c * g - s * s * gp;
}

void kn_table_build(double e0, double* tab)
{
    const int N = kKnTable;
    const double alpha = e0 / 511.0, hc = 3.14159265358979323846 / N, h = (double)0.01f;
    static const double xg[4] = {0.1834346424956498, 0.5255324099163290, 0.7966664774136267, 0.9602898564975363};
    static const double wg[4] = {0.3626837833783620, 0.3137066458778873, 0.2223810344533745, 0.1012285362903763};
    struct Node { double y[3], d[3]; };                    // G, U, V and their derivatives
    Node prev{};
    double G = 0.0;
    for (int i = 0; i <= N; ++i) {
        const double th = i * hc;
        if (i > 0) {                       // exact-to-rounding 8-point Gauss-Legendre per cell
            const double mid = th - 0.5 * hc, half = 0.5 * hc;
            double acc = 0.0;
            for (int k = 0; k < 4; ++k)
                acc += wg[k] * (kn_shape_sin(mid - half * xg[k], alpha) + kn_shape_sin(mid + half * xg[k], alpha));
            G += half * acc;
        }
        const double F = kn_shape_sin(th, alpha), P = kn_shape_sin_prime(th, alpha), eps = 1e-4;
        const double Q = (kn_shape_sin_prime(th + eps, alpha) - kn_shape_sin_prime(th - eps, alpha)) / (2.0 * eps);
        const Node now{{G, G + 0.5 * h * F + h * h / 12.0 * P, G - 0.5 * h * F + h * h / 12.0 * P},
                       {F, F + 0.5 * h * P + h * h / 12.0 * Q, F - 0.5 * h * P + h * h / 12.0 * Q}};
        for (int q = 0; q < 3 && i > 0; ++q) {             // the cell's cubic Hermite polynomial
            double* c = tab + 4 * N * q + 4 * (i - 1);
            const double dy = now.y[q] - prev.y[q], d0 = hc * prev.d[q], d1 = hc * now.d[q];
            c[0] = prev.y[q];
            c[1] = d0;
            c[2] = 3.0 * dy - 2.0 * d0 - d1;
            c[3] = d0 + d1 - 2.0 * dy;
        }
        prev = now;
    }
    tab[kKnTotal] = G;
}

double kn_normalisation(double e0)
{
    const float step = 0.01f;
    const int n = (int)((float)3.14159265358979323846 / step);
    const double alpha = e0 / 511.0;
    double sum = 0.0;
    for (int i = 0; i <= n; ++i) {
        const double th = (double)((float)i * step);
        const double c = std::cos(th), sn = std::sin(th);
        const double f1 = alpha * (1.0 - c), f2 = 1.0 + c * c, p = 1.0 + f1;
        sum += f2 / p / p * (1.0 + f1 * f1 / f2 / p) * sn * (double)step;
    }
    return sum;
}

}  // namespace sysmat
