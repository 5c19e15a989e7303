// The photoelectric element in the reference's float program (PESysMatGen.cu:951-1364), with its
// own 8 x 16 x 8 sub-elements and voxel centre (pe_element_ref) or any division and source points
// (pe_element_sampled), included by pe.cu inside its anonymous namespace.
//
// One warp per element, in phases that each loop over rounds (a round: 32 rays, one per lane, to
// a compact patch of sub-elements; the reference division: 4 z x 4 x x 2 depth):
//   1. kept objects: a cheap slope filter, then the reference cone test on what is left; each
//      kept object's geometry goes into the warp's record array (build_kept);
//   2. masks: which kept objects meet which round's slope box (round_masks; one lane per object,
//      so what depends on the object alone is formed once and not once per round);
//   3. holes and layers: each ray's attenuation in the collimator, into ws.att;
//   4. crystals: the other crystals' attenuation, added to it in the reference's order;
//   5. self attenuation, absorption, solid angle: the ray's contribution;
//   6. the sum.
// Why phases: a warp scheduler's instruction cache holds about 8 KB (512 instructions; measured
// on B200 with straight-line multiply-add loops: 0.93-0.98 issues per cycle up to there, 0.5-0.65
// beyond).  One loop over rounds with the whole body in it ran at that second rate whatever was
// shortened in it; every phase's loop fits the first.
// The walks take two rounds at a time, for two independent chains per lane, and a block's warps start
// each element together, which keeps the warps of a scheduler in the same phase.
// Bound by instruction issue (DRAM moves a few MB per launch).  Crystals 1984..2015 x one plane of
// configuration 2: 82.7e3 warp instructions per element at 58 % of the issue slots in one loop,
// 48.1e3 at 68 % now, 36.9 -> 18.1 ms, every float the same.  Two blocks of 8 warps at 128
// registers: three blocks at 80 issue at 70 % but need 11 % more instructions (spills); one block
// of 16 warps is 2 % slower, 40 % on matrices of few elements.  Forming the hole terms of a ray only
// in rounds that have holes is 7 % slower (registers).
//
// The fused multiply-adds are written out: they are the ones that the compiler chose for the
// reference's own expressions, and which product of a sum of two is fused changes the last
// bit.  With them the distance to the sub-element (:1218-1219) and the length of the ray in the
// cylinder chord (:696) are the same float, and cos(theta) is the direction's y component.

constexpr int kPassRounds = 16;          // rounds per pass: half of an element
constexpr int kUnits = 192;              // record units of 32 B: a hole takes one, a crystal two
constexpr int kNear = 512;               // sampled form: objects near the bundle of any source point

struct RefWarp {
    static constexpr int units = kUnits;
    // kept objects in the reference's order.  Hole i at rec[2 i]: (x, z, voxel - x, voxel - z),
    // (y1, y2, R, mu); crystal i (of those kept) at rec[2 nh + 4 i]: (x, y, z, mu), (cos(-rot),
    // sin(-rot), w, t), (h, voxel in its frame), slope rectangle
    float4 rec[2 * kUnits];
    unsigned short id[kUnits];           // hole ids
    unsigned mask[kUnits / 32][32];      // per round: the kept objects that meet its slope box
    float4 box[32];                      // the rounds' slope boxes
    float reach[32];                     // and the largest slope length in each
    float att[kPassRounds * 32];         // [round][lane]: attenuation outside crystal d, then contribution
    float len[256];                      // hole length of the open layer (elements kept in several chunks)
    int cand[64];                        // build_kept: source positions awaiting the cone test
    unsigned short near[kNear];          // sampled form: objects near the ray bundle of any source point
    float4 inner[kMaxLayers];            // plate "through both faces" slope rectangles
    Elem elem;
    // per sub-element index along x (0..7), depth (8..23), z (24..31): its centre, centre - voxel,
    // lower face - voxel, upper face - voxel in crystal d's frame
    float4 sub[32];
};

struct RefSmem {
    Superset sup;
    RefWarp w[kWarps];
};

// Attenuation beyond which expf(-att) is 0: half the smallest float is exp(-103.97).
constexpr float kDark = 104.5f;

// What build_kept leaves: entries [0, nh) are holes, [nh, count) crystals; even: the holes share
// layer, cap planes and radius.
struct Kept {
    int count, nh;
    bool even;
};

// How a crystal is divided: this lane's sub-element in a round, sub-element centres, and the
// table rows (centre, centre - voxel, lower face - voxel, upper face - voxel) of an index
// (:1207-1217), given rf = RN(1 / f).  The products are rounded before the sums, as the reference's
// build rounds them.
__device__ __forceinline__ float sub_centre(int i, float f, float rf, float size)
{
    return __fadd_rn(-size / 2.0f, __fmul_rn(div_by((float)i + 0.5f, f, rf), size));
}

__device__ __forceinline__ float4 sub_row(int i, float f, float rf, float size, float p)
{
    const float c = sub_centre(i, f, rf, size);
    const float u1 = __fmul_rn(div_by((float)i, f, rf) - 0.5f, size);
    const float u2 = __fmul_rn(div_by((float)i + 1.0f, f, rf) - 0.5f, size);
    return make_float4(c, c - p, __fsub_rn(u1, p), __fsub_rn(u2, p));
}

// The reference's 8 x 16 x 8, rows kept in ws.sub.
struct RefDivision {
    static constexpr float fx = 8.0f, fy = 16.0f, fz = 8.0f;
    static constexpr int rays = 2;       // rounds that the walks take at a time
    __device__ __forceinline__ void indices(int r, int lane, int& ix, int& iy, int& iz) const
    {
        ix = 4 * ((r >> 3) & 1) + ((lane >> 1) & 3);
        iy = 2 * (r & 7) + (lane & 1);
        iz = 4 * (r >> 4) + (lane >> 3);
    }
    __device__ __forceinline__ bool dead(int, int) const { return false; }
    template <class W>
    __device__ __forceinline__ float3 centre(const W& ws, int ix, int iy, int iz) const
    {
        return make_float3(ws.sub[ix].x, ws.sub[8 + iy].x, ws.sub[24 + iz].x);
    }
    template <class W>
    __device__ __forceinline__ float4 row_x(const W& ws, int i) const { return ws.sub[i]; }
    template <class W>
    __device__ __forceinline__ float4 row_y(const W& ws, int i) const { return ws.sub[8 + i]; }
    template <class W>
    __device__ __forceinline__ float4 row_z(const W& ws, int i) const { return ws.sub[24 + i]; }
    // lane l's table row: x (l < 8), depth (l < 24), z
    __device__ __forceinline__ static float4 entry(const Elem& e, int lane)
    {
        const int i = lane < 8 ? lane : (lane < 24 ? lane - 8 : lane - 24);
        const bool depth = lane >= 8 && lane < 24;
        return sub_row(i, depth ? fy : fx, depth ? 1.0f / fy : 1.0f / fx, lane < 8 ? e.w : (lane < 24 ? e.t : e.h),
                       lane < 8 ? e.xIs : (lane < 24 ? e.yIs : e.zIs));
    }
};

// The reference division from round `base`.
struct RefDivisionAt : RefDivision {
    int base;
    __device__ __forceinline__ explicit RefDivisionAt(int b) : base(b) {}
    __device__ __forceinline__ void indices(int r, int lane, int& ix, int& iy, int& iz) const
    {
        RefDivision::indices(base + r, lane, ix, iy, iz);
    }
};

// nx x ny x nz (x, depth, z), 32 to a round in (z, depth, x) order, x fastest, from sub-element
// `base`; lanes past the end repeat the last one and are dead.  Every phase forms a ray's indices and
// centre again, so quotients share reciprocals: with IEEE and integer divisions there, elements of few
// rays and objects (48 x 4 crystals around 1024 voxels) took 0.84 ms at 2 x 8 x 2, 0.73 ms now.
struct AnyDivision {
    static constexpr int rays = 1;
    int nx, ny, n_sub, base;
    float fx, fy, fz, rx, ry, rz, rxy;   // the numbers, their reciprocals, and 1 / (nx ny)
    __device__ __forceinline__ AnyDivision(int nx_, int ny_, int nz_, int base_)
        : nx(nx_), ny(ny_), n_sub(nx_ * ny_ * nz_), base(base_), fx((float)nx_), fy((float)ny_), fz((float)nz_),
          rx(rcp_rn(fx)), ry(rcp_rn(fy)), rz(rcp_rn(fz)), rxy(rcp_rn(fx * fy))
    {
    }
    // (s + 1/2) / n is at least 1 / (2 n) from a whole number, and at most 4096 sub-elements keep the
    // rounding of the product below 5e-4 / n
    __device__ __forceinline__ void indices(int r, int lane, int& ix, int& iy, int& iz) const
    {
        const int s = min(base + 32 * r + lane, n_sub - 1);
        iz = (int)(((float)s + 0.5f) * rxy);
        const int rem = s - iz * (nx * ny);
        iy = (int)(((float)rem + 0.5f) * rx);
        ix = rem - iy * nx;
    }
    __device__ __forceinline__ bool dead(int r, int lane) const { return base + 32 * r + lane >= n_sub; }
    template <class W>
    __device__ __forceinline__ float3 centre(const W& ws, int ix, int iy, int iz) const
    {
        return make_float3(sub_centre(ix, fx, rx, ws.elem.w), sub_centre(iy, fy, ry, ws.elem.t),
                           sub_centre(iz, fz, rz, ws.elem.h));
    }
    template <class W>
    __device__ __forceinline__ float4 row_x(const W& ws, int i) const { return sub_row(i, fx, rx, ws.elem.w, ws.elem.xIs); }
    template <class W>
    __device__ __forceinline__ float4 row_y(const W& ws, int i) const { return sub_row(i, fy, ry, ws.elem.t, ws.elem.yIs); }
    template <class W>
    __device__ __forceinline__ float4 row_z(const W& ws, int i) const { return sub_row(i, fz, rz, ws.elem.h, ws.elem.zIs); }
};

// World position of the sub-element with centre (xDs, yDs, zDs) in crystal d's frame.
__device__ __forceinline__ void ray_end(const Elem& e, float xDs, float yDs, float zDs, float& xD, float& yD, float& zD)
{
    xD = e.xd + __fmaf_rn(xDs, e.cosr, -__fmul_rn(zDs, e.sinr));
    zD = e.zd + __fmaf_rn(zDs, e.cosr, __fmul_rn(xDs, e.sinr));
    yD = e.yd + yDs;
}

// x^2 + y^2 + z^2 as the reference's ray lengths round it.
__device__ __forceinline__ float norm2(float x, float y, float z)
{
    return __fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x)));
}

// Whether object i may meet the slope rectangle rd of crystal d (approximate reciprocals, within
// the rectangles' margins), seen from any source within (spread, spread, spread_z) of (xs, ys, zs);
// objects close to the source always may.
__device__ __forceinline__ bool near_bundle(const DevGeom& g, float xs, float ys, float zs, const float4& rd, int i,
                                            float spread = 0.0f, float spread_z = 0.0f)
{
    float x0, x1, z0, z1, y0, y1;
    if (i < g.n_holes) {
        const float4 a = __ldg(&g.hole.a[i]);
        const float r = __ldg(&g.hole.b[i].x);
        x0 = a.x - r, x1 = a.x + r, z0 = a.w - r, z1 = a.w + r, y0 = a.y, y1 = a.z;
    } else {
        const float4 p = __ldg(&g.cry.pos[i - g.n_holes]);
        const float4 s = __ldg(&g.cry.size[i - g.n_holes]);
        const float4 t = __ldg(&g.cry.trig[i - g.n_holes]);
        const float hx = 0.5f * (s.x * fabsf(t.x) + s.z * fabsf(t.y)), hz = 0.5f * (s.x * fabsf(t.y) + s.z * fabsf(t.x));
        x0 = p.x - hx, x1 = p.x + hx, z0 = p.z - hz, z1 = p.z + hz, y0 = p.y - 0.5f * s.y, y1 = p.y + 0.5f * s.y;
    }
    y0 -= ys + spread;
    y1 -= ys - spread;
    if (!(y0 >= kMinDepth) || !(y1 >= kMinDepth)) return true;
    const float r0 = rcp_approx(y0), r1 = rcp_approx(y1);
    x0 -= xs + spread, x1 -= xs - spread, z0 -= zs + spread_z, z1 -= zs - spread_z;
    return fminf(x0 * r0, x0 * r1) - kSlopeMargin <= rd.y && fmaxf(x1 * r0, x1 * r1) + kSlopeMargin >= rd.x &&
           fminf(z0 * r0, z0 * r1) - kSlopeMargin <= rd.w && fmaxf(z1 * r0, z1 * r1) + kSlopeMargin >= rd.z;
}

// Slope rectangle of crystal d's bounding cylinder from any source within (spread, spread, spread_z)
// of (xs, ys, zs); false when the crystal is too close to the sources for one.
__device__ __forceinline__ bool bundle_rect(const DevGeom& g, int d, float xs, float ys, float zs, float spread,
                                            float spread_z, float4& rd)
{
    const float4 P = __ldg(&g.cry.pos[d]), S = __ldg(&g.cry.size[d]);
    const float foot = 0.5f * sqrtf(S.x * S.x + S.z * S.z), rx = foot + spread, rz = foot + spread_z;
    const float y0 = P.y - 0.5f * S.y - ys - spread, y1 = P.y + 0.5f * S.y - ys + spread;
    if (!(y0 >= kMinDepth)) return false;
    const float r0 = 1.0f / y0, r1 = 1.0f / y1, x = P.x - xs, z = P.z - zs;
    rd = make_float4(fminf((x - rx) * r0, (x - rx) * r1) - kSlopeMargin, fmaxf((x + rx) * r0, (x + rx) * r1) + kSlopeMargin,
                     fminf((z - rz) * r0, (z - rz) * r1) - kSlopeMargin, fmaxf((z + rz) * r0, (z + rz) * r1) + kSlopeMargin);
    return true;
}

// Reference cone test of object i (:1120-1184).
__device__ __forceinline__ bool in_cone(const DevGeom& g, const Elem& e, int i)
{
    const float4 od = object_data(g, i);
    const float L = sqrtf((e.xI - od.x) * (e.xI - od.x) + (e.yI - od.y) * (e.yI - od.y) +
                          (e.zI - od.z) * (e.zI - od.z));
    const float crit = i < g.n_holes ? od.w / L : od.w / L / 2.0f;
    const float vx = (od.x - e.xI) / L, vy = (od.y - e.yI) / L, vz = (od.z - e.zI) / L;
    return sqrtf((vz - e.uz) * (vz - e.uz) + (vy - e.uy) * (vy - e.uy) + (vx - e.ux) * (vx - e.ux)) <=
           crit + e.crit_self;
}

// Kept objects of the element from source positions [cursor, n_src) of the ids src (the block's
// superset, say; nullptr: all objects), in order.  The slope filter leaves a few percent of the superset, so what
// passes it is queued and the cone test (two square roots and four divisions) runs on full
// groups of 32.  Stops before a group that would overflow the records; returns the position to
// go on from.
template <class W>
__device__ __forceinline__ int build_kept(const DevGeom& g, const unsigned short* src, W& ws, const Elem& e,
                                          int d, int cursor, int n_src, int lane, Kept& kept)
{
    const unsigned below = (1u << lane) - 1u;
    int n = 0, nh = 0, units = 0, queued = 0;
    bool even = true;
    float4 first = make_float4(0.0f, 0.0f, 0.0f, 0.0f);   // y1, y2, R, layer of the first kept hole
    while (true) {
        while (queued < 32 && cursor < n_src) {
            const int j = cursor + lane;
            bool maybe = false;
            if (j < n_src) {
                const int id = src ? src[j] : j;
                maybe = id - g.n_holes != d && (!e.filt || near_bundle(g, e.xI, e.yI, e.zI, e.rd, id));
            }
            const unsigned m = __ballot_sync(0xffffffffu, maybe);
            if (maybe) ws.cand[queued + __popc(m & below)] = j;
            queued += __popc(m);
            cursor += 32;
        }
        __syncwarp();
        if (queued == 0) break;
        const int take = queued < 32 ? queued : 32;
        int id = 0;
        bool keep = false;
        if (lane < take) {
            id = src ? src[ws.cand[lane]] : ws.cand[lane];
            keep = in_cone(g, e, id);
        }
        const bool hole = id < g.n_holes;
        const unsigned mh = __ballot_sync(0xffffffffu, keep && hole), mc = __ballot_sync(0xffffffffu, keep && !hole);
        const int need = __popc(mh) + 2 * __popc(mc);
        if (units + need > W::units) {
            cursor = ws.cand[0];
            break;
        }
        const int holes = nh + __popc(mh);                // no hole comes after a crystal
        float4 caps = first;
        if (keep && hole) {
            const float4 a = __ldg(&g.hole.a[id]);
            const float4 b = __ldg(&g.hole.b[id]);
            const int pos = nh + __popc(mh & below);
            ws.rec[2 * pos] = make_float4(a.x, a.w, e.xI - a.x, e.zI - a.w);
            ws.rec[2 * pos + 1] = make_float4(a.y, a.z, b.x, b.y);
            ws.id[pos] = (unsigned short)id;
            caps = make_float4(a.y, a.z, b.x, (float)layer_of_hole(g, id));
        } else if (keep) {
            const int o = id - g.n_holes;
            const float4 po = __ldg(&g.cry.pos[o]), so = __ldg(&g.cry.size[o]), to = __ldg(&g.cry.trig[o]);
            const float vx = e.xI - po.x, vz = e.zI - po.z;   // :1305-1307
            float4* r = &ws.rec[2 * holes + 4 * (n - nh + __popc(mc & below))];
            r[0] = make_float4(po.x, po.y, po.z, __ldg(&g.cry.mu[o].x));
            r[1] = make_float4(to.z, to.w, so.x, so.y);
            r[2] = make_float4(so.z, __fmaf_rn(vx, to.z, -__fmul_rn(vz, to.w)), e.yI - po.y,
                               __fmaf_rn(vx, to.w, __fmul_rn(vz, to.z)));
            r[3] = e.filt ? crystal_rect(po, so, to, e.xI, e.yI, e.zI) : open_rect();
        }
        if (nh == 0 && mh != 0u) {
            const int src = __ffs(mh) - 1;
            first.x = __shfl_sync(0xffffffffu, caps.x, src);
            first.y = __shfl_sync(0xffffffffu, caps.y, src);
            first.z = __shfl_sync(0xffffffffu, caps.z, src);
            first.w = __shfl_sync(0xffffffffu, caps.w, src);
            if (!(keep && hole)) caps = first;
        }
        even = even && __all_sync(0xffffffffu, caps.x == first.x && caps.y == first.y && caps.z == first.z &&
                                                   caps.w == first.w);
        n += __popc(mh) + __popc(mc);
        nh = holes;
        units += need;
        const int rest = queued - take;
        const int moved = lane < rest ? ws.cand[32 + lane] : 0;
        __syncwarp();
        if (lane < rest) ws.cand[lane] = moved;
        queued = rest;
        __syncwarp();
    }
    kept = Kept{n, nh, even};
    return cursor;
}

__device__ __forceinline__ float warp_min(float x)
{
    float y;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float warp_max(float x)
{
    float y;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
    return y;
}

// ws.box and ws.reach of the first n rounds, from the rays themselves.
template <class W, class Div>
__device__ __forceinline__ void ray_boxes(W& ws, const Div& dv, int n, int lane)
{
    const Elem& e = ws.elem;
    for (int r = 0; r < n; ++r) {
        int ix, iy, iz;
        dv.indices(r, lane, ix, iy, iz);
        const float3 q = dv.centre(ws, ix, iy, iz);
        float x, y, z;
        ray_end(e, q.x, q.y, q.z, x, y, z);
        const float rdy = e.filt ? rcp_approx(y - e.yI) : 0.0f;
        const float a = (x - e.xI) * rdy, b = (z - e.zI) * rdy;
        const float4 box = make_float4(warp_min(a), warp_max(a), warp_min(b), warp_max(b));
        if (lane == 0) {
            const float px = fmaxf(fabsf(box.x), fabsf(box.y)), pz = fmaxf(fabsf(box.z), fabsf(box.w));
            ws.box[r] = box;
            ws.reach[r] = sqrtf(px * px + pz * pz);
        }
    }
    __syncwarp();
}

// Slope boxes of the rounds (lane = round): the slopes of a box of points behind the voxel are
// extreme at its corners.  All zero when the rectangles are open.
__device__ __forceinline__ void round_boxes(RefWarp& ws, const Elem& e, int lane)
{
    float4 b = make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float x, y, z;
        ray_end(e, ws.sub[4 * ((lane >> 3) & 1) + 3 * (k & 1)].x, ws.sub[8 + 2 * (lane & 7) + ((k >> 1) & 1)].x,
                ws.sub[24 + 4 * (lane >> 4) + 3 * (k >> 2)].x, x, y, z);
        const float r = e.filt ? rcp_approx(y - e.yI) : 0.0f;
        const float a = (x - e.xI) * r, c = (z - e.zI) * r;
        b.x = fminf(b.x, a);
        b.y = fmaxf(b.y, a);
        b.z = fminf(b.z, c);
        b.w = fmaxf(b.w, c);
    }
    const float px = fmaxf(fabsf(b.x), fabsf(b.y)), pz = fmaxf(fabsf(b.z), fabsf(b.w));
    ws.box[lane] = b;
    ws.reach[lane] = sqrtf(px * px + pz * pz);
    __syncwarp();
}

// What a round's slope box is tested against: an object's slope rectangle and its shadow.  Seen
// from the voxel, a y-aligned object with centre offset C, footprint half axes a, b (a crystal) or
// radius R (a hole) meets a ray of slope p only if |C x p| <= |a x p| + |b x p| + R |p|.  Objects
// close to the voxel (open rectangles) meet every box, a default Shadow none.
struct Shadow {
    float4 rect = make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY);
    float cx = 0.0f, cz = 0.0f, ax = 0.0f, az = 0.0f, bx = 0.0f, bz = 0.0f, R = INFINITY;
    float sx = 1e-3f, sz = 1e-3f;        // extents that scale the box's half widths and the margin

    // a: x, y1, y2, z of the hole
    __device__ __forceinline__ void hole(const Elem& e, float4 a, float r)
    {
        rect = e.filt ? hole_rect(a, r, e.xI, e.yI, e.zI) : open_rect();
        if (isinf(rect.x)) return;
        cx = e.xI - a.x, cz = e.zI - a.w, R = r * 1.0001f;
        sx += fabsf(cx), sz += fabsf(cz);
    }
    // half axes (hw c, hw s) and (-hh s, hh c) of the crystal's footprint, its rectangle known
    __device__ __forceinline__ void crystal(const Elem& e, float4 known, float x, float z, float hw, float hh, float c,
                                            float s)
    {
        rect = known;
        if (isinf(rect.x)) return;
        cx = e.xI - x, cz = e.zI - z, R = 0.0f;
        ax = hw * c, az = hw * s, bx = -hh * s, bz = hh * c;
        sx += fabsf(cx) + fabsf(ax) + fabsf(bx), sz += fabsf(cz) + fabsf(az) + fabsf(bz);
    }
    __device__ __forceinline__ bool meets(const float4& box, float reach) const
    {
        const float mx = 0.5f * (box.x + box.y), mz = 0.5f * (box.z + box.w);
        const float ex = 0.5f * (box.y - box.x) + kSlopeMargin, ez = 0.5f * (box.w - box.z) + kSlopeMargin;
        const float far = fabsf(cx * mz - cz * mx) - fabsf(ax * mz - az * mx) - fabsf(bx * mz - bz * mx);
        return rects_overlap(rect, box) && !(far > sx * ez + sz * ex + R * reach);
    }
};

// ws.mask for rounds [r0, r1): the kept objects that meet each round's slope box.
template <class W>
__device__ __forceinline__ void round_masks(W& ws, const Elem& e, const Kept& k, int r0, int r1, int lane)
{
    for (int w = 0; w * 32 < k.count; ++w) {
        const int j = w * 32 + lane;
        Shadow s;
        if (j < k.nh) {
            const float4 A = ws.rec[2 * j], B = ws.rec[2 * j + 1];
            s.hole(e, make_float4(A.x, B.x, B.y, A.y), B.z);
        } else if (j < k.count) {
            const float4* r = &ws.rec[2 * k.nh + 4 * (j - k.nh)];
            const float4 A = r[0], B = r[1];
            s.crystal(e, r[3], A.x, A.z, 0.5f * B.z, 0.5f * r[2].x, B.x, -B.y);
        }
        unsigned mine = 0u;
        for (int r = r0; r < r1; ++r) {
            const unsigned m = __ballot_sync(0xffffffffu, s.meets(ws.box[r], ws.reach[r]));
            if (lane == r) mine = m;
        }
        if (lane >= r0 && lane < r1) ws.mask[w][lane] = mine;
    }
    __syncwarp();
}

// The set bits of the masks of rounds r and q (q = r: one round) between entries [j0, j1), in order.
struct Entries {
    const unsigned (*mask)[32];
    int r, q, w, w1, j0, j1;
    unsigned m;

    __device__ __forceinline__ Entries(const unsigned (*mask_)[32], int r_, int j0_, int j1_) : Entries(mask_, r_, r_, j0_, j1_)
    {
    }
    __device__ __forceinline__ Entries(const unsigned (*mask_)[32], int r_, int q_, int j0_, int j1_)
        : mask(mask_), r(r_), q(q_), j0(j0_), j1(j1_)
    {
        w = j0 >> 5;
        w1 = (j1 + 31) >> 5;
        m = w < w1 ? word() : 0u;
    }
    __device__ __forceinline__ unsigned word() const
    {
        unsigned x = mask[w][r] | mask[w][q];
        if (w == j0 >> 5) x &= 0xffffffffu << (j0 & 31);
        if (w == j1 >> 5) x &= (1u << (j1 & 31)) - 1u;
        return x;
    }
    __device__ __forceinline__ bool more()
    {
        while (m == 0u && w + 1 < w1) {
            ++w;
            m = word();
        }
        return m != 0u;
    }
    __device__ __forceinline__ int take()
    {
        const int j = w * 32 + __ffs(m) - 1;
        m &= m - 1u;
        return j;
    }
};

// Attenuation of one ray so far: accumulated mu L, and the open layer with its hole length.
struct Walk {
    float att, len;
    int lay;
};

// A ray from the voxel in the walk over holes: the terms of the reference cylinder chord
// (:688-799) that depend only on the ray, and those of the cap planes at hand.
struct HoleRay {
    float tio, kx, ky, kz, iky, rx, rz, kk, ikk;
    float ta, tb, xl, xr, zl, zr;
    float full;                  // chord of a ray inside the hole at both caps
    bool steep;                  // |ky| large enough for div_by
};

__device__ __forceinline__ void hole_ray_init(HoleRay& c, float dx, float dy, float dz)
{
    c.tio = sqrt_mid(norm2(dx, dy, dz));
    const float itio = rcp_rn(c.tio);
    c.kx = div_by(dx, c.tio, itio);
    c.ky = div_by(dy, c.tio, itio);
    c.kz = div_by(dz, c.tio, itio);
    c.iky = rcp_rn(c.ky);
    c.steep = fabsf(c.ky) >= kMinDivisor;
    c.rx = div_by(c.kx, c.ky, c.iky);
    c.rz = div_by(c.kz, c.ky, c.iky);
    if (!c.steep) {              // a ray along the plates
        c.rx = c.kx / c.ky;
        c.rz = c.kz / c.ky;
    }
    c.kk = __fmaf_rn(c.kx, c.kx, __fmul_rn(c.kz, c.kz));
    c.ikk = rcp_rn(c.kk);
}

__device__ __forceinline__ void hole_ray_caps(HoleRay& c, const Elem& e, float y1, float y2)
{
    const float u1 = y1 - e.yI, u2 = y2 - e.yI;
    c.xl = __fmaf_rn(c.rx, u1, e.xI);
    c.xr = __fmaf_rn(c.rx, u2, e.xI);
    c.zl = __fmaf_rn(c.rz, u1, e.zI);
    c.zr = __fmaf_rn(c.rz, u2, e.zI);
    c.ta = div_by(u1, c.ky, c.iky);
    c.tb = div_by(u2, c.ky, c.iky);
    if (!c.steep) {
        c.ta = u1 / c.ky;
        c.tb = u2 / c.ky;
    }
    c.full = fabsf(c.tb - c.ta);
    if (c.ta <= 0.0001f || c.tb <= 0.0001f || c.ta >= c.tio || c.tb >= c.tio) c.full = 0.0f;
    // closer than 0.001: the reference returns 0; with both cap parameters 0 every case below does
    if (fabsf(y1 - y2) < 0.001f) c.ta = c.tb = c.full = 0.0f;
}

// Chord of hole A = (x, z, voxel - x, voxel - z) of radius r; kr = RN(kk r), r2 = RN(r^2).
// Straight-line: the reference's four cap/side cases are selects (a warp whose lanes meet
// different cases runs it once, and two holes interleave).
struct ChordParts {
    bool fl, fr;                 // inside the hole at the front and back cap
    float cross, sd;             // the cross term and the root of the discriminant
};

__device__ __forceinline__ float hole_chord(const HoleRay& c, const float4& A, float r, float kr, float r2,
                                            ChordParts* parts = nullptr)
{
    const float dxl = c.xl - A.x, dzl = c.zl - A.y, dxr = c.xr - A.x, dzr = c.zr - A.y;
    const bool fl = __fmaf_rn(dzl, dzl, __fmul_rn(dxl, dxl)) <= r2;
    const bool fr = __fmaf_rn(dzr, dzr, __fmul_rn(dxr, dxr)) <= r2;
    const float cross = __fmaf_rn(c.kx, A.w, -__fmul_rn(c.kz, A.z));
    const float disc = __fmaf_rn(kr, r, -__fmul_rn(cross, cross));
    const bool meets = disc > 0.00001f;
    const float sd = sqrt_mid(meets ? disc : 1.0f);
    const float b = -__fmaf_rn(c.kx, A.z, __fmul_rn(c.kz, A.w));
    const float t1 = div_by(b - sd, c.kk, c.ikk), t2 = div_by(b + sd, c.kk, c.ikk);
    const float ea = fl ? c.ta : t1, eb = fr ? c.tb : t2;
    const bool ok = meets && (fl || fr || (t1 >= c.ta && t2 <= c.tb)) &&
                    !(eb <= 0.0001f || ea <= 0.0001f || eb >= c.tio || ea >= c.tio);
    if (parts) *parts = ChordParts{fl, fr, cross, sd};
    return (fl && fr) ? c.full : (ok ? eb - ea : 0.0f);
}

__device__ __forceinline__ void close_layers_ref(const DevGeom& g, Walk& s, int upto, const HoleRay& c)
{
    while (s.lay < upto) {                                    // :1281-1284
        float lcol = div_by(g.layer[s.lay].thickness, c.ky, c.iky);
        if (!c.steep) lcol = g.layer[s.lay].thickness / c.ky;
        if ((lcol - s.len) >= 0.00001f) s.att = __fmaf_rn(g.layer[s.lay].mu_total, lcol - s.len, s.att);
        s.len = 0.0f;
        ++s.lay;
    }
}

// Holes and layers along the rays of rounds [r0, r1), Div::rays rounds at a time.  first: the rays
// start here (plate penalty, :1240-1254), otherwise they go on from ws.att / ws.len in layer lay0;
// at the end the layers below lay1 are closed.  A ray that the plate penalty blocked (every
// mu >= 0) gets infinite attenuation.  Every branch on an entry is uniform across the warp, and a
// ray that misses a hole adds an exact zero.  A lane always has two independent chords in hand
// (the serial chain of one leaves issue slots idle): one hole for the rays of two rounds, or with
// one round and EVEN two holes for its ray.  EVEN (all kept holes alike, the usual collimator): the
// cap terms are formed once per ray.
template <bool COUNT, bool ELL, bool EVEN, class Div>
__device__ __forceinline__ void walk_holes(const DevGeom& g, RefWarp& ws, const Div& dv, int nh, int r0, int r1, bool first,
                                           int lay0, int lay1, bool carry, int lane, int& n_hits, int& n_evals,
                                           int& n_blocked)
{
    constexpr int NR = Div::rays;
    const Elem& e = ws.elem;
    for (int r = r0; r < r1; r += NR) {
        HoleRay c[NR];
        Walk s[NR];
        bool skip[NR];
        float3 end[ELL ? NR : 1];
#pragma unroll
        for (int n = 0; n < NR; ++n) {
            int ix, iy, iz;
            dv.indices(r + n, lane, ix, iy, iz);
            const float3 q = dv.centre(ws, ix, iy, iz);
            float xD, yD, zD;
            ray_end(e, q.x, q.y, q.z, xD, yD, zD);
            if constexpr (ELL) end[n] = make_float3(xD, yD, zD);
            hole_ray_init(c[n], xD - e.xI, yD - e.yI, zD - e.zI);
            s[n] = Walk{0.0f, 0.0f, lay0};
            if (first) {
                const float rdy = e.filt ? rcp_approx(yD - e.yI) : 0.0f;             // open rectangles: slope 0
                skip[n] = plate_penalty(g, ws.inner, e, xD, yD, zD, (xD - e.xI) * rdy, (zD - e.zI) * rdy, s[n].att) &&
                          g.nonneg_mu;
                skip[n] = skip[n] || dv.dead(r + n, lane);
                if constexpr (COUNT) n_blocked += skip[n];
            } else {
                s[n].att = ws.att[((r + n) & (kPassRounds - 1)) * 32 + lane];
                s[n].len = ws.len[((r + n) & 7) * 32 + lane];
                skip[n] = isinf(s[n].att);
            }
        }
        Entries it(ws.mask, r, r + NR - 1, 0, nh);
        if (EVEN && it.more()) {
            const float4 B = ws.rec[1];
            const int m = layer_of_hole(g, ws.id[0]);
            const float r2 = __fmul_rn(B.z, B.z);
            float kr[NR];
#pragma unroll
            for (int n = 0; n < NR; ++n) {
                if (m != s[n].lay) close_layers_ref(g, s[n], m, c[n]);
                hole_ray_caps(c[n], e, B.x, B.y);
                kr[n] = __fmul_rn(c[n].kk, B.z);
            }
            do {
                const int j = it.take();
                const float4 A = ws.rec[2 * j];
                const float mu = ws.rec[2 * j + 1].w;
                if constexpr (NR == 2) {
                    float tmp[NR];
#pragma unroll
                    for (int n = 0; n < NR; ++n) tmp[n] = hole_chord(c[n], A, B.z, kr[n], r2);
#pragma unroll
                    for (int n = 0; n < NR; ++n) {
                        s[n].len = s[n].len + tmp[n];                             // :1276-1278
                        s[n].att = __fmaf_rn(mu, tmp[n], s[n].att);
                        if constexpr (COUNT) {
                            if (!skip[n]) n_hits += tmp[n] != 0.0f, ++n_evals;
                        }
                    }
                } else {
                    const bool pair = it.m != 0u;
                    const int j2 = pair ? it.take() : j;
                    const float4 A2 = ws.rec[2 * j2];
                    const float mu2 = ws.rec[2 * j2 + 1].w;
                    const float tmp = hole_chord(c[0], A, B.z, kr[0], r2);
                    const float two = hole_chord(c[0], A2, B.z, kr[0], r2);
                    const float tmp2 = pair ? two : 0.0f;
                    s[0].len = s[0].len + tmp;                                    // :1276-1278
                    s[0].att = __fmaf_rn(mu, tmp, s[0].att);
                    s[0].len = s[0].len + tmp2;
                    s[0].att = __fmaf_rn(mu2, tmp2, s[0].att);
                }
            } while (it.more());
        }
        if (!EVEN) {
            float y1 = NAN, y2 = NAN;                     // cap planes at hand (NaN never compares equal)
            while (it.more()) {
                const int j = it.take();
                const float4 A = ws.rec[2 * j], B = ws.rec[2 * j + 1];
                const int id = ws.id[j], m = layer_of_hole(g, id);
                float4 S = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if constexpr (ELL) {
                    if (g.hole_shape) S = __ldg(&g.hole_shape[id]);
                }
                const bool ell = ELL && S.x > 0.0f;
                const bool caps = !ell && !(B.x == y1 && B.y == y2);
                if (caps) {
                    y1 = B.x;
                    y2 = B.y;
                }
#pragma unroll
                for (int n = 0; n < NR; ++n) {
                    if (m != s[n].lay) close_layers_ref(g, s[n], m, c[n]);
                    float tmp = 0.0f;
                    if (ell) {                                                    // elliptical hole
                        const float3 q = end[ELL ? n : 0];
                        if (!skip[n])
                            tmp = ell_chord(e.xI, e.yI, e.zI, q.x, q.y, q.z, A.x, B.x, B.y, A.y, S.x, S.y, S.z, S.w);
                    } else {
                        if (caps) hole_ray_caps(c[n], e, y1, y2);
                        tmp = hole_chord(c[n], A, B.z, __fmul_rn(c[n].kk, B.z), __fmul_rn(B.z, B.z));
                    }
                    s[n].len = s[n].len + tmp;                                    // :1276-1278
                    s[n].att = __fmaf_rn(B.w, tmp, s[n].att);
                    if constexpr (COUNT) {
                        if (!skip[n]) n_hits += tmp != 0.0f, ++n_evals;
                    }
                }
            }
        }
#pragma unroll
        for (int n = 0; n < NR; ++n) {
            if (s[n].lay < lay1) close_layers_ref(g, s[n], lay1, c[n]);
            // past kDark the contribution is exactly 0 whatever follows (every mu >= 0): as if blocked
            skip[n] = skip[n] || (s[n].att > kDark && g.nonneg_mu);
            ws.att[((r + n) & (kPassRounds - 1)) * 32 + lane] = skip[n] ? INFINITY : s[n].att;
            if (carry) ws.len[((r + n) & 7) * 32 + lane] = s[n].len;
        }
    }
}

// Full-crossing chord of the segment voxel -> sub-element in a crystal's frame (box_chord of the
// centred box w x t x h; a = the voxel, b = the sub-element): the interval tests of box_chord
// as selects on the final interval (an interval that is empty after two axes stays empty).
__device__ __forceinline__ float crystal_chord(float xa, float ya, float za, float xb, float yb, float zb, float w,
                                               float t, float h)
{
    const float dx = xb - xa, dy = yb - ya, dz = zb - za;
    if (fabsf(dx) < kEps || fabsf(dy) < kEps || fabsf(dz) < kEps)
        return box_chord_parallel(xa, ya, za, xb, yb, zb, -0.5f * w, -0.5f * t, -0.5f * h, 0.5f * w, 0.5f * t,
                                  0.5f * h, 0);
    const float tio = sqrt_mid(norm2(dy, dx, dz));
    const float ix = div_rn(tio, dx), iy = div_rn(tio, dy), iz = div_rn(tio, dz);
    const float x0 = (-0.5f * w - xa) * ix, x1 = (0.5f * w - xa) * ix;
    const float y0 = (-0.5f * t - ya) * iy, y1 = (0.5f * t - ya) * iy;
    const float z0 = (-0.5f * h - za) * iz, z1 = (0.5f * h - za) * iz;
    const float tmin = fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fminf(z0, z1));
    const float tmax = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(z0, z1));
    const bool out = (tmax - tmin) < kEps || tmin >= tio || tmax >= tio || tmin <= kEps || tmax <= kEps;
    return out ? 0.0f : tmax - tmin;
}

// Chord of the ray to (xD, yD, zD) in the crystal recorded at rec (0 for a lane it does not concern),
// and the crystal's mu.
__device__ __forceinline__ float record_chord(const float4* rec, float xD, float yD, float zD, bool in, float& mu)
{
    const float4 A = rec[0], B = rec[1], C = rec[2];
    const float vx = xD - A.x, vz = zD - A.z;                             // :1318-1320
    const float xb = __fmaf_rn(vx, B.x, -__fmul_rn(vz, B.y)), zb = __fmaf_rn(vz, B.x, __fmul_rn(vx, B.y));
    mu = A.w;
    return in ? crystal_chord(C.y, C.z, C.w, xb, yD - A.y, zb, B.z, B.w, C.x) : 0.0f;
}

// Other crystals along the rays of rounds [r0, r1), Div::rays rounds at a time: kept entries [nh,
// count), added to ws.att in the reference's order (:1290-1325).
template <bool COUNT, class Div>
__device__ __forceinline__ void walk_crystals(const DevGeom& g, RefWarp& ws, const Div& dv, int nh, int count, int r0, int r1,
                                              int lane, int& n_hits, int& n_evals)
{
    constexpr int NR = Div::rays;
    const Elem& e = ws.elem;
    for (int r = r0; r < r1; r += NR) {
        Entries it(ws.mask, r, r + NR - 1, nh, count);
        if (!it.more()) continue;
        float xD[NR], yD[NR], zD[NR], sa_a[NR], sa_b[NR], att[NR];
#pragma unroll
        for (int n = 0; n < NR; ++n) {
            int ix, iy, iz;
            dv.indices(r + n, lane, ix, iy, iz);
            const float3 q = dv.centre(ws, ix, iy, iz);
            ray_end(e, q.x, q.y, q.z, xD[n], yD[n], zD[n]);
            const float rdy = e.filt ? rcp_approx(yD[n] - e.yI) : 0.0f;
            sa_a[n] = (xD[n] - e.xI) * rdy, sa_b[n] = (zD[n] - e.zI) * rdy;
            att[n] = ws.att[((r + n) & (kPassRounds - 1)) * 32 + lane];
        }
        do {
            const float4* rec = &ws.rec[2 * nh + 4 * (it.take() - nh)];
            const float4 rect = rec[3];
            bool in[NR], any = false;
#pragma unroll
            for (int n = 0; n < NR; ++n) {
                in[n] = !isinf(att[n]) && in_rect(rect, sa_a[n], sa_b[n]);
                any = any || in[n];
            }
            if (!__any_sync(0xffffffffu, any)) continue;
            float la[NR], mu;
#pragma unroll
            for (int n = 0; n < NR; ++n) la[n] = record_chord(rec, xD[n], yD[n], zD[n], in[n], mu);
#pragma unroll
            for (int n = 0; n < NR; ++n) {
                att[n] = __fmaf_rn(la[n], mu, att[n]);
                if constexpr (COUNT) n_hits += (la[n] != 0.0f), n_evals += in[n];
            }
        } while (it.more());
#pragma unroll
        for (int n = 0; n < NR; ++n) ws.att[((r + n) & (kPassRounds - 1)) * 32 + lane] = att[n];
    }
}

// Length of the interval [tmin, tmax] between the voxel and the end point (tio): the end of
// box_chord_inside as selects.
__device__ __forceinline__ float inside_length(float tmin, float tmax, float tio)
{
    const bool out = (tmax - tmin) < kEps || tmin >= tio || tmax <= kEps;
    const float len = fminf(tmax, tio) - (tmin > kEps ? tmin : 0.0f);
    return out ? 0.0f : len;
}

// Both box chords of finish_ray when the ray is parallel to an axis within eps (the reference's
// slow cases): inside = the crystal and the sub-element boxes to the sub-element's centre,
// otherwise the sub-element box along the extended ray to (xo, yo, zo).
static __device__ __noinline__ float2 finish_parallel(float xi, float yi, float zi, float xo, float yo, float zo, float w,
                                                      float t, float h, int ix, int iy, int iz, float fx, float fy,
                                                      float fz, int inside)
{
    const float ux1 = ((float)ix / fx - 0.5f) * w, ux2 = (((float)ix + 1.0f) / fx - 0.5f) * w;
    const float uy1 = ((float)iy / fy - 0.5f) * t, uy2 = (((float)iy + 1.0f) / fy - 0.5f) * t;
    const float uz1 = ((float)iz / fz - 0.5f) * h, uz2 = (((float)iz + 1.0f) / fz - 0.5f) * h;
    float2 l = make_float2(0.0f, 0.0f);
    if (!inside) {
        l.x = box_chord_parallel(xi, yi, zi, xo, yo, zo, ux1, uy1, uz1, ux2, uy2, uz2, 0);
    } else if (!(fabsf(yo - yi) < 0.001f)) {
        l.x = box_chord_parallel(xi, yi, zi, xo, yo, zo, -w / 2.0f, -t / 2.0f, -h / 2.0f, w / 2.0f, t / 2.0f, h / 2.0f, 1);
        l.y = box_chord_parallel(xi, yi, zi, xo, yo, zo, ux1, uy1, uz1, ux2, uy2, uz2, 1);
    }
    return l;
}

// What crystal d makes of a ray to its sub-element (ix, iy, iz) (:1223-1231, :1329-1357): the length
// of crystal d before the sub-element, the absorption chord and the solid angle.
struct RayEnd {
    float self, labs, sa;
};

template <class W, class Div>
__device__ __forceinline__ RayEnd ray_end_terms(const W& ws, const Div& dv, int ix, int iy, int iz)
{
    const Elem& e = ws.elem;
    const float4 X = dv.row_x(ws, ix), Y = dv.row_y(ws, iy), Z = dv.row_z(ws, iz);
    const float w = e.w, t = e.t, h = e.h;
    float l1, l2;
    if (fabsf(X.y) < kEps || fabsf(Y.y) < kEps || fabsf(Z.y) < kEps) {
        const float2 l = finish_parallel(e.xIs, e.yIs, e.zIs, X.x, Y.x, Z.x, w, t, h, ix, iy, iz, dv.fx, dv.fy, dv.fz, 1);
        l1 = l.x;
        l2 = l.y;
    } else {
        const float tio = sqrt_mid(norm2(X.y, Y.y, Z.y));
        const float rx = div_rn(tio, X.y), ry = div_rn(tio, Y.y), rz = div_rn(tio, Z.y);
        float a = (-w / 2.0f - e.xIs) * rx, b = (w / 2.0f - e.xIs) * rx;
        float tmin = fminf(a, b), tmax = fmaxf(a, b);
        a = (-t / 2.0f - e.yIs) * ry, b = (t / 2.0f - e.yIs) * ry;
        tmin = fmaxf(tmin, fminf(a, b)), tmax = fminf(tmax, fmaxf(a, b));
        a = (-h / 2.0f - e.zIs) * rz, b = (h / 2.0f - e.zIs) * rz;
        tmin = fmaxf(tmin, fminf(a, b)), tmax = fminf(tmax, fmaxf(a, b));
        l1 = inside_length(tmin, tmax, tio);
        a = X.z * rx, b = X.w * rx;
        tmin = fminf(a, b), tmax = fmaxf(a, b);
        a = Y.z * ry, b = Y.w * ry;
        tmin = fmaxf(tmin, fminf(a, b)), tmax = fminf(tmax, fmaxf(a, b));
        a = Z.z * rz, b = Z.w * rz;
        tmin = fmaxf(tmin, fminf(a, b)), tmax = fminf(tmax, fmaxf(a, b));
        l2 = inside_length(tmin, tmax, tio);
    }
    float xD, yD, zD;
    ray_end(e, X.x, Y.x, Z.x, xD, yD, zD);
    const float dsq = norm2(xD - e.xI, yD - e.yI, zD - e.zI);
    const float sq = sqrt_mid(dsq), isq = rcp_rn(sq);
    // absorption: the chord of the ray extended 1000 mm past the sub-element (:1352-1357)
    const float xt = X.x + div_by(1000.0f * X.y, sq, isq);
    const float yt = Y.x + div_by(1000.0f * Y.y, sq, isq);
    const float zt = Z.x + div_by(1000.0f * Z.y, sq, isq);
    const float dx = xt - e.xIs, dy = yt - e.yIs, dz = zt - e.zIs;
    float labs;
    if (fabsf(dx) < kEps || fabsf(dy) < kEps || fabsf(dz) < kEps) {
        labs = finish_parallel(e.xIs, e.yIs, e.zIs, xt, yt, zt, w, t, h, ix, iy, iz, dv.fx, dv.fy, dv.fz, 0).x;
    } else {
        const float tio = sqrt_mid(norm2(dy, dx, dz));
        const float rx = div_rn(tio, dx), ry = div_rn(tio, dy), rz = div_rn(tio, dz);
        float a = X.z * rx, b = X.w * rx;
        float tmin = fminf(a, b), tmax = fmaxf(a, b);
        a = Y.z * ry, b = Y.w * ry;
        tmin = fmaxf(tmin, fminf(a, b)), tmax = fminf(tmax, fmaxf(a, b));
        a = Z.z * rz, b = Z.w * rz;
        tmin = fmaxf(tmin, fminf(a, b)), tmax = fminf(tmax, fmaxf(a, b));
        const bool out = (tmax - tmin) < kEps || tmin >= tio || tmax >= tio || tmin <= kEps || tmax <= kEps;
        labs = out ? 0.0f : tmax - tmin;
    }
    // solid angle in double, as the reference's 4*M_PI promotion makes it: the largest of three
    // exact double products times one reciprocal, rounded once (rounding keeps the order, so this
    // is the largest of the three rounded values; the reciprocal in place of the reference's
    // divisions rounds identically except in double-rounding ties)
    const double rq = 1.0 / ((4.0 * 3.14159265358979323846) * (double)dsq * (double)sq);
    const float ax = t * h / dv.fz / dv.fy, az = w * t / dv.fx / dv.fy, ay = w * h / dv.fx / dv.fz;
    const double px = (double)ax * (double)fabsf((xD - e.xI) * e.cosr - (zD - e.zI) * e.sinr);
    const double pz = (double)az * (double)fabsf((xD - e.xI) * e.sinr + (zD - e.zI) * e.cosr);
    const double py = (double)ay * (double)fabsf(yD - e.yI);
    const double pm = px >= py ? (px >= pz ? px : pz) : (py >= pz ? py : pz);
    const float sa = (float)(pm * rq);
    return RayEnd{l1 - l2, labs, sa};
}

// Contribution of sub-element (ix, iy, iz), given the attenuation outside crystal d.
template <class Div>
__device__ __forceinline__ float finish_ray(const RefWarp& ws, const Div& dv, int ix, int iy, int iz, float att)
{
    const Elem& e = ws.elem;
    const RayEnd q = ray_end_terms(ws, dv, ix, iy, iz);
    const float eff = 1.0f * expf(-__fmaf_rn(q.self, e.mu_t, att));
    const float absf = div_by((1.0f - expf(-q.labs * e.mu_t)) * e.mu_pe, e.mu_t, e.imu_t);
    return eff * q.sa * absf;
}

// Work counts of one lane (COUNT instances).
struct Counts {
    int hole_hits = 0, cry_hits = 0, blocked = 0, hole_evals = 0, cry_evals = 0;
    long long entries = 0;
};

// Attenuation outside crystal d of the rays of rounds [r0, r1), into ws.att.  single: the kept
// objects k are the element's and ws.mask holds the rounds'; otherwise the list is taken in
// chunks, each ray's open-layer length carried in ws.len.
template <bool COUNT, bool ELL, class Div>
__device__ __forceinline__ void attenuation_pass(const DevGeom& g, RefWarp& ws, const Div& dv, const unsigned short* src,
                                                 int n_src, int d, bool single, int r0, int r1, int lane, int cursor,
                                                 Kept& k, Counts& n)
{
    const Elem& e = ws.elem;
    int lay = 0;
    for (bool first = true;; first = false) {
        if (!single) {
            cursor = build_kept(g, src, ws, e, d, first ? 0 : cursor, n_src, lane, k);
            round_masks(ws, e, k, r0, r1, lane);
        }
        const bool last = cursor >= n_src;
        // this chunk ends the holes when crystals follow or no object does
        const int lay1 = last || k.nh < k.count ? g.n_layers : (k.nh > 0 ? layer_of_hole(g, ws.id[k.nh - 1]) : lay);
        if (Div::rays == 1 && g.n_layers == 0) {         // no collimator: no hole, layer or plate
            for (int r = r0; r < r1 && first; ++r)
                ws.att[(r & (kPassRounds - 1)) * 32 + lane] = dv.dead(r, lane) ? INFINITY : 0.0f;
        } else if (!ELL && k.even)
            walk_holes<COUNT, ELL, true>(g, ws, dv, k.nh, r0, r1, first, lay, lay1, !single, lane, n.hole_hits,
                                         n.hole_evals, n.blocked);
        else
            walk_holes<COUNT, ELL, false>(g, ws, dv, k.nh, r0, r1, first, lay, lay1, !single, lane, n.hole_hits,
                                          n.hole_evals, n.blocked);
        lay = lay1;
        if (k.nh < k.count)
            walk_crystals<COUNT>(g, ws, dv, k.nh, k.count, r0, r1, lane, n.cry_hits, n.cry_evals);
        if constexpr (COUNT) {
            for (int r = r0; r < r1; ++r)
                for (int w = 0; w * 32 < k.count; ++w) n.entries += __popc(ws.mask[w][r]);
        }
        __syncwarp();
        if (last) break;
    }
}

// Element (d, v): the reference's float chain over sub-elements in its order (MODE 0) or an FP64
// sum (MODE 1).
template <int MODE, bool COUNT, bool ELL>
__device__ double pe_element_ref(const DevGeom& g, const Superset& sup, RefWarp& ws, int d, long long v, float cr,
                                 float sr, int lane, unsigned long long* counters)
{
    const unsigned short* src = sup.s_count >= 0 ? sup.sid : nullptr;
    const int n_src = src ? sup.s_count : g.n_holes + g.n_det;
    const RefDivision dv;
    int cursor;
    Kept k;
    {
        Elem el;
        if (!init_element(g, ws.inner, d, v, cr, sr, lane, el)) return 0.0;
        if (lane == 0) ws.elem = el;
        ws.sub[lane] = RefDivision::entry(el, lane);
        cursor = build_kept(g, src, ws, el, d, 0, n_src, lane, k);   // ends in a __syncwarp
    }
    const Elem& e = ws.elem;
    round_boxes(ws, e, lane);
    Counts n;
    const bool single = cursor >= n_src;
    if (single) round_masks(ws, e, k, 0, 32, lane);
    // an element kept in several chunks goes a quarter at a time, so that the rays' open-layer
    // lengths fit ws.len
    const int per = single ? kPassRounds : 8;
    float chain = 0.0f;
    double dacc = 0.0;
    for (int q0 = 0; q0 < 32; q0 += kPassRounds) {
        for (int r0 = q0; r0 < q0 + kPassRounds; r0 += per) {
            attenuation_pass<COUNT, ELL>(g, ws, dv, src, n_src, d, single, r0, r0 + per, lane, cursor, k, n);
        }
        for (int r = q0; r < q0 + kPassRounds; ++r) {
            int ix, iy, iz;
            dv.indices(r, lane, ix, iy, iz);
            const float att = ws.att[(r & (kPassRounds - 1)) * 32 + lane];
            const float c = isinf(att) ? 0.0f : finish_ray(ws, dv, ix, iy, iz, att);
            if constexpr (MODE == 0) ws.att[(r & (kPassRounds - 1)) * 32 + lane] = c;
            else dacc += (double)c;
        }
        __syncwarp();
        if constexpr (MODE == 0) {
            for (int k = 0; k < 32; ++k) {        // (iz, ix): 16 depths each, two per round
                const float* c = &ws.att[((k >> 2) & 1) * 256 + (k >> 3) * 8 + (k & 3) * 2];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const float2 two = *reinterpret_cast<const float2*>(c + 32 * u);
                    chain = chain + two.x;
                    chain = chain + two.y;
                }
            }
            __syncwarp();
        }
    }
    if constexpr (COUNT) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            n.hole_hits += __shfl_xor_sync(0xffffffffu, n.hole_hits, off);
            n.cry_hits += __shfl_xor_sync(0xffffffffu, n.cry_hits, off);
            n.blocked += __shfl_xor_sync(0xffffffffu, n.blocked, off);
            n.hole_evals += __shfl_xor_sync(0xffffffffu, n.hole_evals, off);
            n.cry_evals += __shfl_xor_sync(0xffffffffu, n.cry_evals, off);
        }
        if (lane == 0) {
            atomicAdd(&counters[0], 1024ull);
            atomicAdd(&counters[1], (unsigned long long)n.hole_hits);
            atomicAdd(&counters[2], (unsigned long long)n.cry_hits);
            atomicAdd(&counters[3], 1ull);
            atomicAdd(&counters[4], (unsigned long long)n.blocked);
            atomicAdd(&counters[5], single ? 0ull : 1ull);                 // chunked elements
            atomicAdd(&counters[6], (unsigned long long)k.count);          // kept objects (last chunk)
            atomicAdd(&counters[7], (unsigned long long)n.entries);        // entries over all rounds
            atomicAdd(&counters[8], sup.s_count < 0 ? 1ull : 0ull);        // superset overflow
            atomicAdd(&counters[9], (unsigned long long)(sup.s_count < 0 ? 0 : sup.s_count));
            atomicAdd(&counters[10], (unsigned long long)n.hole_evals);
            atomicAdd(&counters[11], (unsigned long long)n.cry_evals);
        }
    }
    if constexpr (MODE == 0) {
        return chain;
    } else {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) dacc += __shfl_xor_sync(0xffffffffu, dacc, off);
        return dacc;
    }
}

// Element of the sampled form: the mean over the voxel's sx x sy x sz source points (centres of
// a grid over the voxel) of the reference's element with crystal d divided into nx x ny x nz
// sub-elements (x, depth, z), every contribution summed in FP64.  Each source point has its own
// cone test and kept objects, drawn from one list per voxel of the objects near the ray bundle of
// any source point (a few percent of the block's superset).  The configuration-2 sampling, 96
// crystals x 4608 voxels: 38.0 -> 16.7 ms, bound by instruction issue.  With 8 x 16 x 8 and 1 x 1 x 1 it runs
// pe_element_ref<1>'s float program, summed in another order.
template <bool ELL>
__device__ double pe_element_sampled(const DevGeom& g, const Superset& sup, RefWarp& ws, int d, long long v, float cr,
                                     float sr, int lane, const Sampling& sm)
{
    const int n_pts = sm.sx * sm.sy * sm.sz;
    AnyDivision dv(sm.nx, sm.ny, sm.nz, 0);
    const int n_rounds = (dv.n_sub + 31) / 32;
    const unsigned short* src = sup.s_count >= 0 ? sup.sid : nullptr;
    int n_src = src ? sup.s_count : g.n_holes + g.n_det;
    double dacc = 0.0;
    if (src && n_pts > 1) {               // the voxel's list
        Elem el;
        if (!init_element(g, ws.inner, d, v, cr, sr, lane, el)) return 0.0;
        const float hx = 0.5f * (fabsf(g.wx) + fabsf(g.wy)), hz = 0.5f * fabsf(g.wz);
        float4 rd;
        if (bundle_rect(g, d, el.xI, el.yI, el.zI, hx, hz, rd)) {
            int n = 0;
            for (int base = 0; base < n_src && n <= kNear; base += 32) {
                const int j = base + lane;
                const int id = j < n_src ? src[j] : 0;
                const bool maybe = j < n_src && near_bundle(g, el.xI, el.yI, el.zI, rd, id, hx, hz);
                const unsigned m = __ballot_sync(0xffffffffu, maybe);
                const int pos = n + __popc(m & ((1u << lane) - 1u));
                if (maybe && pos < kNear) ws.near[pos] = (unsigned short)id;
                n += __popc(m);
            }
            if (n <= kNear) {             // otherwise every source point filters the superset
                src = ws.near;
                n_src = n;
            }
        }
    }
    for (int p = 0; p < n_pts; ++p) {
        const int jx = p % sm.sx, jy = (p / sm.sx) % sm.sy, jz = p / (sm.sx * sm.sy);
        __syncwarp();                     // the previous point's records are no longer read
        int cursor;
        Kept k;
        {
            Elem el;
            if (!init_element(g, ws.inner, d, v, cr, sr, lane, el, ((float)jx + 0.5f) / (float)sm.sx,
                              ((float)jy + 0.5f) / (float)sm.sy, ((float)jz + 0.5f) / (float)sm.sz))
                return 0.0;               // the crystal's mu does not depend on the point
            if (lane == 0) ws.elem = el;
            cursor = build_kept(g, src, ws, el, d, 0, n_src, lane, k);   // ends in a __syncwarp
        }
        const bool single = cursor >= n_src;
        const int per = single ? kPassRounds : 8;
        Counts unused;
        for (int q0 = 0; q0 < n_rounds; q0 += per) {
            const int n = min(per, n_rounds - q0);
            dv.base = 32 * q0;
            if (ws.elem.filt) {
                ray_boxes(ws, dv, n, lane);
            } else {                      // open rectangles: every round meets every kept object
                if (lane < n) {
                    ws.box[lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    ws.reach[lane] = 0.0f;
                }
                __syncwarp();
            }
            if (single) round_masks(ws, ws.elem, k, 0, n, lane);
            attenuation_pass<false, ELL>(g, ws, dv, src, n_src, d, single, 0, n, lane, cursor, k, unused);
            for (int r = 0; r < n; ++r) {
                int ix, iy, iz;
                dv.indices(r, lane, ix, iy, iz);
                const float att = ws.att[r * 32 + lane];
                if (!isinf(att)) dacc += (double)finish_ray(ws, dv, ix, iy, iz, att);
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) dacc += __shfl_xor_sync(0xffffffffu, dacc, off);
    return dacc / (double)n_pts;
}
