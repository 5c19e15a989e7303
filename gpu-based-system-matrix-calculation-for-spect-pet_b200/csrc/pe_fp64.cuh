// FP64 mode of the photoelectric element (SYSMAT_MODE_FP64), included by pe.cu inside its
// anonymous namespace.
//
// The element is the reference's program (PESysMatGen.cu:951-1364) evaluated in double from
// the float parameter arrays: voxel source, crystal frames, cone test, sub-element positions,
// plate, hole, layer and crystal chords, attenuation sum, exponentials and solid angle.  The
// reference's float program loses up to ~2e-5 of an element to rounding: y + FOV rounded to
// float moves cap planes and plate faces by an ulp of ~60 mm, and T/cos(theta) - sum L cancels.
// In double those errors are ~1e-15.
//
// The culling machinery is the float kernel's: block superset, slope rectangles and the rounds'
// masks (Shadow) are geometric filters with margins far above float rounding, so every object they
// skip has a zero chord in double too.  The kept list's cone test, which is part of the reference's
// model rather than a filter, is evaluated in double.

// Per-element constants in double.
struct Elem64 {
    double xI, yI, zI;            // voxel centre
    double xIs, yIs, zIs;         // voxel in crystal d's frame
    double xd, yd, zd, w, t, h;   // crystal d
    double cr, sr;                // cos rot, sin rot
    double mu_t, mu_pe;
    double ux, uy, uz, crit_self; // cone test (:1110-1116)
};

// Element constants for the source point at fractions (fx, fy, fz) of voxel v's extent (1/2:
// the voxel centre, the reference's source).
__device__ __forceinline__ void init_elem64(const DevGeom& g, int d, long long v, float rotation, Elem64& E,
                                            double fx = 0.5, double fy = 0.5, double fz = 0.5)
{
    const long long nxy = (long long)g.nx * g.ny;
    const int iz = (int)(v / nxy);
    const long long r = v - (long long)iz * nxy;
    const int iy = (int)(r / g.nx);
    const int ix = (int)(r - (long long)iy * g.nx);
    const double ang = (double)rotation * (double)g.angle_step;   // :1006
    double sa, ca;
    sincos(ang, &sa, &ca);
    double x = ((double)ix - (double)g.nx / 2.0 + fx) * (double)g.wx;
    double y = ((double)iy - (double)g.ny / 2.0 + fy) * (double)g.wy;
    const double z = ((double)iz - (double)g.nz / 2.0 + fz) * (double)g.wz + (double)g.shz;
    x = x + (double)g.shx;
    y = y + (double)g.shy;
    E.xI = x * ca - y * sa;
    E.yI = x * sa + y * ca;
    E.zI = z;
    const D4 P = g.t64.cry_pos[d], S = g.t64.cry_size[d], T = g.t64.cry_trig[d];
    E.xd = P.x; E.yd = P.y; E.zd = P.z; E.mu_t = P.w;
    E.w = S.x; E.t = S.y; E.h = S.z; E.mu_pe = S.w;
    E.cr = T.x; E.sr = T.y;
    E.xIs = (E.xI - E.xd) * T.z - (E.zI - E.zd) * T.w;              // :1066-1068
    E.yIs = E.yI - E.yd;
    E.zIs = (E.xI - E.xd) * T.w + (E.zI - E.zd) * T.z;
    const double dist = sqrt((E.yd - E.yI) * (E.yd - E.yI) + (E.xd - E.xI) * (E.xd - E.xI) +
                             (E.zd - E.zI) * (E.zd - E.zI));
    E.crit_self = sqrt(E.w * E.w + E.h * E.h + E.t * E.t) / dist / 2.0;
    E.ux = (E.xd - E.xI) / dist;
    E.uy = (E.yd - E.yI) / dist;
    E.uz = (E.zd - E.zI) / dist;
}

#include "pe_ids.cuh"

// The mode's phases (pe_ids.cuh).  Divisions become reciprocals (rcp64, sqrt64: Newton steps in
// double from a float seed, an ulp or so): nothing here is matched to a float program bit for bit,
// and the library's division and root each carry a range branch and a call into every loop.
struct Mode64 {
    struct Consts { Elem64 e64; };
    using Warp = IdWarp<Mode64>;

    struct Ray {
        double xD, yD, zD;
        double tio, kx, kz, ky, iky, rx, rz, kk, ikk;
        double y1, y2, ta, tb, xl, xr, zl, zr, full;      // cap planes at hand
        float sa_a, sa_b;
    };
    struct CryRay {
        double xD, yD, zD;
        float sa_a, sa_b;
    };
    struct State {
        double att, len;
        int lay;
        __device__ __forceinline__ void begin() { att = 0.0; len = 0.0; }
        __device__ __forceinline__ void resume(double a, double o) { att = a; len = o; }
        __device__ __forceinline__ double open() const { return len; }
    };

    static constexpr int kUnitBytes = 0;                  // reads the double tables
    static __device__ __forceinline__ void records(const DevGeom&, Warp&, int, int, int) {}

    // Sub-element centre of the 8 x 16 x 8 division in crystal d's frame (:1207-1217).
    static __device__ __forceinline__ void centre(const Elem64& E, int ix, int iy, int iz, double& xs, double& ys, double& zs)
    {
        xs = -E.w / 2.0 + ((double)ix + 0.5) / 8.0 * E.w;
        zs = -E.h / 2.0 + ((double)iz + 0.5) / 8.0 * E.h;
        ys = -E.t / 2.0 + ((double)iy + 0.5) / 16.0 * E.t;
    }
    static __device__ __forceinline__ void end(const Elem64& E, int ix, int iy, int iz, double& xD, double& yD, double& zD)
    {
        double xs, ys, zs;
        centre(E, ix, iy, iz, xs, ys, zs);
        xD = E.xd + diff2(xs, E.cr, zs, E.sr);
        zD = E.zd + sum2(xs, E.sr, zs, E.cr);
        yD = E.yd + ys;
    }
    template <class Div>
    static __device__ __forceinline__ Ray ray(const Warp& ws, const Div&, int ix, int iy, int iz)
    {
        const Elem64& E = ws.c.e64;
        Ray q;
        end(E, ix, iy, iz, q.xD, q.yD, q.zD);
        const double dx = q.xD - E.xI, dy = q.yD - E.yI, dz = q.zD - E.zI;
        q.tio = sqrt64(norm3(dx, dy, dz));
        const double it = rcp64(q.tio);
        q.kx = dx * it;
        q.ky = dy * it;
        q.kz = dz * it;
        q.iky = fabs(q.ky) > 1e-30 ? rcp64(q.ky) : 1.0 / q.ky;
        q.rx = q.kx * q.iky;
        q.rz = q.kz * q.iky;
        q.kk = sum2(q.kx, q.kx, q.kz, q.kz);
        q.ikk = rcp64(q.kk);                              // NaN for an axial ray, whose discriminant is 0
        q.y1 = NAN;                                       // never compares equal
        const float rdy = ws.elem.filt ? rcp_approx((float)dy) : 0.0f;
        q.sa_a = (float)dx * rdy;
        q.sa_b = (float)dz * rdy;
        return q;
    }
    template <class Div>
    static __device__ __forceinline__ CryRay cry_ray(const Warp& ws, const Div&, int ix, int iy, int iz)
    {
        const Elem64& E = ws.c.e64;
        CryRay q;
        end(E, ix, iy, iz, q.xD, q.yD, q.zD);
        const float rdy = ws.elem.filt ? rcp_approx((float)(q.yD - E.yI)) : 0.0f;
        q.sa_a = (float)(q.xD - E.xI) * rdy;
        q.sa_b = (float)(q.zD - E.zI) * rdy;
        return q;
    }
    // Plate penalty (:1240-1254); the float "through both faces" rectangle skips rays whose chord
    // is at least the plate thickness.
    static __device__ __forceinline__ bool penalty(const DevGeom& g, const Warp& ws, const Ray& q, double& att)
    {
        bool blocked = false;
        for (int m = 0; m < g.n_layers; ++m) {
            if (in_rect(ws.inner[m], q.sa_a, q.sa_b)) continue;
            const Elem64& E = ws.c.e64;
            if (plate_chord64(E.xI, E.yI, E.zI, q.xD, q.yD, q.zD, g.t64.layer + kLayer64 * m) < (double)0.1f) {
                att = att + 100000.0;
                blocked = true;
            }
        }
        return blocked;
    }
    static __device__ __forceinline__ void close(const DevGeom& g, const Ray& q, State& s, int upto)
    {
        while (s.lay < upto) {                            // :1281-1284
            const double* Ly = g.t64.layer + kLayer64 * s.lay;
            const double lcol = Ly[6] * q.iky;            // cos(theta) is the direction's y component
            if ((lcol - s.len) >= (double)0.00001f) s.att = s.att + Ly[7] * (lcol - s.len);
            s.len = 0.0;
            ++s.lay;
        }
    }
    // The cylinder chord (chord64.cuh says which of its forms) as selects.
    static __device__ __forceinline__ void hole(const DevGeom& g, const Warp& ws, Ray& q, int, int id, State& s)
    {
        const Elem64& E = ws.c.e64;
        const D4 a = g.t64.hole_a[id], b = g.t64.hole_b[id];
        double tmp;
        const D4 S = g.t64.hole_shape ? g.t64.hole_shape[id] : D4{0.0, 0.0, 1.0, 0.0};
        if (S.x > 0.0) {
            tmp = ell_chord64_call(E.xI, E.yI, E.zI, q.xD, q.yD, q.zD, a.x, a.y, a.z, a.w, S.x, S.y, S.z, S.w);
        } else {
            if (!(a.y == q.y1 && a.z == q.y2)) {
                q.y1 = a.y;
                q.y2 = a.z;
                const double u1 = a.y - E.yI, u2 = a.z - E.yI;
                q.xl = E.xI + q.rx * u1;
                q.xr = E.xI + q.rx * u2;
                q.zl = E.zI + q.rz * u1;
                q.zr = E.zI + q.rz * u2;
                q.ta = u1 * q.iky;
                q.tb = u2 * q.iky;
                q.full = fabs(q.tb - q.ta);
                if (q.ta <= 0.0001 || q.tb <= 0.0001 || q.ta >= q.tio || q.tb >= q.tio) q.full = 0.0;
                if (fabs(a.y - a.z) < 0.001) q.ta = q.tb = q.full = 0.0;   // the chord is 0
            }
            const double r2 = b.x * b.x;
            const double dxl = q.xl - a.x, dzl = q.zl - a.w, dxr = q.xr - a.x, dzr = q.zr - a.w;
            const bool fl = sum2(dxl, dxl, dzl, dzl) <= r2, fr = sum2(dxr, dxr, dzr, dzr) <= r2;
            const double ox = E.xI - a.x, oz = E.zI - a.w;
            const double cr = diff2(q.kx, oz, q.kz, ox);
            const double disc = diff2(q.kk, r2, cr, cr);
            const bool meets = disc > 0.00001;
            const double sd = sqrt64(meets ? disc : 1.0);
            const double bb = -sum2(q.kx, ox, q.kz, oz);
            const double t1 = (bb - sd) * q.ikk, t2 = (bb + sd) * q.ikk;
            const double ea = t1 > q.ta ? t1 : q.ta, eb = t2 < q.tb ? t2 : q.tb;
            const bool ok = meets && eb > ea && !(eb <= 0.0001 || ea <= 0.0001 || eb >= q.tio || ea >= q.tio);
            tmp = (fl && fr) ? q.full : (ok ? eb - ea : 0.0);
        }
        s.len = s.len + tmp;                              // :1276-1278
        s.att = s.att + b.y * tmp;
    }
    // mu times the chord in crystal o (:1290-1325), box_chord64 as selects.
    static __device__ __forceinline__ double crystal(const DevGeom& g, const Warp& ws, const CryRay& q, int, int o)
    {
        const Elem64& E = ws.c.e64;
        const D4 P = g.t64.cry_pos[o], S = g.t64.cry_size[o], T = g.t64.cry_trig[o];
        const double xa = diff2(E.xI - P.x, T.z, E.zI - P.z, T.w), ya = E.yI - P.y;
        const double za = sum2(E.xI - P.x, T.w, E.zI - P.z, T.z);
        const double xb = diff2(q.xD - P.x, T.z, q.zD - P.z, T.w), yb = q.yD - P.y;
        const double zb = sum2(q.xD - P.x, T.w, q.zD - P.z, T.z);
        const double dx = xb - xa, dy = yb - ya, dz = zb - za;
        if (fabs(dx) < kEps64 || fabs(dy) < kEps64 || fabs(dz) < kEps64)
            return box_chord64_call(xa, ya, za, xb, yb, zb, S.x, S.y, S.z) * P.w;
        const double tio = sqrt64(norm3(dx, dy, dz));
        const double ix = tio * rcp64(dx), iy = tio * rcp64(dy), iz = tio * rcp64(dz);
        double tmin, tmax;
        clip_first(-0.5 * S.x - xa, 0.5 * S.x - xa, ix, tmin, tmax);
        clip(-0.5 * S.y - ya, 0.5 * S.y - ya, iy, tmin, tmax);
        clip(-0.5 * S.z - za, 0.5 * S.z - za, iz, tmin, tmax);
        const bool out = (tmax - tmin) < kEps64 || tmin >= tio || tmax >= tio || tmin <= kEps64 || tmax <= kEps64;
        return out ? 0.0 : (tmax - tmin) * P.w;
    }
    // Self attenuation, absorption and solid angle (:1223-1231, :1329-1357).  The extended ray of
    // the absorption chord has the ray's own direction, so its slab crossings are the ray's.
    static __device__ __forceinline__ double finish(const Warp& ws, int ix, int iy, int iz, double att)
    {
        const Elem64& E = ws.c.e64;
        const double w = E.w, t = E.t, h = E.h;
        double xs, ys, zs;
        centre(E, ix, iy, iz, xs, ys, zs);
        const double xD = E.xd + diff2(xs, E.cr, zs, E.sr) - E.xI, zD = E.zd + sum2(xs, E.sr, zs, E.cr) - E.zI;
        const double yD = E.yd + ys - E.yI;
        const double sq = sqrt64(norm3(xD, yD, zD)), isq = rcp64(sq);
        const double ux1 = ((double)ix / 8.0 - 0.5) * w, ux2 = (((double)ix + 1.0) / 8.0 - 0.5) * w;
        const double uy1 = ((double)iy / 16.0 - 0.5) * t, uy2 = (((double)iy + 1.0) / 16.0 - 0.5) * t;
        const double uz1 = ((double)iz / 8.0 - 0.5) * h, uz2 = (((double)iz + 1.0) / 8.0 - 0.5) * h;
        const double dx = xs - E.xIs, dy = ys - E.yIs, dz = zs - E.zIs;
        double l1, l2, labs;
        if (fabs(dx) < kEps64 || fabs(dy) < kEps64 || fabs(dz) < kEps64) {
            l1 = box_inside64_call(E.xIs, E.yIs, E.zIs, xs, ys, zs, -w / 2.0, -t / 2.0, -h / 2.0, w / 2.0, t / 2.0, h / 2.0);
            l2 = box_inside64_call(E.xIs, E.yIs, E.zIs, xs, ys, zs, ux1, uy1, uz1, ux2, uy2, uz2);
            const double ext = 1000.0 * isq;
            labs = box_full64_call(E.xIs, E.yIs, E.zIs, xs + dx * ext, ys + dy * ext, zs + dz * ext, ux1, uy1, uz1, ux2,
                                   uy2, uz2);
        } else {
            const double tio = sqrt64(norm3(dx, dy, dz));
            const double rx = tio * rcp64(dx), ry = tio * rcp64(dy), rz = tio * rcp64(dz);
            double tmin, tmax;
            clip_first(-w / 2.0 - E.xIs, w / 2.0 - E.xIs, rx, tmin, tmax);
            clip(-t / 2.0 - E.yIs, t / 2.0 - E.yIs, ry, tmin, tmax);
            clip(-h / 2.0 - E.zIs, h / 2.0 - E.zIs, rz, tmin, tmax);
            l1 = inside(tmin, tmax, tio);
            clip_first(ux1 - E.xIs, ux2 - E.xIs, rx, tmin, tmax);
            clip(uy1 - E.yIs, uy2 - E.yIs, ry, tmin, tmax);
            clip(uz1 - E.zIs, uz2 - E.zIs, rz, tmin, tmax);
            l2 = inside(tmin, tmax, tio);
            const double far = tio + 1000.0 * tio * isq;
            const bool out = (tmax - tmin) < kEps64 || tmin >= far || tmax >= far || tmin <= kEps64 || tmax <= kEps64;
            labs = out ? 0.0 : tmax - tmin;
        }
        att = att + (l1 - l2) * E.mu_t;
        const double absf = -expm1(-labs * E.mu_t) * E.mu_pe * rcp64(E.mu_t);
        const double rq = isq * isq * isq * (1.0 / (4.0 * 3.14159265358979323846));
        const double sax = t * h / 8.0 / 16.0 * fabs(diff2(xD, E.cr, zD, E.sr));
        const double saz = w * t / 8.0 / 16.0 * fabs(sum2(xD, E.sr, zD, E.cr));
        const double say = w * h / 8.0 / 8.0 * fabs(yD);
        const double sxy = (sax >= say) ? sax : say;
        return exp(-att) * (((sxy >= saz) ? sxy : saz) * rq) * absf;
    }
    static __device__ __forceinline__ void clip_first(double lo, double hi, double inv, double& tmin, double& tmax)
    {
        const double u = lo * inv, v = hi * inv;
        tmin = u < v ? u : v;
        tmax = u < v ? v : u;
    }
    static __device__ __forceinline__ void clip(double lo, double hi, double inv, double& tmin, double& tmax)
    {
        double a, b;
        clip_first(lo, hi, inv, a, b);
        tmin = a > tmin ? a : tmin;
        tmax = b < tmax ? b : tmax;
    }
    // box_chord_inside64's interval: the length from the box entry to the end point inside it.
    static __device__ __forceinline__ double inside(double tmin, double tmax, double tio)
    {
        const bool out = (tmax - tmin) < kEps64 || tmin >= tio || tmax <= kEps64;
        const double len = (tmax < tio ? tmax : tio) - (tmin > kEps64 ? tmin : 0.0);
        return out ? 0.0 : len;
    }
};

// Element in double.
__device__ double pe_element64(const DevGeom& g, const Superset& sup, IdWarp<Mode64>& ws, int d, long long v, float cr,
                               float sr, float rotation, int lane)
{
    const unsigned short* src = sup.s_count >= 0 ? sup.sid : nullptr;
    const int n_src = src ? sup.s_count : g.n_holes + g.n_det;
    int cursor, count, nh;
    {
        Elem el;
        if (!init_element(g, ws.inner, d, v, cr, sr, lane, el)) return 0.0;   // mu_t <= 0.01 (:1107, :1194)
        if (lane == 0) {
            ws.elem = el;
            init_elem64(g, d, v, rotation, ws.c.e64);
        }
        ws.sub[lane] = RefDivision::entry(el, lane);
        __syncwarp();
        cursor = build_ids(g, src, ws, el, ws.c.e64, d, 0, n_src, lane, count, nh);
    }
    const bool single = cursor >= n_src;
    double dacc = 0.0;
    for (int q0 = 0; q0 < 32; q0 += kIdRounds) {
        const RefDivisionAt dv(q0);
        ray_boxes(ws, dv, kIdRounds, lane);
        id_pass(g, ws, dv, src, n_src, d, single, kIdRounds, lane, cursor, count, nh);
        for (int r = 0; r < kIdRounds; ++r) {
            int ix, iy, iz;
            dv.indices(r, lane, ix, iy, iz);
            const double att = ws.att[r * 32 + lane];
            if (!isinf(att)) dacc += Mode64::finish(ws, ix, iy, iz, att);
        }
        __syncwarp();
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) dacc += __shfl_xor_sync(0xffffffffu, dacc, off);
    return dacc;
}
