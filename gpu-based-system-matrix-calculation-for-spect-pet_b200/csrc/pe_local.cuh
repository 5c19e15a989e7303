// Local-coordinate FP32 mode of the photoelectric element (SYSMAT_MODE_LOCAL), included by
// pe.cu inside its anonymous namespace.  No reference counterpart: it evaluates the
// reference's element (PESysMatGen.cu:951-1364; same cone test, chords, thresholds and solid
// angle) in float arithmetic that stays within 1e-5 of the FP64 restatement.
//
// The reference's float program loses up to ~2e-5 of an element because it works in absolute
// coordinates: cap planes and plate faces are y + FOV rounded to float (an ulp of ~60 mm),
// chords are differences of ray parameters measured from the voxel (~80 mm), and the septal
// length T/cos - sum L cancels.  These errors are shared by all rays of an element, so they do
// not average out.  Here every quantity that is large or shared is formed once per element in
// double and only small differences are rounded to float:
//   - per element (lane 0, in the warp's shared slot): the voxel centre, crystal d's centre
//     and the slopes of the central ray voxel -> centre, the plate boxes relative to the
//     voxel; per kept object (ModeLocal::records): a hole's offset from the central
//     ray at its entry plane, its depth below the voxel and its length; a crystal's centre
//     relative to crystal d's, in its own frame;
//   - per ray, in float: the sub-element's offset from crystal d's centre, the slope
//     difference to the central ray (formed without cancellation), hole chords as y-extents
//     inside the hole's circle (or ellipse) in the hole's frame, the septal length (T - sum of extents) /
//     cos, crystal chords measured from the sub-element, self-attenuation and absorption
//     chords from the sub-element centre in crystal d's frame;
//   - the 1024 contributions are summed with Neumaier's compensated summation, per lane and
//     across the warp.
// The culling (superset, slope rectangles, masks) is the float kernel's; its margins are far
// above float rounding, and the kept list's cone test is the double one of the FP64 mode.

struct ElemL {
    Elem64 e64;                  // double constants of the cone test (init_elem64)
    double rxc, rzc;             // slopes dx/dy, dz/dy of the ray voxel -> crystal d's centre
    double idyc;                 // 1 / dy of that ray
    float fdx, fdy, fdz;         // crystal d's centre minus the voxel
    float frxc, frzc;
    float cr, sr, cmr, smr;      // cos, sin of rot_d and of -rot_d
    float w, t, h, mu_t, mu_pe;
    float plate[kMaxLayers][6];  // plate boxes minus the voxel: x1, y1, z1, x2, y2, z2
    int nx, ny, nz;              // sub-elements along x, depth (y), z (the reference: 8, 16, 8)
    float rfx, rfy, rfz;         // 1/nx, 1/ny, 1/nz
};

__device__ __forceinline__ void init_elem_local(const DevGeom& g, int d, long long v, float rotation, int nx, int ny,
                                                int nz, ElemL& L, double fx = 0.5, double fy = 0.5, double fz = 0.5)
{
    init_elem64(g, d, v, rotation, L.e64, fx, fy, fz);
    L.nx = nx;
    L.ny = ny;
    L.nz = nz;
    L.rfx = 1.0f / (float)nx;
    L.rfy = 1.0f / (float)ny;
    L.rfz = 1.0f / (float)nz;
    const Elem64& E = L.e64;
    const double dx = E.xd - E.xI, dy = E.yd - E.yI, dz = E.zd - E.zI;
    L.idyc = 1.0 / dy;
    L.rxc = dx * L.idyc;
    L.rzc = dz * L.idyc;
    L.fdx = (float)dx;
    L.fdy = (float)dy;
    L.fdz = (float)dz;
    L.frxc = (float)L.rxc;
    L.frzc = (float)L.rzc;
    const D4 T = g.t64.cry_trig[d];
    L.cr = (float)T.x;
    L.sr = (float)T.y;
    L.cmr = (float)T.z;
    L.smr = (float)T.w;
    const float4 S = __ldg(&g.cry.size[d]);
    const float4 M = __ldg(&g.cry.mu[d]);
    L.w = S.x; L.t = S.y; L.h = S.z;
    L.mu_t = M.x; L.mu_pe = M.y;
    for (int m = 0; m < g.n_layers; ++m) {
        const double* Ly = g.t64.layer + kLayer64 * m;
        L.plate[m][0] = (float)(Ly[0] - E.xI);
        L.plate[m][1] = (float)(Ly[2] - E.yI);
        L.plate[m][2] = (float)(Ly[4] - E.zI);
        L.plate[m][3] = (float)(Ly[1] - E.xI);
        L.plate[m][4] = (float)(Ly[3] - E.yI);
        L.plate[m][5] = (float)(Ly[5] - E.zI);
    }
}

// Distances from p along u (|u| = 1) to where the line leaves the slab [lo, hi]: fwd along
// u, bwd along -u; iu = 1 / u.  This form's error budget (1e-5 of FP64 per element) allows a
// reciprocal multiply where the reference's exact program divides.
__device__ __forceinline__ void slab_exit(float p, float iu, float lo, float hi, float& fwd, float& bwd)
{
    if (iu > 0.0f) { fwd = (hi - p) * iu; bwd = (p - lo) * iu; }
    else           { fwd = (lo - p) * iu; bwd = (p - hi) * iu; }
}

// The reference box chord (PESysMatGen.cu:20-312) of the segment voxel -> P through the box
// [lo, hi], evaluated from the near end P (q = P - voxel, in the box's frame): only full
// crossings strictly between the two ends count.
__device__ __forceinline__ float box_chord_near(const float P[3], const float q[3], const float lo[3],
                                                const float hi[3])
{
    bool par[3];
    int npar = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        par[a] = fabsf(q[a]) < kEps;
        npar += par[a];
    }
    if (npar == 3) return 0.0f;
    if (npar == 2) {                                             // axis-parallel ray (:33-66)
        const int m = !par[0] ? 0 : (!par[1] ? 1 : 2);
        for (int a = 0; a < 3; ++a) {
            if (a == m) continue;
            const float p0 = P[a] - q[a];
            if (!(p0 >= lo[a] && p0 <= hi[a])) return 0.0f;
        }
        const float p0 = P[m] - q[m], p1 = P[m];
        if ((p0 <= lo[m] && p1 >= hi[m]) || (p1 <= lo[m] && p0 >= hi[m])) return fabsf(hi[m] - lo[m]);
        return 0.0f;
    }
    float s2 = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (par[a]) {
            const float p0 = P[a] - q[a];
            if (p0 >= hi[a] || p0 <= lo[a]) return 0.0f;          // :69-72
        } else {
            s2 += q[a] * q[a];
        }
    }
    const float tio = sqrtf(s2);
    float smin = -INFINITY, smax = INFINITY;                      // along P + s * (-q / tio)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (par[a]) continue;
        float f, b;
        slab_exit(P[a], __fdividef(-tio, q[a]), lo[a], hi[a], f, b);
        smin = fmaxf(smin, -b);
        smax = fminf(smax, f);
    }
    if (!(smin <= smax)) return 0.0f;
    if ((smax - smin) < kEps) return 0.0f;
    // the reference's parameters from the voxel are t = tio - s
    if (smin <= 0.0f || smax >= tio - kEps) return 0.0f;
    return smax - smin;
}

static __device__ __noinline__ float box_chord_near_call(float Px, float Py, float Pz, float qx, float qy, float qz, float hx,
                                                        float hy, float hz)
{
    const float P[3] = {Px, Py, Pz}, q[3] = {qx, qy, qz}, lo[3] = {-hx, -hy, -hz}, hi[3] = {hx, hy, hz};
    return box_chord_near(P, q, lo, hi);
}

// Parameters where the line from p with direction cosine 1 / iu enters and leaves [-half, half].
__device__ __forceinline__ void slab_ends(float p, float iu, float half, float& enter, float& leave)
{
    const float u = (half - p) * iu, v = (-half - p) * iu;
    enter = fminf(u, v);
    leave = fmaxf(u, v);
}

// Hole chord as a y-extent (see the file comment): the ray's offset from the hole axis at the
// hole's entry plane is (u0, w0), its slopes are (rx, rz) per unit y (a = rx^2 + rz^2, ia =
// 1/a), the hole spans [0, th] in y from that plane, dy below the voxel.  Cap/side cases and
// thresholds follow the reference (PESysMatGen.cu:688-799); the t parameters (length from the
// voxel: ta = dy * sec, ...) enter only its threshold tests.  Offsets, slopes and the roots are
// in double: near a tangent, and for a hole met far from where the ray enters the plate, the
// chord is ill-conditioned in them, and float offsets or slopes would move it by ~1e-5 mm.
// tq scales the reference's discriminant threshold (1 for a circle; an ellipse passes its
// offsets and slopes divided by its semi-axes with r = 1, and tq = rho_x^4 rho_z^4).
__device__ __forceinline__ float hole_extent(double u0d, double w0d, double rxd, double rzd, double ad, double iad,
                                             float r, float th, float dy, float sec, float tio, float ky,
                                             double tq = 1.0)
{
    const double u1d = __fma_rn(rxd, (double)th, u0d), w1d = __fma_rn(rzd, (double)th, w0d);
    const double r2 = (double)r * (double)r;
    const bool fl = sum2(u0d, u0d, w0d, w0d) <= r2;
    const bool fr = sum2(u1d, u1d, w1d, w1d) <= r2;
    const float ta = dy * sec, tb = (dy + th) * sec;
    const float full = (ta <= 0.0001f || tb <= 0.0001f || ta >= tio || tb >= tio) ? 0.0f : th;
    const double cross = diff2(u0d, rzd, w0d, rxd);
    const double qd = diff2(ad, r2, cross, cross);                 // b^2 - a c (Lagrange identity)
    const bool meets = (double)(ky * ky) * tq * qd > (double)0.00001f;   // the reference's discriminant
    const double bd = sum2(u0d, rxd, w0d, rzd);
    const double sq = (double)sqrt_mid(meets ? (float)qd : 1.0f);
    const double s1 = (-bd - sq) * iad, s2 = (-bd + sq) * iad;
    const double ea = fl ? 0.0 : s1, eb = fr ? (double)th : s2;
    const float t1 = (dy + (float)ea) * sec, t2 = (dy + (float)eb) * sec;
    const bool ok = meets && (fl || fr || (s1 >= 0.0 && s2 <= (double)th)) &&
                    !(t2 <= 0.0001f || t1 <= 0.0001f || t2 >= tio || t1 >= tio);
    const float side = (float)((fl || fr) ? eb - ea : 2.0 * sq * iad);
    const float len = (fl && fr) ? full : (ok ? side : 0.0f);
    return fabsf(th) < kEps ? 0.0f : len;
}

// Elliptical hole (length_ellipticalcylinder_ray, PESysMatGen.cu:801-947, the y-parallel
// cylinder ((u'/rho_x)^2 + (w'/rho_z)^2 <= 1 in the hole's frame turned by theta): the ray's
// offset (u, w) and slopes (rx, rz) turned into that frame (u' = u cos + w sin,
// w' = -u sin + w cos, as the reference turns the segment's points) and divided by the
// semi-axes reduce it to the unit circle, whose y-extent hole_extent gives with the
// discriminant threshold rescaled: the reference's b^2 - a c equals rho_x^4 rho_z^4 ky^2 times
// the unit circle's.  Rewrites the arguments of hole_extent in place.
__device__ __forceinline__ void to_unit_circle(double& u, double& w, double& rx, double& rz, double& a, double& ia,
                                               float& r, double& tq, float ex, float ez, float ct, float st)
{
    const double c = (double)ct, s = (double)st, iex = 1.0 / (double)ex, iez = 1.0 / (double)ez;
    const double p = sum2(u, c, w, s) * iex, q = diff2(w, c, u, s) * iez;
    const double al = sum2(rx, c, rz, s) * iex, be = diff2(rz, c, rx, s) * iez;
    u = p;
    w = q;
    rx = al;
    rz = be;
    a = sum2(al, al, be, be);
    ia = 1.0 / a;
    r = 1.0f;
    const double e2 = (double)ex * (double)ex * (double)ez * (double)ez;
    tq = e2 * e2;
}

// One ray of the local form: the sub-element's offset from crystal d's centre and the ray
// terms derived from it.
struct RayL {
    float ox, oy, oz;            // sub-element centre minus crystal d's centre (world axes)
    float qx, qy, qz;            // sub-element centre minus the voxel
    float sq, sec, ky;           // ray length, 1 / cos, cos
    float rx, rz;                // slopes
    double dsec;                 // 1 / cos in double (septal lengths: heavily attenuated rays)
    double ddrx, ddrz;           // slope difference to the central ray, in double
    double drx_, drz_, da, dia;  // slopes in double, a = rx^2 + rz^2 and 1/a
};

__device__ __forceinline__ RayL ray_local(const ElemL& L, float xDs, float yDs, float zDs)
{
    RayL r;
    r.ox = diff2(xDs, L.cr, zDs, L.sr);
    r.oy = yDs;
    r.oz = sum2(xDs, L.sr, zDs, L.cr);
    r.qx = L.fdx + r.ox;
    r.qy = L.fdy + r.oy;
    r.qz = L.fdz + r.oz;
    r.sq = sqrt_mid(norm3(r.qx, r.qy, r.qz));
    r.ky = __fdividef(r.qy, r.sq);
    r.sec = __fdividef(r.sq, r.qy);
    const float den = __fdividef(1.0f, r.qy * L.fdy);
    r.rx = __fmaf_rn(diff2(r.ox, L.fdy, L.fdx, r.oy), den, L.frxc);
    r.rz = __fmaf_rn(diff2(r.oz, L.fdy, L.fdz, r.oy), den, L.frzc);
    const Elem64& E = L.e64;
    const double cx = E.xd - E.xI, cy = E.yd - E.yI, cz = E.zd - E.zI;   // voxel -> crystal d's centre
    const double dx = cx + (double)r.ox, dy = cy + (double)r.oy, dz = cz + (double)r.oz;
    const double idy = fabs(dy) > 1e-30 ? rcp64(dy) : 1.0 / dy;   // a ray level with the plates: infinite
    r.dsec = sqrt64(norm3(dx, dy, dz)) * idy;
    const double f = idy * L.idyc;
    r.ddrx = __dmul_rn(diff2((double)r.ox, cy, cx, (double)r.oy), f);
    r.ddrz = __dmul_rn(diff2((double)r.oz, cy, cz, (double)r.oy), f);
    r.drx_ = L.rxc + r.ddrx;
    r.drz_ = L.rzc + r.ddrz;
    r.da = sum2(r.drx_, r.drx_, r.drz_, r.drz_);
    r.dia = rcp64(r.da);                       // NaN for the central axis, whose discriminant is below the threshold
    return r;
}

// The three lengths of finish_local when the ray is parallel to an axis within eps.
static __device__ __noinline__ float3 finish_lengths_parallel(float sq, float vx, float vy, float vz, float xDs, float yDs,
                                                              float zDs, float w, float t, float h, float ux1, float uy1,
                                                              float uz1, float ux2, float uy2, float uz2)
{
    // crystal entry and sub-element entry, as distances back from the sub-element centre
    // (box_chord_inside, :321-324 and its parallel-axis cases); absorption: the full chord of
    // the extended ray through the sub-element (box_chord to 1000 mm past it, :1352-1357)
    const float D3[3] = {xDs, yDs, zDs}, vq[3] = {vx, vy, vz}, ulo[3] = {ux1, uy1, uz1}, uhi[3] = {ux2, uy2, uz2};
    const float clo[3] = {-w / 2.0f, -t / 2.0f, -h / 2.0f}, chi[3] = {w / 2.0f, t / 2.0f, h / 2.0f};
    float l1 = 0.0f, l2 = 0.0f;
    float b1 = INFINITY, b2 = INFINITY, f2 = INFINITY, fa = INFINITY, ba = INFINITY;
    const bool y_ok = fabsf(vq[1]) >= 0.001f;
    bool ok1 = y_ok, ok2 = y_ok, ok_abs = true;
    const float ext = 1.0f + __fdividef(1000.0f, sq);
    int npar_abs = 0, m_abs = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) npar_abs += fabsf(vq[a] * ext) < kEps;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float p0 = D3[a] - vq[a];                 // the voxel's coordinate
        const bool par_in = fabsf(vq[a]) < kEps;
        const bool par_abs = fabsf(vq[a] * ext) < kEps;
        const float iv = __fdividef(sq, vq[a]);      // 1 / (direction cosine along a)
        float f, b;
        if (par_in) {
            if (p0 >= chi[a] || p0 <= clo[a]) ok1 = false;
            if (p0 >= uhi[a] || p0 <= ulo[a]) ok2 = false;
        } else {
            slab_exit(D3[a], iv, clo[a], chi[a], f, b);
            b1 = fminf(b1, b);
            slab_exit(D3[a], iv, ulo[a], uhi[a], f, b);
            b2 = fminf(b2, b);
            f2 = fminf(f2, f);
        }
        if (par_abs) {
            if (npar_abs == 1 ? (p0 >= uhi[a] || p0 <= ulo[a]) : !(p0 >= ulo[a] && p0 <= uhi[a])) ok_abs = false;
        } else {
            m_abs = a;
            if (par_in) slab_exit(D3[a], iv, ulo[a], uhi[a], f, b);
            else { f = f2; b = b2; }
            fa = fminf(fa, f);
            ba = fminf(ba, b);
        }
    }
    if (ok1) l1 = b1;
    if (ok2) l2 = b2;
    float labs = 0.0f;
    if (ok_abs && npar_abs < 3) labs = (npar_abs == 2) ? fabsf(uhi[m_abs] - ulo[m_abs]) : fa + ba;
    if (labs < kEps) labs = 0.0f;
    return make_float3(l1, l2, labs);
}

// Self attenuation, absorption and solid angle of sub-element (ix, iy, iz) of the L.nx x L.ny
// x L.nz division, from its centre (xDs, yDs, zDs) in crystal d's frame (:1223-1231,
// :1329-1357).
__device__ __forceinline__ float finish_local(const ElemL& L, int ix, int iy, int iz, float xDs, float yDs, float zDs,
                                              double att)
{
    struct { float qx, qy, qz, sq; } r;                  // the ray's end minus the voxel, its length
    r.qx = L.fdx + diff2(xDs, L.cr, zDs, L.sr);
    r.qy = L.fdy + yDs;
    r.qz = L.fdz + sum2(xDs, L.sr, zDs, L.cr);
    const float qq = norm3(r.qx, r.qy, r.qz);
    r.sq = sqrt_mid(qq);
    const float w = L.w, t = L.t, h = L.h;
    const float gx = L.rfx, gy = L.rfy, gz = L.rfz;
    const float vq[3] = {diff2(r.qx, L.cmr, r.qz, L.smr), r.qy, sum2(r.qx, L.smr, r.qz, L.cmr)};   // ray in d's frame
    const float D3[3] = {xDs, yDs, zDs};
    const float ulo[3] = {__fmaf_rn((float)ix, gx, -0.5f) * w, __fmaf_rn((float)iy, gy, -0.5f) * t,
                          __fmaf_rn((float)iz, gz, -0.5f) * h};
    const float uhi[3] = {__fmaf_rn((float)ix + 1.0f, gx, -0.5f) * w, __fmaf_rn((float)iy + 1.0f, gy, -0.5f) * t,
                          __fmaf_rn((float)iz + 1.0f, gz, -0.5f) * h};
    const float clo[3] = {-w / 2.0f, -t / 2.0f, -h / 2.0f}, chi[3] = {w / 2.0f, t / 2.0f, h / 2.0f};

    // crystal entry and sub-element entry, as distances back from the sub-element centre
    // (box_chord_inside); absorption: the full chord of the extended ray through the sub-element
    // (box_chord to 1000 mm past it, :1352-1357)
    float l1, l2, labs;
    if (fabsf(vq[0]) < kEps || fabsf(vq[1]) < kEps || fabsf(vq[2]) < kEps) {
        const float3 l = finish_lengths_parallel(r.sq, vq[0], vq[1], vq[2], xDs, yDs, zDs, w, t, h, ulo[0], ulo[1], ulo[2],
                                                 uhi[0], uhi[1], uhi[2]);
        l1 = l.x, l2 = l.y, labs = l.z;
    } else {
        l1 = INFINITY;
        l2 = INFINITY;
        labs = INFINITY;                                 // forward part
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float iv = __fdividef(r.sq, vq[a]);    // 1 / (direction cosine along a)
            float f, b;
            slab_exit(D3[a], iv, clo[a], chi[a], f, b);
            l1 = fminf(l1, b);
            slab_exit(D3[a], iv, ulo[a], uhi[a], f, b);
            l2 = fminf(l2, b);
            labs = fminf(labs, f);
        }
        labs = labs + l2;
        if (labs < kEps) labs = 0.0f;
    }
    att = att + (double)__fmul_rn(l1 - l2, L.mu_t);
    // exp(-att) = exp(-hi) exp(-lo), hi = att rounded to float: keeps expf's relative accuracy
    const float a_hi = (float)att, a_lo = (float)(att - (double)a_hi);
    const float eff = expf(-a_hi) * (1.0f - a_lo);
    const float absf = -expm1f(-labs * L.mu_t) * L.mu_pe / L.mu_t;
    // solid angle in double, as the reference's 4*M_PI promotion makes it
    const double dsq = (double)qq;
    const double rq = rcp64((4.0 * 3.14159265358979323846) * dsq * (double)r.sq);
    const float ax = t * h * gz * gy, az = w * t * gx * gy, ay = w * h * gx * gz;
    const float sax = (float)((double)ax * (double)fabsf(diff2(r.qx, L.cr, r.qz, L.sr)) * rq);
    const float saz = (float)((double)az * (double)fabsf(sum2(r.qx, L.sr, r.qz, L.cr)) * rq);
    const float say = (float)((double)ay * (double)fabsf(r.qy) * rq);
    const float sxy = (sax >= say) ? sax : say;
    const float sa = (sxy >= saz) ? sxy : saz;
    return eff * sa * absf;
}

// Neumaier compensated accumulation of x into (s, c).
__device__ __forceinline__ void neumaier_add(float& s, float& c, float x)
{
    const float t = s + x;
    if (fabsf(s) >= fabsf(x)) c += (s - t) + x;
    else c += (x - t) + s;
    s = t;
}

// The mode's phases (pe_ids.cuh).
template <bool ELL>
struct ModeLocal {
    using Consts = ElemL;
    using Warp = IdWarp<ModeLocal<ELL>>;

    struct Ray {
        RayL r;
        float sa_a, sa_b;
    };
    struct CryRay {
        float ox, oy, oz, qx, qy, qz;
        float sa_a, sa_b;
    };
    // The attenuation sum is kept in double: its float rounding (an ulp of ~50 for the rays that
    // cross the most tungsten) would alone move exp(-att) by ~1e-5.
    struct State {
        double att;
        float ext, hatt;             // hole y-extents of the open layer, plain and mu-weighted
        int lay;
        __device__ __forceinline__ void begin() { att = 0.0; ext = hatt = 0.0f; }
        __device__ __forceinline__ void resume(double a, double o)
        {
            att = a;
            ext = __int_as_float(__double2hiint(o));
            hatt = __int_as_float(__double2loint(o));
        }
        __device__ __forceinline__ double open() const { return __hiloint2double(__float_as_int(ext), __float_as_int(hatt)); }
    };

    static __device__ __forceinline__ float3 centre(const ElemL& L, int ix, int iy, int iz)   // :1207-1217
    {
        return make_float3(__fmaf_rn(((float)ix + 0.5f) * L.rfx, L.w, -0.5f * L.w),
                           __fmaf_rn(((float)iy + 0.5f) * L.rfy, L.t, -0.5f * L.t),
                           __fmaf_rn(((float)iz + 0.5f) * L.rfz, L.h, -0.5f * L.h));
    }
    template <class Div>
    static __device__ __forceinline__ Ray ray(const Warp& ws, const Div&, int ix, int iy, int iz)
    {
        const float3 c = centre(ws.c, ix, iy, iz);
        Ray q;
        q.r = ray_local(ws.c, c.x, c.y, c.z);
        q.sa_a = ws.elem.filt ? q.r.rx : 0.0f;
        q.sa_b = ws.elem.filt ? q.r.rz : 0.0f;
        return q;
    }
    template <class Div>
    static __device__ __forceinline__ CryRay cry_ray(const Warp& ws, const Div&, int ix, int iy, int iz)
    {
        const ElemL& L = ws.c;
        const float3 c = centre(L, ix, iy, iz);
        CryRay q;
        q.ox = diff2(c.x, L.cr, c.z, L.sr);
        q.oy = c.y;
        q.oz = sum2(c.x, L.sr, c.z, L.cr);
        q.qx = L.fdx + q.ox;
        q.qy = L.fdy + q.oy;
        q.qz = L.fdz + q.oz;
        const float rdy = ws.elem.filt ? rcp_approx(q.qy) : 0.0f;
        q.sa_a = q.qx * rdy;
        q.sa_b = q.qz * rdy;
        return q;
    }
    static __device__ __forceinline__ bool penalty(const DevGeom& g, const Warp& ws, const Ray& q, double& att)
    {
        bool blocked = false;                                              // :1240-1254
        for (int m = 0; m < g.n_layers; ++m) {
            if (in_rect(ws.inner[m], q.sa_a, q.sa_b)) continue;
            const float* pb = ws.c.plate[m];
            if (plate_chord(0.0f, 0.0f, 0.0f, q.r.qx, q.r.qy, q.r.qz, pb[0], pb[1], pb[2], pb[3], pb[4], pb[5]) < 0.1f) {
                att = att + 100000.0;
                blocked = true;
            }
        }
        return blocked;
    }
    static __device__ __forceinline__ void close(const DevGeom& g, const Ray& q, State& s, int upto)
    {
        const double sec = q.r.dsec;
        while (s.lay < upto) {                                             // :1276-1284
            const LayerInfo& Ly = g.layer[s.lay];
            if (s.hatt != 0.0f) s.att = __fma_rn((double)s.hatt, sec, s.att);
            const double sept = (double)(Ly.thickness - s.ext) * sec;
            if (sept >= (double)0.00001f) s.att = __fma_rn((double)Ly.mu_total, sept, s.att);
            s.ext = 0.0f;
            s.hatt = 0.0f;
            ++s.lay;
        }
    }
    // Kept hole j at unit j: its offset from the central ray at its entry plane (two doubles), its
    // depth below the voxel, length, radius and mu.  Kept crystal at units 2 j - nh, + 1: crystal d's
    // centre relative to its own in its frame, mu; cos(-rot), sin(-rot), w, t; h.
    static constexpr int kUnitBytes = 32;
    static __device__ __forceinline__ void records(const DevGeom& g, Warp& ws, int count, int nh, int lane)
    {
        const ElemL& L = ws.c;
        for (int j = lane; j < count; j += 32) {
            const int id = ws.id[j];
            if (j < nh) {
                const D4 a = g.t64.hole_a[id];
                const float4 hb = __ldg(&g.hole.b[id]);
                const double dy = a.y - L.e64.yI;
                *reinterpret_cast<double2*>(&ws.rec[2 * j]) =
                    make_double2(__fma_rn(L.rxc, dy, L.e64.xI - a.x), __fma_rn(L.rzc, dy, L.e64.zI - a.w));
                ws.rec[2 * j + 1] = make_float4((float)dy, (float)(a.z - a.y), hb.x, hb.y);
            } else {
                const int o = id - g.n_holes, u = 2 * (2 * j - nh);
                const D4 P = g.t64.cry_pos[o], T = g.t64.cry_trig[o];
                const double ex = L.e64.xd - P.x, ey = L.e64.yd - P.y, ez = L.e64.zd - P.z;
                const float4 so = __ldg(&g.cry.size[o]);
                ws.rec[u] = make_float4((float)diff2(ex, T.z, ez, T.w), (float)ey, (float)sum2(ex, T.w, ez, T.z),
                                        __ldg(&g.cry.mu[o].x));
                ws.rec[u + 1] = make_float4((float)T.z, (float)T.w, so.x, so.y);
                ws.rec[u + 2] = make_float4(so.z, 0.0f, 0.0f, 0.0f);
            }
        }
    }
    static __device__ __forceinline__ void hole(const DevGeom& g, const Warp& ws, const Ray& q, int j, int id, State& s)
    {
        const RayL& r = q.r;
        const double2 off = *reinterpret_cast<const double2*>(&ws.rec[2 * j]);
        const float4 B = ws.rec[2 * j + 1];
        double u0 = __fma_rn(r.ddrx, (double)B.x, off.x), w0 = __fma_rn(r.ddrz, (double)B.x, off.y);
        double rx = r.drx_, rz = r.drz_, da = r.da, ia = r.dia, tq = 1.0;
        float rad = B.z;
        if constexpr (ELL) {
            const D4 S = g.t64.hole_shape ? g.t64.hole_shape[id] : D4{0.0, 0.0, 1.0, 0.0};
            if (S.x > 0.0)
                to_unit_circle(u0, w0, rx, rz, da, ia, rad, tq, (float)S.x, (float)S.y, (float)S.z, (float)S.w);
        }
        const float ext = hole_extent(u0, w0, rx, rz, da, ia, rad, B.y, B.x, r.sec, r.sq, r.ky, tq);
        s.ext = s.ext + ext;
        s.hatt = __fmaf_rn(B.w, ext, s.hatt);
    }
    // mu times the chord in a crystal (:1290-1325): box_chord_near as selects where no axis is parallel.
    static __device__ __forceinline__ double crystal(const DevGeom&, const Warp& ws, const CryRay& q, int unit, int)
    {
        const float4 A = ws.rec[2 * unit], B = ws.rec[2 * unit + 1];
        const float h = ws.rec[2 * unit + 2].x;
        const float Px = A.x + diff2(q.ox, B.x, q.oz, B.y), Py = A.y + q.oy, Pz = A.z + sum2(q.ox, B.y, q.oz, B.x);
        const float vx = diff2(q.qx, B.x, q.qz, B.y), vy = q.qy, vz = sum2(q.qx, B.y, q.qz, B.x);
        float len;
        if (fabsf(vx) < kEps || fabsf(vy) < kEps || fabsf(vz) < kEps) {
            len = box_chord_near_call(Px, Py, Pz, vx, vy, vz, 0.5f * B.z, 0.5f * B.w, 0.5f * h);
        } else {
            const float tio = sqrt_mid(norm3(vx, vy, vz));
            float smin, smax, a, b;                       // along P + s * (-v / tio)
            slab_ends(Px, __fdividef(-tio, vx), 0.5f * B.z, smin, smax);
            slab_ends(Py, __fdividef(-tio, vy), 0.5f * B.w, a, b);
            smin = fmaxf(smin, a), smax = fminf(smax, b);
            slab_ends(Pz, __fdividef(-tio, vz), 0.5f * h, a, b);
            smin = fmaxf(smin, a), smax = fminf(smax, b);
            // the reference's parameters from the voxel are t = tio - s
            const bool out = !(smin <= smax) || (smax - smin) < kEps || smin <= 0.0f || smax >= tio - kEps;
            len = out ? 0.0f : smax - smin;
        }
        return (double)(len * A.w);
    }
};

// The element of the local form.  smp: the crystal division and the voxel's source points (the
// element is the mean over the centres of an sx x sy x sz grid over the voxel, as in the
// sampled form); nullptr = the reference's 8 x 16 x 8 division and the voxel centre.
// sub_out (one source point only): each sub-element's contribution is also written there, at
// index (iz * ny + iy) * nx + ix (the scatter grid's crystal-cell weights).
template <bool ELL, bool SMP>
__device__ double pe_element_local(const DevGeom& g, const Superset& sup, IdWarp<ModeLocal<ELL>>& ws, int d, long long v,
                                   float cr, float sr, float rotation, int lane, const Sampling* smp = nullptr,
                                   float* sub_out = nullptr)
{
    const unsigned short* src = sup.s_count >= 0 ? sup.sid : nullptr;
    const int n_src = src ? sup.s_count : g.n_holes + g.n_det;
    const int nx = SMP ? smp->nx : 8, ny = SMP ? smp->ny : 16, nz = SMP ? smp->nz : 8;
    const int n_sub = nx * ny * nz, n_rounds = (n_sub + 31) / 32;
    const int sxn = SMP ? smp->sx : 1, syn = SMP ? smp->sy : 1, szn = SMP ? smp->sz : 1;
    const int n_pts = sxn * syn * szn;
    float sum = 0.0f, comp = 0.0f;
    for (int p = 0; p < n_pts; ++p) {
        // source point at fractions ((j + 0.5) / n) of the voxel along x, y, z
        const int jx = p % sxn, jy = (p / sxn) % syn, jz = p / (sxn * syn);
        const double fxd = ((double)jx + 0.5) / (double)sxn, fyd = ((double)jy + 0.5) / (double)syn;
        const double fzd = ((double)jz + 0.5) / (double)szn;
        __syncwarp();                                    // the previous point's constants and lists are done
        int cursor, count, nh;
        {
            Elem el;
            if (!init_element(g, ws.inner, d, v, cr, sr, lane, el, (float)fxd, (float)fyd, (float)fzd)) {   // mu_t <= 0.01
                if (sub_out) {                                                                     // (:1107, :1194)
                    for (int i = lane; i < n_sub; i += 32) sub_out[i] = 0.0f;
                }
                return 0.0;
            }
            if (lane == 0) {
                ws.elem = el;
                init_elem_local(g, d, v, rotation, nx, ny, nz, ws.c, fxd, fyd, fzd);
            }
            if constexpr (!SMP) ws.sub[lane] = RefDivision::entry(el, lane);
            __syncwarp();
            cursor = build_ids(g, src, ws, el, ws.c.e64, d, 0, n_src, lane, count, nh);
        }
        const bool single = cursor >= n_src;
        for (int q0 = 0; q0 < n_rounds; q0 += kIdRounds) {
            const int n = min(kIdRounds, n_rounds - q0);
            auto pass = [&](const auto& dv) {
                ray_boxes(ws, dv, n, lane);
                id_pass(g, ws, dv, src, n_src, d, single, n, lane, cursor, count, nh);
                for (int r = 0; r < n; ++r) {
                    int ix, iy, iz;
                    dv.indices(r, lane, ix, iy, iz);
                    const double att = ws.att[r * 32 + lane];
                    const float3 c = ModeLocal<ELL>::centre(ws.c, ix, iy, iz);
                    float term = 0.0f;
                    if (!isinf(att)) {
                        term = finish_local(ws.c, ix, iy, iz, c.x, c.y, c.z, att);
                        neumaier_add(sum, comp, term);
                    }
                    if (SMP && sub_out && !dv.dead(r, lane)) sub_out[(iz * ny + iy) * nx + ix] = term;
                }
                __syncwarp();
            };
            if constexpr (SMP) pass(AnyDivision(nx, ny, nz, 32 * q0));
            else pass(RefDivisionAt(q0));
        }
    }
    // warp sum of the (sum, compensation) pairs, compensated as well
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float os = __shfl_xor_sync(0xffffffffu, sum, off);
        const float oc = __shfl_xor_sync(0xffffffffu, comp, off);
        neumaier_add(sum, comp, os);
        comp += oc;
    }
    return ((double)sum + (double)comp) / (double)n_pts;
}
