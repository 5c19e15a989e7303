// Forward projection p = A(theta) x and its vector-Jacobian product, computed brick by brick
// without storing A.  Included by pe.cu inside its anonymous namespace (it uses the element
// set-up, candidate lists and phases of the photoelectric kernel).
//
// theta = (mu_W, mu_crystal, hole radius, collimator offset dx, dy, dz, tilt):
//   mu_W        attenuation of every collimator layer (Params_Collimator[(m+1)*10+5]);
//   mu_crystal  total attenuation of every crystal (Params_Detector[12d+7]; mu_pe fixed);
//   radius      radius of every hole (Params_Collimator[100+9h+4]);
//   dx, dz      shift of every hole centre; dy shift of the hole caps and layer planes;
//   tilt        rotation of the hole pattern about the y axis (x' = x cos - z sin,
//               z' = x sin + z cos), the one collimator rotation that keeps holes
//               parallel to y as the reference's cylinder chord requires; it turns an
//               elliptical hole's frame with it (theta_h + tilt).
// Elliptical holes (PESysMatGen.cu:801-947, sysmat_set_hole_shapes) contribute the partials
// of their chord with respect to the centre, the caps and the frame angle; their chord does
// not read the radius field (it only bounds the ellipse for the cone test), so the radius
// partial has no elliptical term.
// The derivative of A[d,v] = sum_s Omega_s exp(-att_s) absf_s follows the reference's float
// program branch by branch (PESysMatGen.cu:1240-1357): each non-zero hole chord contributes
// its analytic partials, the layer term mu_L (T/cos - sum L) its own, crystal chords and the
// self-attenuation term their lengths.  Thresholds (plate penalty, eps cut-offs, the 1e-5
// layer-term gate) are piecewise constant and contribute nothing.

constexpr int kThetaN = 7;

// Partials of a hole's chord with respect to its radius r, its centre (x, z) and a common shift dy
// of both cap planes (elliptical holes: dr is the partial of the frame angle).
struct CylGrad {
    float dr, dx, dz, dy;
};

// Partials of hole_chord (same case analysis), zero for a zero chord L and for cap to cap: with
// disc = kk r^2 - C^2, the side crossings are t1,2 = (-(kx ox + kz oz) -+ sqrt(disc)) / kk.
__device__ __forceinline__ CylGrad hole_chord_grad(const HoleRay& c, const ChordParts& p, float L, float r)
{
    const float isq = rcp_rn(p.sd), C = p.cross;
    const float dsq_r = c.kk * r * isq, dsq_x = -C * c.kz * isq, dsq_z = C * c.kx * isq;
    const float dt2_r = dsq_r * c.ikk, dt2_x = (c.kx + dsq_x) * c.ikk, dt2_z = (c.kz + dsq_z) * c.ikk;
    const float dt1_r = -dsq_r * c.ikk, dt1_x = (c.kx - dsq_x) * c.ikk, dt1_z = (c.kz - dsq_z) * c.ikk;
    // side to side t2 - t1; cap y1 to side t2 - ta (fl); side to cap y2 tb - t1 (fr)
    const float a1 = p.fl ? 0.0f : 1.0f, a2 = p.fr ? 0.0f : 1.0f;
    CylGrad g{a2 * dt2_r - a1 * dt1_r, a2 * dt2_x - a1 * dt1_x, a2 * dt2_z - a1 * dt1_z, 0.0f};
    if (p.fl) g.dy = -c.iky;
    if (p.fr) g.dy = c.iky;
    return (L == 0.0f || (p.fl && p.fr)) ? CylGrad{0.0f, 0.0f, 0.0f, 0.0f} : g;
}

// Partials of the elliptical-cylinder chord (ell_chord, same case analysis) with respect to the
// centre (xc, zc), a common shift dy of both cap planes and the frame angle theta (carried in
// CylGrad.dr).  In the hole's frame the ray is p(t) = (u0 + kx t, y_in + ky t, w0 + kz t) and
// the side crossings solve a t^2 + 2 b t + c = 0 with a = kx^2 rz^2 + kz^2 rx^2,
// b = kx u0 rz^2 + kz w0 rx^2, c = rz^2 u0^2 + rx^2 w0^2 - rx^2 rz^2; the centre moves
// (u0, w0) and the angle turns (u0, w0) and (kx, kz) together.
__device__ __forceinline__ float ell_chord_grad(float xi, float yi, float zi, float xo, float yo, float zo,
                                                float xc, float y1, float y2, float zc, float rx, float rz,
                                                float ct, float st, CylGrad& gr)
{
    gr = CylGrad{0.0f, 0.0f, 0.0f, 0.0f};
    const float L = ell_chord(xi, yi, zi, xo, yo, zo, xc, y1, y2, zc, rx, rz, ct, st);
    if (L == 0.0f) return L;
    const EllFrame f = ell_frame(xi, yi, zi, xo, yo, zo, xc, y1, y2, zc, rx, rz, ct, st);   // same case flags
    const float kx = f.kx, ky = f.ky, kz = f.kz;
    const bool fl = f.fl, fr = f.fr;
    if (fl && fr) return L;                     // |tb - ta|: cap to cap, shift and turn invariant
    const float u0 = f.x_in - xc, w0 = f.z_in - zc;
    const float rx2 = rx * rx, rz2 = rz * rz;
    const float a = kx * kx * rz2 + kz * kz * rx2;
    const float b = kx * u0 * rz2 + kz * w0 * rx2;
    const float c = rz2 * u0 * u0 + rx2 * w0 * w0 - rx2 * rz2;
    const float sq = sqrtf(b * b - a * c);
    const float ia = 1.0f / a, isq = 0.5f / sq;
    const float t1 = (-b - sq) * ia, t2 = (-b + sq) * ia;
    // d(t1), d(t2) for a parameter moving (u0, w0, kx, kz) by (du, dw, dkx, dkz)
    auto dts = [&](float du, float dw, float dkx, float dkz, float& d1, float& d2) {
        const float da = 2.0f * (kx * dkx * rz2 + kz * dkz * rx2);
        const float db = (dkx * u0 + kx * du) * rz2 + (dkz * w0 + kz * dw) * rx2;
        const float dc = 2.0f * (rz2 * u0 * du + rx2 * w0 * dw);
        const float dsq = (2.0f * b * db - da * c - a * dc) * isq;
        d1 = (-db - dsq - t1 * da) * ia;
        d2 = (-db + dsq - t2 * da) * ia;
    };
    float x1, x2, z1, z2, p1, p2;
    dts(-ct, st, 0.0f, 0.0f, x1, x2);           // xc: u0 = (x - xc) ct + ..., w0 = -(x - xc) st + ...
    dts(-st, -ct, 0.0f, 0.0f, z1, z2);          // zc
    dts(w0, -u0, kz, -kx, p1, p2);              // frame angle
    if (!fl && !fr) {                           // side to side
        gr = CylGrad{p2 - p1, x2 - x1, z2 - z1, 0.0f};
    } else if (fl) {                            // cap y1 to side: t2 - ta
        gr = CylGrad{p2, x2, z2, -1.0f / ky};
    } else {                                    // side to cap y2: tb - t1
        gr = CylGrad{-p1, -x1, -z1, 1.0f / ky};
    }
    return L;
}

// The gradient's element runs the phases of pe_ref.cuh with each ray's partials kept beside its
// attenuation (one loop with chords, partials and contributions in it held the kernel to its
// instruction fetch, as there).  The voxels of a brick with activity share its items' warps, so a brick
// with one active voxel in eight does not leave seven warps idle.  96 rows of configuration 5: 44.8 ->
// 20.1 ms (phases 37 -> 23, shared voxels 23 -> 21), bound by instruction issue; four rounds per pass and
// 128 record units are what the partials leave of the shared memory.
constexpr int kGradRounds = 4;           // rounds per pass
constexpr int kGradUnits = 128;
constexpr int kGradRays = kGradRounds * 32;

struct GradWarp {
    static constexpr int units = kGradUnits;
    float4 rec[2 * kGradUnits];          // as RefWarp
    unsigned short id[kGradUnits];
    unsigned mask[kGradUnits / 32][32];
    float4 box[32];
    float reach[32];
    // [round][lane] of: attenuation outside crystal d (infinite: skipped) and its partials in theta order
    float att[kGradRays], da[kThetaN][kGradRays];
    float open[6][kGradRays];            // the open layer's length and partials (several chunks)
    int cand[64];
    float4 inner[kMaxLayers];
    Elem elem;
    float4 sub[32];
};

struct GradSmem {
    Superset sup;
    GradWarp w[kWarps];
};

// One ray's attenuation with its partials (index: theta order) and the open layer's sums of hole
// chords and of their partials (radius, x, z, y, tilt).
struct WalkGrad {
    float att, len;
    int lay;
    float da[kThetaN];                   // da[1] belongs to the crystals
    float lr, lx, lz, ly, lp;
};

__device__ __forceinline__ void close_layers_grad(const DevGeom& g, WalkGrad& s, int upto, const HoleRay& c)
{
    while (s.lay < upto) {                                    // :1281-1284
        const float mu = g.layer[s.lay].mu_total;
        float lcol = div_by(g.layer[s.lay].thickness, c.ky, c.iky);
        if (!c.steep) lcol = g.layer[s.lay].thickness / c.ky;
        if ((lcol - s.len) >= 0.00001f) {
            s.att = __fmaf_rn(mu, lcol - s.len, s.att);
            s.da[0] += lcol - s.len;
            s.da[2] -= mu * s.lr;
            s.da[3] -= mu * s.lx;
            s.da[4] -= mu * s.ly;
            s.da[5] -= mu * s.lz;
            s.da[6] -= mu * s.lp;
        }
        s.len = 0.0f;
        s.lr = s.lx = s.lz = s.ly = s.lp = 0.0f;
        ++s.lay;
    }
}

// Attenuation outside crystal d and its partials, rounds [0, kGradRounds) of division dv.
template <bool ELL, class Div>
__device__ __forceinline__ void grad_pass(const DevGeom& g, GradWarp& ws, const Div& dv, const unsigned short* src, int n_src,
                                          int d, bool single, int lane, int cursor, Kept& k)
{
    const Elem& e = ws.elem;
    int lay = 0;
    for (bool first = true;; first = false) {
        if (!single) cursor = build_kept(g, src, ws, e, d, first ? 0 : cursor, n_src, lane, k);
        round_masks(ws, e, k, 0, kGradRounds, lane);
        const bool last = single || cursor >= n_src;
        const int lay1 = last || k.nh < k.count ? g.n_layers : (k.nh > 0 ? layer_of_hole(g, ws.id[k.nh - 1]) : lay);
        for (int r = 0; r < kGradRounds; ++r) {                           // holes and layers
            const int slot = r * 32 + lane;
            int ix, iy, iz;
            dv.indices(r, lane, ix, iy, iz);
            const float3 q = dv.centre(ws, ix, iy, iz);
            float xD, yD, zD;
            ray_end(e, q.x, q.y, q.z, xD, yD, zD);
            HoleRay c;
            hole_ray_init(c, xD - e.xI, yD - e.yI, zD - e.zI);
            WalkGrad s;
            s.lay = lay;
            bool skip;
            if (first) {
                s.att = s.len = 0.0f;
                s.lr = s.lx = s.lz = s.ly = s.lp = 0.0f;
#pragma unroll
                for (int i = 0; i < kThetaN; ++i) s.da[i] = 0.0f;
                const float rdy = e.filt ? rcp_approx(yD - e.yI) : 0.0f;
                skip = plate_penalty(g, ws.inner, e, xD, yD, zD, (xD - e.xI) * rdy, (zD - e.zI) * rdy, s.att) && g.nonneg_mu;
            } else {
                s.att = ws.att[slot];
#pragma unroll
                for (int i = 0; i < kThetaN; ++i) s.da[i] = ws.da[i][slot];
                s.len = ws.open[0][slot], s.lr = ws.open[1][slot], s.lx = ws.open[2][slot];
                s.lz = ws.open[3][slot], s.ly = ws.open[4][slot], s.lp = ws.open[5][slot];
                skip = isinf(s.att);
            }
            float y1 = NAN, y2 = NAN;                     // cap planes at hand (NaN never compares equal)
            Entries it(ws.mask, r, 0, k.nh);
            while (it.more()) {
                const int j = it.take();
                const float4 A = ws.rec[2 * j], B = ws.rec[2 * j + 1];
                const int id = ws.id[j], m = layer_of_hole(g, id);
                if (m != s.lay) close_layers_grad(g, s, m, c);
                float tmp = 0.0f, dr = 0.0f, dth = 0.0f;  // radius and frame-angle partials
                CylGrad gr{0.0f, 0.0f, 0.0f, 0.0f};
                float4 S = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if constexpr (ELL) {
                    if (g.hole_shape) S = __ldg(&g.hole_shape[id]);
                }
                if (ELL && S.x > 0.0f) {                  // elliptical hole: gr.dr holds the angle partial
                    if (!skip)
                        tmp = ell_chord_grad(e.xI, e.yI, e.zI, xD, yD, zD, A.x, B.x, B.y, A.y, S.x, S.y, S.z, S.w, gr);
                    dth = gr.dr;
                } else {
                    if (!(B.x == y1 && B.y == y2)) {
                        y1 = B.x;
                        y2 = B.y;
                        hole_ray_caps(c, e, y1, y2);
                    }
                    ChordParts p;
                    tmp = hole_chord(c, A, B.z, __fmul_rn(c.kk, B.z), __fmul_rn(B.z, B.z), &p);
                    gr = hole_chord_grad(c, p, tmp, B.z);
                    dr = gr.dr;
                }
                s.len = s.len + tmp;                                      // :1276-1278
                s.att = __fmaf_rn(B.w, tmp, s.att);
                const float dp = -A.y * gr.dx + A.x * gr.dz + dth;        // tilt about the y axis
                s.lr += dr; s.lx += gr.dx; s.lz += gr.dz; s.ly += gr.dy; s.lp += dp;
                if (B.w != 0.0f) {                                        // the hole's own medium
                    s.da[2] += B.w * dr; s.da[3] += B.w * gr.dx; s.da[4] += B.w * gr.dy;
                    s.da[5] += B.w * gr.dz; s.da[6] += B.w * dp;
                }
            }
            if (s.lay < lay1) close_layers_grad(g, s, lay1, c);
            ws.att[slot] = skip ? INFINITY : s.att;
#pragma unroll
            for (int i = 0; i < kThetaN; ++i) ws.da[i][slot] = s.da[i];
            if (!single) {
                ws.open[0][slot] = s.len, ws.open[1][slot] = s.lr, ws.open[2][slot] = s.lx;
                ws.open[3][slot] = s.lz, ws.open[4][slot] = s.ly, ws.open[5][slot] = s.lp;
            }
        }
        lay = lay1;
        for (int r = 0; r < kGradRounds && k.nh < k.count; ++r) {         // other crystals (:1290-1325)
            Entries it(ws.mask, r, k.nh, k.count);
            if (!it.more()) continue;
            const int slot = r * 32 + lane;
            int ix, iy, iz;
            dv.indices(r, lane, ix, iy, iz);
            const float3 q = dv.centre(ws, ix, iy, iz);
            float xD, yD, zD;
            ray_end(e, q.x, q.y, q.z, xD, yD, zD);
            const float rdy = e.filt ? rcp_approx(yD - e.yI) : 0.0f;
            const float sa_a = (xD - e.xI) * rdy, sa_b = (zD - e.zI) * rdy;
            float att = ws.att[slot], da = ws.da[1][slot];
            const bool skip = isinf(att);
            do {
                const float4* rec = &ws.rec[2 * k.nh + 4 * (it.take() - k.nh)];
                const bool in = !skip && in_rect(rec[3], sa_a, sa_b);
                if (!__any_sync(0xffffffffu, in)) continue;
                float mu;
                const float la = record_chord(rec, xD, yD, zD, in, mu);
                att = __fmaf_rn(la, mu, att);
                da += la;
            } while (it.more());
            ws.att[slot] = att;
            ws.da[1][slot] = da;
        }
        __syncwarp();
        if (last) break;
    }
}

// Value and theta-partials of element (d, v), summed over its sub-elements in double; every
// lane returns the warp's totals in acc[0..7] (acc[kThetaN] = the value).
template <bool ELL>
__device__ __forceinline__ void pe_element_grad(const DevGeom& g, const Superset& sup, GradWarp& ws, int d, long long v,
                                                float cr, float sr, int lane, double* acc)
{
#pragma unroll
    for (int i = 0; i <= kThetaN; ++i) acc[i] = 0.0;
    const unsigned short* src = sup.s_count >= 0 ? sup.sid : nullptr;
    const int n_src = src ? sup.s_count : g.n_holes + g.n_det;
    int cursor;
    Kept k;
    {
        Elem el;
        if (!init_element(g, ws.inner, d, v, cr, sr, lane, el)) return;
        if (lane == 0) ws.elem = el;
        ws.sub[lane] = RefDivision::entry(el, lane);
        cursor = build_kept(g, src, ws, el, d, 0, n_src, lane, k);   // ends in a __syncwarp
    }
    const Elem& e = ws.elem;
    const bool single = cursor >= n_src;
    for (int q0 = 0; q0 < 32; q0 += kGradRounds) {
        const RefDivisionAt dv(q0);
        ray_boxes(ws, dv, kGradRounds, lane);
        grad_pass<ELL>(g, ws, dv, src, n_src, d, single, lane, cursor, k);
        for (int r = 0; r < kGradRounds; ++r) {
            const int slot = r * 32 + lane;
            const float outside = ws.att[slot];
            if (isinf(outside)) continue;
            int ix, iy, iz;
            dv.indices(r, lane, ix, iy, iz);
            const RayEnd q = ray_end_terms(ws, dv, ix, iy, iz);
            const float eff = 1.0f * expf(-__fmaf_rn(q.self, e.mu_t, outside));
            const float ea = expf(-q.labs * e.mu_t);
            const float absf = div_by((1.0f - ea) * e.mu_pe, e.mu_t, e.imu_t);
            const float dabsf = q.labs * ea * e.mu_pe / e.mu_t - (1.0f - ea) * e.mu_pe / (e.mu_t * e.mu_t);
            const float base = eff * q.sa;
#pragma unroll
            for (int i = 0; i < kThetaN; ++i) {
                const float da = ws.da[i][slot] + (i == 1 ? q.self : 0.0f);
                float dc = -base * absf * da;
                if (i == 1) dc += base * dabsf;
                acc[i] += (double)dc;
            }
            acc[kThetaN] += (double)(base * absf);
        }
        __syncwarp();
    }
#pragma unroll
    for (int i = 0; i <= kThetaN; ++i)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], off);
}

// Projections run the reference-order element (pe_ref.cuh), the gradient its own.
template <int KIND>
struct AdjSmem {
    typename std::conditional<KIND == 1, GradSmem, RefSmem>::type bs;
    double acc[KIND == 1 ? kWarps : 1][kThetaN + 1];
};

// KIND 0: p[d - det_begin] += sum_v A[d,v] x[v] (precise-mode elements).
// KIND 1: grad[i] += sum_{d,v} u[d - det_begin] x[v] dA[d,v]/dtheta_i, grad[7] += u^T A x.
// KIND 2: q[v] += sum_d A[d,v] u[d - det_begin] (back projection; x is not read).
// Elements of zero weight are skipped, and so are bricks whose voxels all have x = 0.
template <int KIND, bool ELL>
__global__ void __launch_bounds__(kThreads, 2) pe_adjoint_kernel(DevGeom g, AdjLaunch L)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    AdjSmem<KIND>& sm = *reinterpret_cast<AdjSmem<KIND>*>(smem_raw);
    Superset& bs = sm.bs.sup;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (KIND == 1 && lane <= kThetaN) sm.acc[wid][lane] = 0.0;
    const float ang = L.rotation * g.angle_step;           // :1006
    const float cr = cosf(ang), sr = sinf(ang);
    const int nbx = (g.nx + L.bx - 1) / L.bx, nby = (g.ny + L.by - 1) / L.by, nbz = (g.nz + L.bz - 1) / L.bz;
    const long long n_bricks = (long long)nbx * nby * nbz;
    const long long total = n_bricks * L.det_count;
    const int n_slots = L.bx * L.by * L.bz;
    for (;;) {
        if (threadIdx.x == 0) bs.item = (long long)atomicAdd(L.work_counter, 1ull);
        __syncthreads();
        const long long item = bs.item;
        if (item >= total) break;
        const int di = (int)(item / n_bricks);
        const long long b = item - (long long)di * n_bricks;
        const int gz = (int)(b / ((long long)nbx * nby));
        const int rem = (int)(b - (long long)gz * nbx * nby);
        const int gy = rem / nbx, gx = rem - gy * nbx;
        const int x0 = gx * L.bx, y0 = gy * L.by, z0 = gz * L.bz;
        const float ud = KIND >= 1 ? L.u[di] : 1.0f;
        // the brick's voxels of non-zero weight, shared evenly by the warps
        int n_active = 0;
        for (int base = 0; base < n_slots; base += kThreads) {
            const int slot = base + threadIdx.x;
            const int ix = x0 + slot % L.bx, iy = y0 + (slot / L.bx) % L.by, iz = z0 + slot / (L.bx * L.by);
            const bool in = slot < n_slots && ix < g.nx && iy < g.ny && iz < g.nz && ud != 0.0f &&
                            (KIND == 2 || L.x[ix + g.nx * ((long long)iy + (long long)g.ny * iz)] != 0.0f);
            n_active += block_append(bs, in, (unsigned short)slot, bs.slot, n_active, 512, lane, wid);
        }
        if (n_active > 0) {
            const int x1 = min(x0 + L.bx, g.nx) - 1, y1 = min(y0 + L.by, g.ny) - 1, z1 = min(z0 + L.bz, g.nz) - 1;
            const int d = L.det_begin + di;
            float ax, ay, az, bxx, byy, bzz;
            voxel_centre(g, x0 + g.nx * ((long long)y0 + g.ny * z0), 1.0f, 0.0f, ax, ay, az);
            voxel_centre(g, x1 + g.nx * ((long long)y1 + g.ny * z1), 1.0f, 0.0f, bxx, byy, bzz);
            const float mx = 0.5f * (ax + bxx), my = 0.5f * (ay + byy), mz = 0.5f * (az + bzz);
            const float rho = 0.5f * sqrtf((bxx - ax) * (bxx - ax) + (byy - ay) * (byy - ay) +
                                           (bzz - az) * (bzz - az)) + 1e-3f;
            build_superset(g, bs, d, mx * cr - my * sr, mx * sr + my * cr, mz, rho, 0.5f * fabsf(bzz - az) + 1e-3f);
            for (int first = 0; first < n_active; first += kWarps) {
                if (first > 0) __syncthreads();            // elements start together (pe_brick)
                if (first + wid >= n_active) continue;
                const int slot = bs.slot[first + wid];
                const int ix = x0 + slot % L.bx, iy = y0 + (slot / L.bx) % L.by, iz = z0 + slot / (L.bx * L.by);
                const long long v = ix + g.nx * ((long long)iy + (long long)g.ny * iz);
                const float xv = KIND == 2 ? 1.0f : L.x[v];
                if constexpr (KIND == 0) {
                    const double val = pe_element_ref<1, false, ELL>(g, bs, sm.bs.w[wid], d, v, cr, sr, lane, nullptr);
                    if (lane == 0) atomicAdd(&L.p[di], val * (double)xv);
                } else if constexpr (KIND == 2) {
                    const double val = pe_element_ref<1, false, ELL>(g, bs, sm.bs.w[wid], d, v, cr, sr, lane, nullptr);
                    if (lane == 0) atomicAdd(&L.q[v], val * (double)ud);
                } else {
                    double acc[kThetaN + 1];
                    pe_element_grad<ELL>(g, bs, sm.bs.w[wid], d, v, cr, sr, lane, acc);
                    const double wgt = (double)ud * (double)xv;
                    if (lane == 0)
#pragma unroll
                        for (int i = 0; i <= kThetaN; ++i) sm.acc[wid][i] += wgt * acc[i];
                }
                __syncwarp();
            }
        }
        __syncthreads();
    }
    if constexpr (KIND == 1) {
        __syncthreads();
        if (threadIdx.x <= kThetaN) {
            double t = 0.0;
            for (int w = 0; w < kWarps; ++w) t += sm.acc[w][threadIdx.x];
            atomicAdd(&L.grad[threadIdx.x], t);
        }
    }
}
