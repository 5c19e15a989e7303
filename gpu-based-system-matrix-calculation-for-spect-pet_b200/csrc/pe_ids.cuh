// Phases of the element modes that read their own geometry tables (pe_fp64.cuh, pe_local.cuh),
// included by pe.cu inside its anonymous namespace: kept objects as ids, round masks, and the walk
// over rounds, as pe_ref.cuh does for the float program (why phases: see there).  The mode supplies
// its constants, which lane 0 fills in before the phases, its ray and its chords:
//
//   Consts                        the element's constants, in shared memory
//   Ray ray(ws, ix, iy, iz)       what the holes need of a ray
//   records(g, ws, count, nh)     per-object terms of the element, kUnitBytes a hole, two units a crystal
//   State                         a ray's attenuation and its open layer (att, open, lay)
//   hole(g, ws, ray, j, id, state)   adds hole id, entry j; close(g, ray, state, upto) closes layers
//   CryRay cry_ray(...), crystal(g, ws, ray, unit, o)    chord times mu of crystal o
//   finish(g, ws, ix, iy, iz, att)                 the contribution
//
// Bound by instruction issue.  Eight rounds per pass and 160 record units are what two blocks of eight
// warps leave of an SM's shared memory.  Configuration 2, 61 crystals x 2303 voxels in the FP64 mode:
// 32.1 -> 16.9 ms; 64 x 2304 in the local mode: 18.8 -> 9.5 ms (the double tables read per entry
// instead of kept as records cost it 4.7 ms).

constexpr int kIdRounds = 8;             // rounds per pass
constexpr int kIdUnits = 160;            // record units: a hole takes one, a crystal two
constexpr int kIdWords = kIdUnits / 32;
constexpr int kCryRects = 64;            // crystals with a lane test

template <class Mode>
struct IdWarp {
    typename Mode::Consts c;
    double att[kIdRounds * 32];          // [round][lane]: attenuation outside crystal d (infinite: skipped)
    double open[kIdRounds * 32];         // the open layer's sums (elements kept in several chunks)
    float4 rec[Mode::kUnitBytes / 16 * kIdUnits + 1];   // per-object terms (Mode::records)
    unsigned short id[kIdUnits];         // kept objects in the reference's order
    unsigned mask[kIdWords][32];         // per round: the kept objects that meet its slope box
    float4 box[32];
    float reach[32];
    float4 rect[kCryRects];              // slope rectangles of the first kept crystals
    int cand[64];                        // build_ids: source positions awaiting the cone test
    float4 inner[kMaxLayers];
    Elem elem;                           // float constants of the filters
    float4 sub[32];                      // as RefWarp
};

template <class Mode>
struct IdSmem {
    Superset sup;
    IdWarp<Mode> w[kWarps];
};

// Cone test of object i (:1120-1184) in double.
__device__ __forceinline__ bool in_cone64(const DevGeom& g, const Elem64& E, int i)
{
    double ox, oy, oz, crit;
    if (i < g.n_holes) {
        const D4 a = g.t64.hole_a[i], b = g.t64.hole_b[i];
        ox = a.x; oy = b.z; oz = a.w;
        crit = b.w;
    } else {
        const D4 P = g.t64.cry_pos[i - g.n_holes], S = g.t64.cry_size[i - g.n_holes];
        ox = P.x; oy = P.y; oz = P.z;
        crit = sqrt(S.x * S.x + S.z * S.z + S.y * S.y) / 2.0;
    }
    const double L = sqrt((E.xI - ox) * (E.xI - ox) + (E.yI - oy) * (E.yI - oy) + (E.zI - oz) * (E.zI - oz));
    const double rl = 1.0 / L;
    const double vx = (ox - E.xI) * rl, vy = (oy - E.yI) * rl, vz = (oz - E.zI) * rl;
    return sqrt((vz - E.uz) * (vz - E.uz) + (vy - E.uy) * (vy - E.uy) + (vx - E.ux) * (vx - E.ux)) <=
           crit * rl + E.crit_self;
}

// As build_kept, with the double cone test, keeping ids.
template <class Mode>
__device__ __forceinline__ int build_ids(const DevGeom& g, const unsigned short* src, IdWarp<Mode>& ws, const Elem& e,
                                         const Elem64& E, int d, int cursor, int n_src, int lane, int& count, int& nh)
{
    const unsigned below = (1u << lane) - 1u;
    int n = 0, holes = 0, queued = 0;
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
            keep = in_cone64(g, E, id);
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        const int kept_holes = __popc(__ballot_sync(0xffffffffu, keep && id < g.n_holes));
        if (2 * (n + __popc(m)) - (holes + kept_holes) > kIdUnits) {
            cursor = ws.cand[0];
            break;
        }
        if (keep) ws.id[n + __popc(m & below)] = (unsigned short)id;
        n += __popc(m);
        holes += kept_holes;
        const int rest = queued - take;
        const int moved = lane < rest ? ws.cand[32 + lane] : 0;
        __syncwarp();
        if (lane < rest) ws.cand[lane] = moved;
        queued = rest;
        __syncwarp();
    }
    count = n;
    nh = holes;
    for (int k = lane; k < n - holes && k < kCryRects; k += 32) {
        const int o = ws.id[holes + k] - g.n_holes;
        ws.rect[k] = e.filt ? crystal_rect(__ldg(&g.cry.pos[o]), __ldg(&g.cry.size[o]), __ldg(&g.cry.trig[o]), e.xI, e.yI,
                                           e.zI)
                            : open_rect();
    }
    __syncwarp();
    Mode::records(g, ws, n, holes, lane);
    __syncwarp();
    return cursor;
}

// round_masks of kept ids.
template <class W>
__device__ __forceinline__ void id_masks(const DevGeom& g, W& ws, const Elem& e, int count, int n_rounds, int lane)
{
    for (int w = 0; w * 32 < count; ++w) {
        const int j = w * 32 + lane;
        Shadow s;
        if (j < count) {
            const int id = ws.id[j];
            if (id < g.n_holes) {
                const float4 a = __ldg(&g.hole.a[id]);
                s.hole(e, a, __ldg(&g.hole.b[id].x));
            } else {
                const int o = id - g.n_holes;
                const float4 P = __ldg(&g.cry.pos[o]), S = __ldg(&g.cry.size[o]), T = __ldg(&g.cry.trig[o]);
                s.crystal(e, e.filt ? crystal_rect(P, S, T, e.xI, e.yI, e.zI) : open_rect(), P.x, P.z, 0.5f * S.x,
                          0.5f * S.z, T.x, T.y);
            }
        }
        unsigned mine = 0u;
        for (int r = 0; r < n_rounds; ++r) {
            const unsigned m = __ballot_sync(0xffffffffu, s.meets(ws.box[r], ws.reach[r]));
            if (lane == r) mine = m;
        }
        if (lane < n_rounds) ws.mask[w][lane] = mine;
    }
    __syncwarp();
}

// Attenuation outside crystal d of the rays of rounds [0, n_rounds), into ws.att.
template <class Mode, class Div>
__device__ __forceinline__ void id_pass(const DevGeom& g, IdWarp<Mode>& ws, const Div& dv, const unsigned short* src,
                                        int n_src, int d, bool single, int n_rounds, int lane, int cursor, int& count,
                                        int& nh)
{
    const Elem& e = ws.elem;
    int lay = 0;
    for (bool first = true;; first = false) {
        if (!single) cursor = build_ids(g, src, ws, e, ws.c.e64, d, first ? 0 : cursor, n_src, lane, count, nh);
        id_masks(g, ws, e, count, n_rounds, lane);
        const bool last = single || cursor >= n_src;
        const int lay1 = last || nh < count ? g.n_layers : (nh > 0 ? layer_of_hole(g, ws.id[nh - 1]) : lay);
        for (int r = 0; r < n_rounds; ++r) {                              // holes and layers
            int ix, iy, iz;
            dv.indices(r, lane, ix, iy, iz);
            typename Mode::Ray q = Mode::ray(ws, dv, ix, iy, iz);
            typename Mode::State s;
            s.lay = lay;
            bool skip;
            if (first) {
                s.begin();
                skip = (Mode::penalty(g, ws, q, s.att) && g.nonneg_mu) || dv.dead(r, lane);
            } else {
                s.resume(ws.att[r * 32 + lane], ws.open[r * 32 + lane]);
                skip = isinf(s.att);
            }
            Entries it(ws.mask, r, 0, nh);
            while (it.more()) {
                const int j = it.take(), id = ws.id[j];
                const int m = layer_of_hole(g, id);
                if (m != s.lay) Mode::close(g, q, s, m);
                Mode::hole(g, ws, q, j, id, s);
            }
            if (s.lay < lay1) Mode::close(g, q, s, lay1);
            ws.att[r * 32 + lane] = skip ? (double)INFINITY : s.att;
            if (!single) ws.open[r * 32 + lane] = s.open();
        }
        lay = lay1;
        for (int r = 0; r < n_rounds && nh < count; ++r) {                // other crystals
            Entries it(ws.mask, r, nh, count);
            if (!it.more()) continue;
            int ix, iy, iz;
            dv.indices(r, lane, ix, iy, iz);
            const typename Mode::CryRay q = Mode::cry_ray(ws, dv, ix, iy, iz);
            double att = ws.att[r * 32 + lane];
            const bool skip = isinf(att);
            do {
                const int j = it.take();
                const bool in = !skip && (j - nh >= kCryRects || in_rect(ws.rect[j - nh], q.sa_a, q.sa_b));
                if (!__any_sync(0xffffffffu, in)) continue;
                double t = 0.0;
                if (in) t = Mode::crystal(g, ws, q, 2 * j - nh, ws.id[j] - g.n_holes);
                att = att + t;
            } while (it.more());
            ws.att[r * 32 + lane] = att;
        }
        __syncwarp();
        if (last) break;
    }
}
