// ix_metrics.cu -- the analytic optical metrics on the device (sm_100a).
//
// evaluate_gem_optical_metrics (color/metrics/evaluate.rs:158-392) for a batch of camera
// poses.  A pose is 180 cells of the 18 x 18 fan (fan.rs), each with 5 aperture rays
// (classify.rs) -- a single-index interior trace of at most 10 bounces
// (ray_trace.rs:264-352), with n_F / n_C companion traces for fire -- and 5 yaw-jittered
// rays for temporal scintillation (scintillation.rs:85): 900 or 1800 independent rays.
// What bounds them is latency: a ray is up to 31 scans of the planes, one after another (its
// entry, then 10 bounces at each of three wavelengths).
// So a ray is traced by 8 lanes that share each scan (ix_interior.cuh), four rays to a
// warp, and the rays of a pose are spread over as many warps as the launch leaves it: 4
// warps of one CTA when the poses fill the GPU, up to a cluster of 8 CTAs x 16 warps for one
// pose alone.  A warp scans the entries of all its rays first (exact scans), then steps its
// four groups' interior traces together, each group taking its next ray when one ends.
// One pose: 4.93 ms with a cell per thread of one CTA, 0.13 ms so; 724 poses without fire: 2.24
// and 0.84 ms (device time; the calls 5.00 -> 0.14 and 3.67 -> 0.83 ms).
// Each ray's result goes to the leading CTA's shared memory (over the cluster), where one
// thread per sum folds them in the reference's (ix, iz, sample) order, so every f32 sum is
// formed exactly as the CPU forms it.
//
// Compiled twice like ix_kernels.cu (IX_EXACT=1 with -fmad=false, IX_EXACT=0).
#include <cooperative_groups.h>

#include "ix_device.cuh"
#include "ix_interior.cuh"
#include "ix_launch.h"

#if IX_EXACT
#define IX_SFX(name) name##_exact
#else
#define IX_SFX(name) name##_fast
#endif

namespace ix {

namespace {

constexpr int GRID = 18;
constexpr int CELLS = GRID * GRID;
constexpr int MAX_ACTIVE = 180;  // cells with gu^2 + gv^2 <= 0.70
constexpr int SUBS = 5;          // rays of a cell in each set
constexpr int MAX_RAYS = MAX_ACTIVE * SUBS;  // of one set
constexpr int MAX_WARPS = 16;    // per CTA
constexpr int MAX_CLUSTER = 8;

enum { FATE_ENTRY_BLOCKED = 0, FATE_LEAKED = 1, FATE_EXITED_UP = 2, FATE_ABSORBED = 3 };

// fresnel_transmittance (ray_trace.rs:35).  The products are rounded before they are used on
// both sides of the test, in the fast build too.
IX_DEV float fresnel_transmittance(float n1, float n2, float cos_i, float cos_t) {
    const float a = __fmul_rn(n1, cos_i), b = __fmul_rn(n1, cos_t);
    const float denom_s = fmaf(n2, cos_t, a);
    const float denom_p = fmaf(n2, cos_i, b);
    if (fabsf(denom_s) < 1e-6f || fabsf(denom_p) < 1e-6f) return 0.0f;
    const float rs = fmaf(n2, -cos_t, a) / denom_s;
    const float rp = fmaf(n2, -cos_i, b) / denom_p;
    return clampf_(1.0f - midpointf_(rs * rs, rp * rp), 0.0f, 1.0f);
}

IX_DEV V3 plane_normal(const float4* planes, int i) {
    const float4 p = planes[i];
    return v3(p.x, p.y, p.z);
}

// trace_wavelength_detail + trace_interior (ray_trace.rs:240-352), unfrosted, as a state the
// warp steps scan by scan.
struct Trace {
    V3 point, dir;
    float index, sin_crit, entry_t;
    uint32_t bounce;
    // Escape::record (ray_trace.rs:110)
    V3 exit_dir;
    float transmittance, exit_cos;
    int facet;
};
// False: total reflection at the entry (FATE_ENTRY_BLOCKED).
IX_DEV bool trace_begin(Trace& T, V3 entry_point, V3 incoming, V3 n_entry, float cos_i, float index) {
    const float inv = 1.0f / index;
    const float sin2_t = (1.0f / (index * index)) * fmaf(cos_i, -cos_i, 1.0f);
    if (sin2_t > 1.0f) return false;
    const float cos_t = sqrtf(__fadd_rn(1.0f, -sin2_t));  // of the sin^2 tested above
    T.dir = normalize(inv * incoming + fmaf(inv, cos_i, -cos_t) * n_entry);
    T.entry_t = fresnel_transmittance(1.0f, index, cos_i, cos_t);
    T.point = entry_point + T.dir * 1e-4f;
    T.sin_crit = 1.0f / index;
    T.index = index;
    T.bounce = 0;
    return true;
}
constexpr int TRACE_ON = -1;
// After one scan: TRACE_ON, or the trace's fate.
IX_DEV int trace_step(Trace& T, const float4* __restrict__ planes, Hit h) {
    if (h.facet < 0) return FATE_ABSORBED;
    const float index = T.index;
    const V3 next = T.point + h.t * T.dir;
    const V3 n_out = plane_normal(planes, h.facet);
    const float cos_theta = clampf_(dot(T.dir, n_out), 0.0f, 1.0f);
    const float sin_theta = sqrtf(fmaxf(fmaf(cos_theta, -cos_theta, 1.0f), 0.0f));
    if (sin_theta < T.sin_crit) {
        const float sin2_out = (index * index) * fmaf(cos_theta, -cos_theta, 1.0f);
        if (sin2_out <= 1.0f) {
            const float cos_out = sqrtf(__fadd_rn(1.0f, -sin2_out));
            const V3 out_dir = normalize(index * T.dir + fmaf(index, -cos_theta, cos_out) * n_out);
            if (n_out.y < -0.05f) return FATE_LEAKED;
            if (!(out_dir.y > 0.05f)) return FATE_ABSORBED;
            T.exit_dir = out_dir;
            T.transmittance = T.entry_t * fresnel_transmittance(index, 1.0f, cos_theta, cos_out);
            T.exit_cos = cos_out;
            T.facet = h.facet;
            return FATE_EXITED_UP;
        }
    }
    T.dir = normalize(T.dir - (2.0f * cos_theta) * n_out);
    T.point = next + T.dir * 1e-4f;
    return ++T.bounce < 10u ? TRACE_ON : FATE_ABSORBED;
}

struct Fan {
    float standoff, lateral;
    // FanGeometry::origin (fan.rs:89).
    // The fast build fuses the lateral steps, for the pose's own rays onto the rounded
    // standoff point they share.
    IX_DEV V3 origin(V3 f, V3 r, V3 u, float gu, float gv, bool temporal) const {
#if !IX_EXACT
        if (!temporal) {
            const V3 a = v3(__fmul_rn(-f.x, standoff), __fmul_rn(-f.y, standoff), __fmul_rn(-f.z, standoff));
            const float x = gu * lateral, y = gv * lateral;
            return v3(fmaf(y, u.x, fmaf(x, r.x, a.x)), fmaf(y, u.y, fmaf(x, r.y, a.y)), fmaf(y, u.z, fmaf(x, r.z, a.z)));
        }
#endif
        return (-f * standoff + (gu * lateral) * r) + (gv * lateral) * u;
    }
};

// A ray's result: RAY_NONE (no entry), or RAY_HIT and its verdict.
enum : uint8_t { RAY_NONE = 0, RAY_HIT = 1, RAY_WINDOWED = 2, RAY_EXTINCT = 4, RAY_RETURNED = 8, RAY_FIRE = 16 };
struct PoseResults {
    uint8_t aperture[MAX_RAYS], temporal[MAX_RAYS];  // [active cell][sample]
    float angle[MAX_RAYS], weight[MAX_RAYS];         // of the rays with RAY_FIRE
};

IX_DEV V3 basis_vec(const MetricsPoseDev& p, int k, int which) {
    const float* b = p.basis[k] + 3 * which;
    return v3(b[0], b[1], b[2]);
}

// The stone's extents as order-preserving integers (ExtentsDev), and half of the narrower
// one; 1 for planes that enclose no solid (fan.rs:34).
#if IX_EXACT
IX_DEV unsigned long long ordered_bits(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return b >> 63 ? ~b : b | 0x8000000000000000ull;
}
#endif
IX_DEV double ordered_value(unsigned long long o) {
    return __longlong_as_double((long long)(o >> 63 ? o & 0x7FFFFFFFFFFFFFFFull : ~o));
}
IX_DEV float stone_half_width(const ExtentsDev& e) {
    if (e.found < 4u) return 1.0f;
    const double dx = __dadd_rn(ordered_value(e.hi[0]), -ordered_value(e.lo[0]));
    const double dz = __dadd_rn(ordered_value(e.hi[1]), -ordered_value(e.lo[1]));
    const double w = dx <= dz ? dx : dz;
    return isfinite(w) && w > 0.0 ? (float)(w * 0.5) : 1.0f;
}

}  // namespace

// SCORE: SCORE_RIG for the studio rigs and the iso-hemisphere, SCORE_EXT for every other
// lighting model (the launch picks by the scoring environment's model).  One cluster per pose.
template <int SCORE>
__global__ void __launch_bounds__(MAX_WARPS * 32)
    IX_SFX(metrics_kernel)(const __grid_constant__ MetricsLaunch L) {
    namespace cg = cooperative_groups;
    __shared__ float4 s_rows[IX_MAX_PLANES], s_pairs[PLANE_PAIR_VECS];
    __shared__ float s_rad[96];
    __shared__ float s_threshold;
    __shared__ uint16_t s_active[MAX_ACTIVE];
    __shared__ PoseResults s_res;  // the leading CTA's collects the pose
    __shared__ float s_fold[4];
    __shared__ uint32_t s_count[8];
    extern __shared__ __align__(8) Hit s_hits[];  // the entry of each of this CTA's rays
    const cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), ranks = cluster.num_blocks();
    const MetricsPoseDev& pose = L.poses[blockIdx.x / ranks];
    const MetricsStoneDev stone = L.stones[pose.stone];
    const int n = (int)stone.n_planes;
    const uint32_t tid = threadIdx.x, lane = tid & 31u;
    stage_planes(L.planes + stone.plane_offset, n, s_rows, s_pairs, (int)tid, (int)blockDim.x);
    if (tid < 32u) {  // the fan's active cells, in order
        uint32_t found = 0;
        for (int first = 0; first < CELLS; first += 32) {
            const int cell = first + (int)lane;
            const float gu = fmaf(((float)(cell / GRID) + 0.5f) / (float)GRID, 2.0f, -1.0f);
            const float gv = fmaf(((float)(cell % GRID) + 0.5f) / (float)GRID, 2.0f, -1.0f);
            const bool in = cell < CELLS && fmaf(gv, gv, gu * gu) <= 0.70f;
            const unsigned m = __ballot_sync(WARP_MASK, in);
            const uint32_t at = found + __popc(m & ((1u << lane) - 1u));
            if (in && at < (uint32_t)MAX_ACTIVE) s_active[at] = (uint16_t)cell;
            found += __popc(m);
        }
        if (lane == 0) s_count[0] = min(found, (uint32_t)MAX_ACTIVE);
    }
    // The exit-lighting threshold; its barriers also publish the planes and the cells.
    const float threshold = exit_lighting_threshold<SCORE>(L.env, L.spec, L.factor, L.dirs, s_rad, &s_threshold);
    const ExitScorerT<SCORE> sc{L.env, L.spec, threshold, L.head_shadow_cos};
    const float nd = fmaxf(dispersion_eval(stone.dispersion, 589.3f), 1.1f);
    const float n_f = fmaxf(dispersion_eval(stone.dispersion, 486.1f), 1.001f);
    const float n_c = fmaxf(dispersion_eval(stone.dispersion, 656.3f), 1.001f);
    const float half_width = stone_half_width(L.extents[pose.stone]);
    const Fan fan{2.5f * half_width, (0.95f * half_width) / sqrtf(0.70f)};
    const uint32_t n_active = s_count[0], n_rays = n_active * SUBS;
    const uint32_t total = L.want_fire ? 2u * n_rays : n_rays;  // aperture rays, then temporal
    const uint32_t groups = blockDim.x >> 3, group = tid >> 3, all = groups * ranks;
    // Ray i of this group is ray (rank * groups + group) + i * all of the pose, its entry at
    // s_hits[i * groups + group].
    const uint32_t mine = rank * groups + group;
    const uint32_t rounds = (total + all - 1) / all;
    PoseResults* const res = cluster.map_shared_rank(&s_res, 0);
    auto ray = [&](uint32_t q, V3& o, V3& dir, V3& forward) {
        const bool temporal = q >= n_rays;
        const uint32_t i = temporal ? q - n_rays : q;
        const int cell = s_active[i / SUBS], k = (int)(i % SUBS);
        const float gu = fmaf(((float)(cell / GRID) + 0.5f) / (float)GRID, 2.0f, -1.0f);
        const float gv = fmaf(((float)(cell % GRID) + 0.5f) / (float)GRID, 2.0f, -1.0f);
        const int which = temporal ? k + 1 : 0;
        const V3 f = basis_vec(pose, which, 0), r = basis_vec(pose, which, 1), u = basis_vec(pose, which, 2);
        o = fan.origin(f, r, u, gu, gv, temporal);
        forward = f;
        dir = f;
        if (!temporal) {
            const float su = k == 1 ? 0.08f : (k == 2 ? -0.08f : 0.0f), sv = k == 3 ? 0.08f : (k == 4 ? -0.08f : 0.0f);
            dir = normalize((f + su * r) + sv * u);
        }
    };
    for (uint32_t i = 0; i < rounds; ++i) {
        const uint32_t q = mine + i * all;
        V3 o = v3(0.0f, 0.0f, 0.0f), dir = o, f;
        if (q < total) ray(q, o, dir, f);
        __syncwarp();
        const Hit h = warp_exact_hit(s_rows, n, o, dir);
        if ((tid & 7u) == 0) s_hits[i * groups + group] = h;
    }
    __syncwarp();
    uint32_t i = 0;          // the group's next ray
    bool on = false;         // it traces one
    uint32_t stage = 0;      // its wavelength: n_d, n_F, n_C
    uint32_t q = 0;
    V3 entry = v3(0.0f, 0.0f, 0.0f), incoming = entry, normal = entry, forward = entry, f_dir = entry;
    float cos_i = 0.0f, t_d = 0.0f, t_f = 0.0f, f_cos = 0.0f;
    int f_facet = 0;
    uint32_t f_bounce = 0;
    Trace T;
    T.point = T.dir = entry;
    auto put = [&](uint8_t code, float angle, float weight) {
        on = false;
        if ((tid & 7u) != 0) return;
        if (q < n_rays) {
            res->aperture[q] = code;
            if (code & RAY_FIRE) {
                res->angle[q] = angle;
                res->weight[q] = weight;
            }
        } else {
            res->temporal[q - n_rays] = code;
        }
    };
    cluster.sync();  // every CTA of the cluster runs: its shared memory may be written
    for (;;) {
        while (!on && i < rounds && mine + i * all < total) {
            q = mine + i * all;
            const Hit h = s_hits[i * groups + group];
            ++i;
            if (h.facet < 0) {
                put(RAY_NONE, 0.0f, 0.0f);
                continue;
            }
            V3 o;
            ray(q, o, incoming, forward);
            entry = o + h.t * incoming;
            normal = plane_normal(s_rows, h.facet);
            cos_i = clampf_(dot(-incoming, normal), 0.0f, 1.0f);
            stage = 0;
            on = trace_begin(T, entry, incoming, normal, cos_i, nd);
            if (!on) put(RAY_HIT, 0.0f, 0.0f);
        }
        if (!__any_sync(WARP_MASK, on)) break;
        Hit h;
        const bool decided = warp_interior_hit(s_rows, s_pairs, n, T.point, T.dir, h);
        if (__any_sync(WARP_MASK, on && !decided)) {
            const Hit e = warp_exact_hit(s_rows, n, T.point, T.dir);
            if (!decided) h = e;
        }
        if (!on) continue;
        const int fate = trace_step(T, s_rows, h);
        if (fate == TRACE_ON) continue;
        if (stage == 0) {
            // classify_aperture_sample (classify.rs:47) / cell_temporal_variance
            // (scintillation.rs:85-117).
            uint8_t code = RAY_HIT;
            bool fire = false;
            if (fate == FATE_LEAKED) {
                code |= RAY_WINDOWED;
            } else if (fate == FATE_ABSORBED) {
                code |= RAY_EXTINCT;
            } else if (!sc.returned(T.exit_dir, forward)) {
                code |= RAY_EXTINCT;
            } else {
                code |= RAY_RETURNED;
                fire = L.want_fire && q < n_rays;
            }
            // fire_sample (classify.rs:162): the same entry at n_F, then at n_C.
            if (fire) {
                t_d = T.transmittance;
                stage = 1;
                fire = trace_begin(T, entry, incoming, normal, cos_i, n_f);
            }
            if (!fire) put(code, 0.0f, 0.0f);
        } else if (fate != FATE_EXITED_UP) {
            put(RAY_HIT | RAY_RETURNED, 0.0f, 0.0f);
        } else if (stage == 1) {
            f_dir = T.exit_dir;
            t_f = T.transmittance;
            f_cos = T.exit_cos;
            f_facet = T.facet;
            f_bounce = T.bounce;
            stage = 2;
            if (!trace_begin(T, entry, incoming, normal, cos_i, n_c)) put(RAY_HIT | RAY_RETURNED, 0.0f, 0.0f);
        } else if (f_facet == T.facet && f_bounce == T.bounce) {
            const float cos_sep = clampf_(dot(f_dir, T.exit_dir), -1.0f, 1.0f);
            put(RAY_HIT | RAY_RETURNED | RAY_FIRE, acosf(cos_sep) * 57.2957795130823208767981548141051703f,
                ((t_d * t_f) * T.transmittance) * (fmaxf(f_cos, 0.0f) * fmaxf(T.exit_cos, 0.0f)));
        } else {
            put(RAY_HIT | RAY_RETURNED, 0.0f, 0.0f);
        }
    }
    cluster.sync();
    if (rank != 0) return;
    // run_grid / sample_cell / finish_metrics (evaluate.rs:302-392, accumulate.rs:99-160): the
    // counts by one warp, each sum by one thread, in order.
    const uint32_t warp = tid >> 5;
    if (warp == 0) {
        uint32_t hit = 0, windowed = 0, extinct = 0, returned = 0;
        for (uint32_t j = lane; j < n_rays; j += 32) {
            const uint8_t c = s_res.aperture[j];
            hit += c & RAY_HIT ? 1u : 0u;
            windowed += c & RAY_WINDOWED ? 1u : 0u;
            extinct += c & RAY_EXTINCT ? 1u : 0u;
            returned += c & RAY_RETURNED ? 1u : 0u;
        }
        s_count[1] = __reduce_add_sync(WARP_MASK, hit);
        s_count[2] = __reduce_add_sync(WARP_MASK, windowed);
        s_count[3] = __reduce_add_sync(WARP_MASK, extinct);
        s_count[4] = __reduce_add_sync(WARP_MASK, returned);
    } else if (tid == 32u && L.want_fire) {
        float fire_sum = 0.0f;
        for (uint32_t j = 0; j < n_rays; ++j)
            if (s_res.aperture[j] & RAY_FIRE) fire_sum = fmaf(s_res.angle[j], s_res.weight[j], fire_sum);
        s_fold[0] = fire_sum;
    } else if (tid == 64u && L.want_fire) {
        float frac_sum = 0.0f, frac_sq = 0.0f, tvar_sum = 0.0f;
        uint32_t cells = 0;
        for (uint32_t a = 0; a < n_active; ++a) {
            uint32_t hit = 0, returned = 0, temporal = 0;
            for (uint32_t k = 0; k < SUBS; ++k) {
                const uint8_t c = s_res.aperture[a * SUBS + k];
                hit += c & RAY_HIT ? 1u : 0u;
                returned += c & RAY_RETURNED ? 1u : 0u;
                temporal += s_res.temporal[a * SUBS + k] & RAY_RETURNED ? 1u : 0u;
            }
            if (hit == 0) continue;
            const float frac = (float)returned / (float)hit;
            frac_sum = frac_sum + frac;
            frac_sq = fmaf(frac, frac, frac_sq);
            ++cells;
            const float tp = (float)temporal / 5.0f;
            tvar_sum = tvar_sum + fmaf(tp, -tp, tp);
        }
        s_fold[1] = frac_sum;
        s_fold[2] = frac_sq;
        s_fold[3] = tvar_sum;
        s_count[5] = cells;
    }
    __syncthreads();
    if (tid != 0) return;
    const uint32_t hits = s_count[1], windowed = s_count[2], extinct = s_count[3], returned = s_count[4];
    const float n_total = (float)(hits > 0 ? hits : 1u);
    float* out = L.out + (size_t)(blockIdx.x / ranks) * 5;
    out[0] = clampf_((float)returned / n_total * 100.0f, 0.0f, 100.0f);
    out[3] = clampf_((float)windowed / n_total * 100.0f, 0.0f, 100.0f);
    out[4] = clampf_((float)extinct / n_total * 100.0f, 0.0f, 100.0f);
    if (!L.want_fire) {
        out[1] = 25.0f;  // placeholder_metrics (evaluate.rs:210)
        out[2] = 75.0f;
        return;
    }
    const float fire_sum = s_fold[0], frac_sum = s_fold[1], frac_sq = s_fold[2], tvar_sum = s_fold[3];
    const uint32_t cells = s_count[5];
    out[1] = fmaxf(fire_sum / n_total * 275.0f, 0.1f);
    float spatial = 0.0f;
    if (cells > 0) {
        const float mean = frac_sum / (float)cells;
        if (mean > 1e-4f) {
            const float var = fmaxf(fmaf(mean, -mean, frac_sq / (float)cells), 0.0f);
            const float cv = sqrtf(var) / mean;
            spatial = clampf_(cv / (1.0f + cv) * 100.0f, 0.0f, 100.0f);
        }
    }
    const float temporal = cells > 0 ? clampf_(tvar_sum / (float)cells / 0.24f * 100.0f, 0.0f, 100.0f) : 0.0f;
    out[2] = clampf_(fmaf(0.4f, temporal, 0.6f * spatial), 0.0f, 100.0f);
}

#if IX_EXACT
// measure_model_width (render_setup/stone_width.rs:27, geometry/stone_metrics/measure.rs): the
// horizontal extents of the solid's vertices, in f64.  A vertex is any point where three
// planes meet and no plane is violated by more than 1e-9: one warp per pair of planes, a lane
// per third plane, the extremes collected with ordered-integer atomics.  121 planes are
// 287,980 triples, 0.3 to 4 ms on a host thread and 18 us here.  Every operation is
// written with its rounding, so that the vertices are the host's bit for bit.
constexpr int WIDTH_THREADS = 256;
__global__ void __launch_bounds__(WIDTH_THREADS) stone_extents_kernel(const __grid_constant__ WidthLaunch L) {
    const WidthStoneDev st = L.stones[blockIdx.y];
    __shared__ double s_pl[IX_MAX_PLANES][4];
    const uint32_t m = st.n_planes;
    for (uint32_t i = threadIdx.x; i < 4 * m; i += blockDim.x) s_pl[i / 4][i % 4] = L.planes[4 * (size_t)st.first + i];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    auto sub2 = [](double a, double b, double c, double d) {
        return __dadd_rn(__dmul_rn(a, b), -__dmul_rn(c, d));
    };
    auto sum3 = [](double a, double b, double c, double d, double e, double f) {
        return __dadd_rn(__dadd_rn(__dmul_rn(a, b), __dmul_rn(c, d)), __dmul_rn(e, f));
    };
    auto cross = [&](const double* a, const double* b, double o[3]) {
        o[0] = sub2(a[1], b[2], a[2], b[1]);
        o[1] = sub2(a[2], b[0], a[0], b[2]);
        o[2] = sub2(a[0], b[1], a[1], b[0]);
    };
    ExtentsDev& out = L.out[blockIdx.y];
    const uint32_t warps = gridDim.x * (WIDTH_THREADS / 32);
    for (uint32_t p = blockIdx.x * (WIDTH_THREADS / 32) + (threadIdx.x >> 5); p < m * m; p += warps) {
        const uint32_t i = p / m, j = p % m;
        if (j <= i) continue;
        double ij[3];
        cross(s_pl[i], s_pl[j], ij);
        for (uint32_t k = j + 1 + lane; k < m; k += 32) {
            double jk[3], ki[3];
            cross(s_pl[j], s_pl[k], jk);
            const double det = sum3(s_pl[i][0], jk[0], s_pl[i][1], jk[1], s_pl[i][2], jk[2]);
            if (fabs(det) < 1e-12) continue;
            cross(s_pl[k], s_pl[i], ki);
            double v[3];
            for (int a = 0; a < 3; ++a)
                v[a] = __ddiv_rn(sum3(s_pl[i][3], jk[a], s_pl[j][3], ki[a], s_pl[k][3], ij[a]), det);
            bool inside = isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2]);
            for (uint32_t q = 0; inside && q < m; ++q)
                inside = __dadd_rn(sum3(s_pl[q][0], v[0], s_pl[q][1], v[1], s_pl[q][2], v[2]), -s_pl[q][3]) <= 1e-9;
            if (!inside) continue;
            atomicAdd(&out.found, 1u);
            atomicMin(&out.lo[0], ordered_bits(v[0]));
            atomicMax(&out.hi[0], ordered_bits(v[0]));
            atomicMin(&out.lo[1], ordered_bits(v[2]));
            atomicMax(&out.hi[1], ordered_bits(v[2]));
        }
    }
}
cudaError_t launch_stone_extents(const WidthLaunch& l, cudaStream_t stream) {
    if (l.n_stones == 0) return cudaSuccess;
    // A warp per pair while the stones are few; several pairs a warp when they fill the GPU.
    uint32_t blocks = (IX_MAX_PLANES * IX_MAX_PLANES + WIDTH_THREADS / 32 - 1) / (WIDTH_THREADS / 32);
    while (blocks > 8 && (uint64_t)blocks * l.n_stones > 4096) blocks /= 2;
    for (uint32_t first = 0; first < l.n_stones; first += 65535u) {
        WidthLaunch part = l;
        part.stones += first;
        part.out += first;
        part.n_stones = min(l.n_stones - first, 65535u);
        stone_extents_kernel<<<dim3(blocks, part.n_stones), WIDTH_THREADS, 0, stream>>>(part);
    }
    return cudaGetLastError();
}
#endif

cudaError_t IX_SFX(launch_metrics)(const MetricsLaunch& l, cudaStream_t stream) {
    if (l.n_poses == 0) return cudaSuccess;
    // Warps a pose gets: 16 per SM shared among the poses, 4 to 16 of a CTA, then CTAs of a
    // cluster.
    const uint64_t target_warps = (uint64_t)l.sm_count * 16;
    uint32_t warps = 4;
    while (warps < MAX_WARPS * MAX_CLUSTER && (uint64_t)2 * warps * l.n_poses <= target_warps) warps *= 2;
    const uint32_t ranks = warps > MAX_WARPS ? warps / MAX_WARPS : 1u;
    const uint32_t threads = (warps / ranks) * 32u, groups = threads / 8u;
    const uint32_t total = (l.want_fire ? 2u : 1u) * MAX_RAYS;
    const uint32_t rounds = (total + groups * ranks - 1) / (groups * ranks);
    if ((uint64_t)l.n_poses * ranks > 0x7FFFFFFFull) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(l.n_poses * ranks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = (size_t)rounds * groups * sizeof(Hit);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ranks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return rig_scored(l.env) ? cudaLaunchKernelEx(&cfg, IX_SFX(metrics_kernel)<SCORE_RIG>, l)
                             : cudaLaunchKernelEx(&cfg, IX_SFX(metrics_kernel)<SCORE_EXT>, l);
}

}  // namespace ix
