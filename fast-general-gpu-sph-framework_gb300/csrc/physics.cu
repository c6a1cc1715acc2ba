// physics.cu — density, force and integration (rows A10-A12), plus the FP64
// state reductions.
//
// Reference behaviour (KemengHuang/Fast-General-GPU-SPH-framework):
//   density    src/solver/density_kernels.cu:160-179 (TRA loop), 278-295
//              (SMS batch), 297-565 (hybrid kernel; 1/rho -> position.w,
//              pressure -> evaluated_velocity.w)
//   force      src/solver/force_kernels.cu:378-435 (SMS batch), 525-561 (TRA
//              loop), 725-1054 (hybrid kernel: spiky pressure, Mueller
//              viscosity, colour-field surface tension -> acceleration)
//   rows       src/solver/kernel_common.cuh:69-112 (TRA row range),
//              614-674 (SMS row range from task micro bounds)
//   integrate  src/solver/integration_kernels.cu:235-336 (knIntegrateVelocityE)
//   checksum   src/simulation/sph_hybrid_system.cpp:43-62
//
// Design here: one persistent kernel per pass and path; each warp repeatedly
// takes a work unit from a device counter — 32 TRA particles (one per lane) or
// a cluster of 16 particles of an SMS task (candidates pruned by the cluster's
// bounding box, staged in batches in shared memory and evaluated two at a time
// with packed FP32x2 arithmetic). The grid is sized from the SM count, so the
// launch needs neither the host-side TRA/SMS counts nor a host
// synchronisation. TRA neighbour rows merge the three x-adjacent cells of each
// (dy, dz) row into one contiguous index range, pruned by micro-x slab as in
// the reference. Candidates are visited rows z-major, then in increasing
// sorted index; the TRA density pass records which interact as bit masks that
// the TRA force pass walks.
#include <algorithm>
#include <type_traits>

#include "gsph_internal.h"

namespace gsph {

namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr float kFloatSmall = 1e-12f;   // core/cuda_math.cuh:14

__device__ __forceinline__ float powf_7(float b) {
    // kernel_common.cuh:51-55, six sequential multiplies
    return b * b * b * b * b * b * b;
}

// Squared distance with one fixed rounding sequence (x^2, then + y^2, then
// + z^2, each fused), shared by the force passes.
__device__ __forceinline__ float sq_dist(float dx, float dy, float dz) {
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// a b + c d and a . b with one fixed rounding sequence. Where an expression
// leaves the compiler a choice of which product to fuse, its choice may differ
// between the builds of a kernel, and the builds have to give the same bits.
__device__ __forceinline__ float mad2(float a, float b, float c, float d) {
    return __fmaf_rn(a, b, __fmul_rn(c, d));
}
__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by,
                                      float bz) {
    return __fmaf_rn(az, bz, mad2(ax, bx, ay, by));
}

// The TRA density pass's cut-off test in one unsigned compare: with
// e = d^2 - kFloatSmall (the subtraction folded into the first fused
// multiply-add), the reference's kFloatSmall <= d^2 <= h^2 is
// 0 <= e <= h^2 - kFloatSmall, and for FP32 values that is
// bits(e) <= bits(h^2 - kFloatSmall) (a negative e has its sign bit set).
// The weight (h^2 - d^2) is then (h^2 - kFloatSmall) - e. Only roundings
// differ from the two-compare form; pairs at the cut-off contribute zero
// either way.
__device__ __forceinline__ float sq_dist_less_small(float dx, float dy, float dz) {
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, -kFloatSmall)));
}

// Start of micro-x slab `lo` of cell c (0 = cell start).
__device__ __forceinline__ int slab_begin(const Frame &f, int c, int s, int e,
                                          int lo) {
    if (lo == 0) return s;
    const uint32_t xs = f.cell_xslab[c];
    if (xs == kXslabUnknown) return s;
    return s + min(int((xs >> (10 * (lo - 1))) & 1023u), e - s);
}
// End of micro-x slab `hi` of cell c (3 = cell end).
__device__ __forceinline__ int slab_end(const Frame &f, int c, int s, int e,
                                        int hi) {
    if (hi == 3) return e;
    const uint32_t xs = f.cell_xslab[c];
    if (xs == kXslabUnknown) return e;
    return s + min(int((xs >> (10 * hi)) & 1023u), e - s);
}

// Contiguous candidate range of one neighbour row: left cell from micro-x
// `lo`, the middle cell, right cell up to micro-x `hi` (kernel_common.cuh:
// 69-112 for TRA with lo = hi = own micro-x; 614-674 for SMS tasks).
__device__ __forceinline__ void row_range(const Frame &f, const SceneGeom &G,
                                          int m, int cx, int lo, int hi,
                                          int &begin, int &end) {
    const int sM = f.cell_start[m];
    const int eM = f.cell_start[m + 1];
    begin = sM;
    end = eM;
    if (cx > 0) begin = slab_begin(f, m - 1, f.cell_start[m - 1], sM, lo);
    if (cx + 1 < G.gx) end = slab_end(f, m + 1, eM, f.cell_start[m + 2], hi);
}

struct MicroPos {
    int cx, cy, cz, lmx;
};

__device__ __forceinline__ MicroPos micro_of(float4 p, const DevParams &P,
                                             const SceneGeom &G) {
    // Same float arithmetic as the key (grid.cu); positions are inside the
    // grid after the arrange stage has clamped/flagged them.
    int mx = int(floorf(p.x * P.rat));
    int my = int(floorf(p.y * P.rat));
    int mz = int(floorf(p.z * P.rat));
    mx = min(max(mx, 0), (G.gx << 2) - 1);
    my = min(max(my, 0), (G.gy << 2) - 1);
    mz = min(max(mz, 0), (G.gz << 2) - 1);
    MicroPos r;
    r.cx = mx >> 2;
    r.cy = my >> 2;
    r.cz = mz >> 2;
    r.lmx = mx & 3;
    return r;
}

// A TRA particle's neighbour rows in four registers: its own cell, the strides
// of a cell in y and z, and in `flags` which of the nine rows lie in the grid (bits 0-8),
// whether the left and right cells do (9, 10) and its micro-x slab (11, 12).
// Eight registers of grid sizes and cell coordinates in the row loop cost a
// batch 18% of the density pass (5.28M particles in 64 scenes 701 us, with this
// 627; one scene, whose sizes come as kernel constants, 588 and 596, so it keeps
// them).
struct RowFrame {
    int own, sy, sz;
    uint32_t flags;
};
__device__ __forceinline__ RowFrame row_frame(const MicroPos &mp, const SceneGeom &G) {
    RowFrame w;
    w.sy = G.gx;
    w.sz = G.gx * G.gy;
    w.own = G.cbase + mp.cx + w.sy * mp.cy + w.sz * mp.cz;
    const uint32_t y = (mp.cy > 0 ? 1u : 0u) | 2u | (mp.cy + 1 < G.gy ? 4u : 0u);
    w.flags = (mp.cz > 0 ? y : 0u) | (y << 3) | (mp.cz + 1 < G.gz ? y << 6 : 0u) |
              (mp.cx > 0 ? 1u << 9 : 0u) | (mp.cx + 1 < G.gx ? 1u << 10 : 0u) |
              (uint32_t(mp.lmx) << 11);
    return w;
}
__device__ __forceinline__ void tra_row_range(const Frame &f, const RowFrame &w, int m,
                                              int &begin, int &end) {
    const int sM = f.cell_start[m];
    const int eM = f.cell_start[m + 1];
    const int lmx = int(w.flags >> 11);
    begin = sM;
    end = eM;
    if (w.flags & (1u << 9)) begin = slab_begin(f, m - 1, f.cell_start[m - 1], sM, lmx);
    if (w.flags & (1u << 10)) end = slab_end(f, m + 1, eM, f.cell_start[m + 2], lmx);
}

struct ForceAcc {
    float px, py, pz;   // pressure sum
    float vx, vy, vz;   // viscosity sum
    float gx, gy, gz;   // colour gradient
    float lap;          // colour laplacian
};

// Monaghan's artificial viscosity of one interacting pair (the optional
// GSPH_VISCOSITY_ARTIFICIAL model, Monaghan 1992): for v_ij . r_ij < 0,
// mu = h v_ij . r_ij / (r^2 + 0.01 h^2), Pi = -alpha c0 mu / rho_mean with
// rho_mean = (rho_i + rho_j) / 2 = (V_i + V_j) / (2 V_i V_j), V = 1/rho.
// Returns Pi (h - r)^2 / r, the factor of r_ij in sum_j Pi grad W / spiky;
// zero for a separating pair.
__device__ __forceinline__ float artificial_pair(float vr, float d2, float k,
                                                 float inv_d, float vi, float vj,
                                                 const DevParams &P) {
    if (!(vr < 0.f)) return 0.f;
    // mu and the mean density's reciprocal under one division
    const float num = -2.f * P.art_coef * P.h * vr * vi * vj;
    const float pij = __fdividef(num, (d2 + P.art_eps) * (vi + vj));
    return pij * k * k * inv_d;
}

// What one interacting pair adds to the accumulator: pressure -r ps, viscosity
// u wk, gradient r gw, laplacian wh lf. kArt: the viscosity slots hold
// Monaghan's sum_j Pi (h - r)^2 / r r_ij instead of the reference's Laplacian
// term.
struct PairTerms {
    float rx, ry, rz, ps;
    float ux, uy, uz, wk;
    float gw, wh, lf;
};
template <bool kArt>
__device__ __forceinline__ PairTerms pair_terms(const float4 &self, const float4 &sev,
                                                const float4 &q, const float4 &qev,
                                                const DevParams &P) {
    PairTerms t;
    t.rx = self.x - q.x;
    t.ry = self.y - q.y;
    t.rz = self.z - q.z;
    const float d2 = sq_dist(t.rx, t.ry, t.rz);
    const float inv_d = rsqrtf(d2);
    const float k = __fmaf_rn(-d2, inv_d, P.h);   // h - r
    const float V = q.w;                          // 1/rho_j
    const float wk = V * k;
    t.ps = wk * (sev.w + qev.w) * k * inv_d;
    if (kArt) {
        const float vr =
            dot3(sev.x - qev.x, sev.y - qev.y, sev.z - qev.z, t.rx, t.ry, t.rz);
        t.ux = t.rx;
        t.uy = t.ry;
        t.uz = t.rz;
        t.wk = artificial_pair(vr, d2, k, inv_d, self.w, V, P);
    } else {
        t.ux = qev.x - sev.x;
        t.uy = qev.y - sev.y;
        t.uz = qev.z - sev.z;
        t.wk = wk;
    }
    const float h2r2 = P.h2 - d2;
    t.wh = V * h2r2;
    t.gw = t.wh * h2r2;
    t.lf = __fmaf_rn(-0.75f, h2r2, d2);
    return t;
}

// kChecked = false for neighbours taken from the density pass's masks: the
// masks were set by the same squared distance and the same cut-off test, so
// the test would always pass.
template <bool kChecked = true, bool kArt = false>
__device__ __forceinline__ void force_pair(const float4 &self,
                                           const float4 &sev, const float4 &q,
                                           const float4 &qev,
                                           const DevParams &P, ForceAcc &a) {
    if (kChecked) {
        const float d2 = sq_dist(self.x - q.x, self.y - q.y, self.z - q.z);
        if (P.h2 < d2 || kFloatSmall > d2) return;
    }
    const PairTerms t = pair_terms<kArt>(self, sev, q, qev, P);
    a.px = __fmaf_rn(t.rx, -t.ps, a.px);
    a.py = __fmaf_rn(t.ry, -t.ps, a.py);
    a.pz = __fmaf_rn(t.rz, -t.ps, a.pz);
    a.vx = __fmaf_rn(t.ux, t.wk, a.vx);
    a.vy = __fmaf_rn(t.uy, t.wk, a.vy);
    a.vz = __fmaf_rn(t.uz, t.wk, a.vz);
    a.gx = __fmaf_rn(t.rx, t.gw, a.gx);
    a.gy = __fmaf_rn(t.ry, t.gw, a.gy);
    a.gz = __fmaf_rn(t.rz, t.gw, a.gz);
    a.lap = __fmaf_rn(t.wh, t.lf, a.lap);
}

__device__ __forceinline__ void write_density(const Frame &f, const DevParams &P,
                                              int self, float sum, bool sms) {
    float rho = sum * P.density_scale + P.self_density;
    // The SMS path of the reference guards rho < 1e-12 before the reciprocal
    // (density_kernels.cu:540-541); the TRA path does not (:353-355).
    const float stored = (sms && rho < kFloatSmall) ? P.rest_density : rho;
    f.pos[self].w = __fdividef(1.0f, stored);
    f.ev[self].w = (powf_7(rho * P.inv_rest_density) - 1) * P.gas_constant;
}

// knIntegrateVelocityE (integration_kernels.cu:235-336), same operation order:
// penalty walls on the old velocity, a = F/rho + g, clamps, semi-implicit
// Euler, damped reflection, ev = (v_new + ev_old) / 2; 1/rho and pressure
// are kept.
__device__ __forceinline__ void integrate_one(const float4 tp, const float4 v4,
                                              const float4 ev, float ax, float ay,
                                              float az, const DevParams &P,
                                              const SceneGeom &G, float4 &pos_out,
                                              float4 &vel_out, float4 &ev_out) {
    float vx = v4.x, vy = v4.y, vz = v4.z;
    const float alpha = 20000000.f;
    const float beta = 200000.f;
    const float kernel = P.wall_kernel;
    float diff;
    diff = kernel - (tp.y - P.bmin);
    if (diff > 0.0f) ay += mad2(alpha, diff, -beta, vy);
    diff = kernel - (G.bmax_y - tp.y);
    if (diff > 0.0f) ay -= mad2(alpha, diff, beta, vy);
    diff = kernel - (tp.x - P.bmin);
    if (diff > 0.0f) ax += mad2(alpha, diff, -beta, vx);
    diff = kernel - (G.bmax_x - tp.x);
    if (diff > 0.0f) ax -= mad2(alpha, diff, beta, vx);
    diff = kernel - (tp.z - P.bmin);
    if (diff > 0.0f) az += mad2(alpha, diff, -beta, vz);
    diff = kernel - (G.bmax_z - tp.z);
    if (diff > 0.0f) az -= mad2(alpha, diff, beta, vz);
    const float acc_limit = 3000000.f;
    const float vel_limit = 36.f;
    ax = __fmaf_rn(ax, tp.w, P.gx_acc);
    ay = __fmaf_rn(ay, tp.w, P.gy_acc);
    az = __fmaf_rn(az, tp.w, P.gz_acc);
    float speed = dot3(ax, ay, az, ax, ay, az);
    if (speed > acc_limit) {
        const float s = sqrtf(acc_limit / speed);
        ax *= s;
        ay *= s;
        az *= s;
    }
    vx = __fmaf_rn(ax, P.time_step, vx);
    vy = __fmaf_rn(ay, P.time_step, vy);
    vz = __fmaf_rn(az, P.time_step, vz);
    speed = dot3(vx, vy, vz, vx, vy, vz);
    if (speed > vel_limit) {
        const float s = sqrtf(vel_limit / speed);
        vx *= s;
        vy *= s;
        vz *= s;
    }
    float px = __fmaf_rn(vx, P.time_step, tp.x);
    float py = __fmaf_rn(vy, P.time_step, tp.y);
    float pz = __fmaf_rn(vz, P.time_step, tp.z);
    if (px >= G.bmax_x) { vx *= P.wall_damping; px = G.bmax_x - kernel; }
    if (px <= P.bmin) { vx *= P.wall_damping; px = P.bmin + kernel; }
    if (py >= G.bmax_y) { vy *= P.wall_damping; py = G.bmax_y - kernel; }
    if (py <= P.bmin) { vy *= P.wall_damping; py = P.bmin + kernel; }
    if (pz >= G.bmax_z) { vz *= P.wall_damping; pz = G.bmax_z - kernel; }
    if (pz <= P.bmin) { vz *= P.wall_damping; pz = P.bmin + kernel; }
    pos_out = make_float4(px, py, pz, tp.w);
    vel_out = make_float4(vx, vy, vz, 0.f);
    ev_out = make_float4((vx + ev.x) * 0.5f, (vy + ev.y) * 0.5f, (ev.z + vz) * 0.5f, ev.w);
}

// Writes the force; with f.pos_next set, also integrates the particle (the
// same arithmetic as k_integrate on the stored force) into the next buffers.
__device__ __forceinline__ void write_force(const Frame &f, const DevParams &P,
                                            int self, const float4 &p,
                                            const float4 &pev, const SceneGeom &G,
                                            const ForceAcc &a, bool sms) {
    float tx, ty, tz;
    if (P.visc_artificial) {
        // -m rho_i sum Pi grad W: the mass is applied below with the rest
        const float c = -P.spiky * __fdividef(1.0f, p.w);
        tx = mad2(a.px, P.half_spiky, a.vx, c);
        ty = mad2(a.py, P.half_spiky, a.vy, c);
        tz = mad2(a.pz, P.half_spiky, a.vz, c);
    } else {
        tx = mad2(a.px, P.half_spiky, a.vx, P.visco_coef);
        ty = mad2(a.py, P.half_spiky, a.vy, P.visco_coef);
        tz = mad2(a.pz, P.half_spiky, a.vz, P.visco_coef);
    }
    const float gx = a.gx * P.grad_color_scale;
    const float gy = a.gy * P.grad_color_scale;
    const float gz = a.gz * P.grad_color_scale;
    float lap = a.lap * P.lplc_color_scale;
    lap *= p.w;   // 1/rho_i
    float sx = 0.f, sy = 0.f, sz = 0.f;
    const float n2 = dot3(gx, gy, gz, gx, gy, gz);
    if (sms) {
        // force_kernels.cu:1030-1043
        const float inv_n = rsqrtf(n2);
        const float nrm = n2 * inv_n;
        if (nrm > P.surface_normal) {
            const float s = P.surface_coe * lap * inv_n;
            sx = gx * s;
            sy = gy * s;
            sz = gz * s;
        }
    } else {
        // force_kernels.cu:796-805
        const float nrm = sqrtf(n2);
        if (nrm > P.surface_normal) {
            sx = gx * P.surface_coe * lap / nrm;
            sy = gy * P.surface_coe * lap / nrm;
            sz = gz * P.surface_coe * lap / nrm;
        }
    }
    tx *= P.mass;
    ty *= P.mass;
    tz *= P.mass;
    const float4 acc = make_float4(tx + sx, ty + sy, tz + sz, 0.f);
    if (f.acc) f.acc[self] = acc;   // null in the fused frames of a step but its last
    if (f.pos_next) {
        float4 po, vo, eo;
        integrate_one(p, f.vel[self], pev, acc.x, acc.y, acc.z, P, G, po, vo, eo);
        f.pos_next[self] = po;
        f.vel_next[self] = vo;
        f.ev_next[self] = eo;
        if (f.hash_next && !sms) {   // SMS particles: launch_hash_sms
            const uint32_t key = micro_key(po, P, G, f.ctr, self);
            f.key_in[self] = key;
            f.slot[self] = cell_slot(f.cell_count, key >> 6, __activemask());
        }
    }
}

// Cell-array bytes past which the TRA density pass prefetches its rows'
// offsets: about half of the GB300's L2.
constexpr size_t kRowPrefetchCellBytes = size_t(64) << 20;

// Up to how many work units (32 particles) per SM the small-scene builds run:
// k_density_tra_rows with a row per warp and with three rows per warp, the four
// lanes per particle of k_force_tra_quad and the small build of k_force_tra.
// The blocks per SM decide, all of which run at once. A row per warp gives way
// where units start to wait (5 per SM), three rows where some SMs have a fourth
// block and the others three (9 to 11, where the single rows are ahead again), and
// for good at a seventh (18). Force: the four lanes are ahead to 4 units in graphs
// and to 5 kernel by kernel, and the line keeps the latter. An SM runs 22 warps
// of the small build at once and 32 of the general one: the general one is better
// from where the small one needs a second wave until it needs one itself; from 34
// to 40 units both do, and the small one's is the fuller. Frames in CUDA graphs on
// 152 SMs, the dam break, us (three runs, 0.1 to 0.5 apart):
//   units per SM            1.6   3.6   4.5   5.0   5.6   8.8   9.6  10.4  12.2  15.2  17.5  18.7
//   density, row per warp  28.0  31.7  38.4  40.7  41.9  47.4  46.7  51.7  53.6  59.8  63.5  66.6
//   density, three rows    31.4  34.4  40.9  38.8  38.7  44.3  50.3  51.8  54.3  56.3  58.1  69.0
//   density, general       44.8  49.1  55.5  52.8  53.0  56.9  56.1  57.3  58.3  61.5  63.8  66.2
//   units per SM            1.6   3.6   4.0   4.5   5.0   5.6  13.2  17.5  20.0
//   force, four lanes      28.0  31.0  37.6  38.2  40.7  41.0  63.0  71.4  81.3
//   force, small           33.5  34.6  35.7  37.1  38.7  38.7  54.0  58.0  66.7
//   force, general         36.9  39.3        41.2  43.5  43.5  60.5  65.4  72.9
//   units per SM           21.3  22.7  25.7  28.9  32.4  34.2  36.1  38.1  40.1  42.2  44.4  53.9
//   force, small           75.8  78.5  80.5  83.8  84.7  87.6  87.5  92.9  91.7 101.4 100.8 112.9
//   force, general         75.5  76.5  77.0  78.7  80.7  87.8  89.7  95.2  92.2  98.0  97.1 110.3
// The same fluid in motion agrees (row per warp / three rows at 9.6 units 55.6 /
// 59.2, at 12.2 58.2 / 57.7; four lanes / small at 4.0 37.7 / 36.6; small / general at
// 22.7 83.0 / 80.6, at 38.1 95.4 / 99.3, at 42.2 105.7 / 103.4), and so do frames
// launched kernel by kernel, but for the four lanes (four lanes / small at 4.0
// 41.7 / 43.7, 4.5 43.3 / 44.8, 5.0 47.8 / 49.2, 5.6 49.7 / 49.2; row per warp / three
// rows at 9.6 55.1 / 59.5, 12.2 62.9 / 62.7; small / general at 20.0 76.2 / 78.6, 21.3
// 83.4 / 81.2, 36.1 95.6 / 96.0, 42.2 107.8 / 104.8).
constexpr int kRowsMax1 = 5, kRowsAgain1 = 9, kRowsAgainMax1 = 11;
constexpr int kRowsMax3 = 18;
constexpr int kForceQuadMax = 5;
constexpr int kForceSmallMax = 21, kForceSmallAgain = 34, kForceSmallAgainMax = 40;
// From how many units per SM a host step's force pass goes in parts
// (System::force_downloading): a part costs launches and a tail, and has to be worth
// it. Host steps, us, whole / in parts:
//   units per SM          27       44       54       65       77       90      105      206
//   one at a time    169/197  208/218  235/246  262/268  298/296  336/324  379/355  663/599
//   queued           139/171  176/196  193/219  215/241  240/258  265/280  299/307  530/512
constexpr int kForcePartsMin = 76;
// From how many units per SM the SMS side is put first in line (tra_fills).
// Frames with the TRA side first / the SMS side first, us (three runs, 0.1 to 0.7
// apart): in graphs, kernel by kernel, and the same for the fluid in motion, which
// has a few SMS tasks:
//   units per SM        54            105            140            206             811
//   graphs        107.3/109.2    168.7/170.1    217.4/215.9    297.7/296.5   1042.8/1036.8
//   by kernel     114.0/115.5    175.7/177.3    232.0/223.1    315.2/303.9   1071.2/1045.1
//   motion        120.7/120.7    185.2/180.0    232.8/226.4    321.9/314.9   1124.9/1112.9
//   by kernel     135.8/126.9    209.1/187.6    260.8/234.3    353.1/322.9   1160.9/1121.8
// (Below the line it pays with SMS work and costs 1 to 2 us without.)
constexpr int kTraFills = 128;

// Warps per block of the density and force kernels: 8 by default; each
// kernel is also built for 4 (gsph_tuning.warps_per_block), with twice the
// CTAs per SM for the same occupancy.
constexpr int kWarpsPerBlock = 8;
// Coordinate of padding candidates: far outside any kernel radius.
constexpr float kFar = 1.0e18f;

// Next work unit of a warp from a device counter (one atomic per unit).
__device__ __forceinline__ int next_unit(int *counter) {
    int u = 0;
    if ((threadIdx.x & 31) == 0) u = atomicAdd(counter, 1);
    return __shfl_sync(kFull, u, 0);
}

// ------------------------------------------------------------ density TRA --
// One particle per lane, 32 consecutive TRA particles per work unit
// (density_kernels.cu:318-366). Which candidates of each row interact is also
// recorded as a bit mask for the force pass.
//
// kRowPrefetch: each lane first prefetches its nine rows' cell offsets and
// slab words into L1, so that the per-row set-up inside the row loop waits on
// L1 rather than DRAM. Chosen on the host when the cell arrays are too large
// to stay in L2 (large batches); otherwise the extra instructions cost more
// than they save.
//
// kMany: the build for several scenes (RowFrame).
template <int W, bool kRowPrefetch, bool kMany>
__global__ void __launch_bounds__(W * 32, 6 * kWarpsPerBlock / W)
k_density_tra(Frame f, DevParams P) {
    chain_wait();
    const int lane = threadIdx.x & 31;
    const int middle = f.ctr->middle;
    const int units = (middle + 31) >> 5;
    const bool ident = !f.ctr->any_sms;   // all TRA: compact is the identity
    for (;;) {
        const int u = next_unit(&f.ctr->work_density);
        if (u >= units) break;
        const int idx = (u << 5) + lane;
        if (idx >= middle) continue;
        const int self = ident ? idx : f.compact[idx];
        const float4 p = f.pos[self];
        const SceneGeom G = geom_of_particle(f.scenes, self);
        const MicroPos mp = micro_of(p, P, G);
        uint32_t *masks = f.nbr_mask + size_t(u) * 9 * 32 + lane;
        int incomplete = 0;
        int found = 0;
        float sum = 0.f;
        const float cut = P.h2 - kFloatSmall;
        const uint32_t cut_bits = __float_as_uint(cut);
        if (kRowPrefetch) {
            const int left = mp.cx > 0 ? 1 : 0;
#pragma unroll
            for (int r = 0; r < 9; ++r) {
                const int ny = mp.cy + (r % 3) - 1;
                const int nz = mp.cz + (r / 3) - 1;
                if (ny >= 0 && ny < G.gy && nz >= 0 && nz < G.gz) {
                    const int m = G.cbase + mp.cx - left + G.gx * (ny + G.gy * nz);
                    asm volatile("prefetch.global.L1 [%0];" :: "l"(f.cell_start + m));
                    asm volatile("prefetch.global.L1 [%0];" :: "l"(f.cell_xslab + m));
                }
            }
        }
        const RowFrame rows = row_frame(mp, G);   // kMany only
        for (int r = 0; r < 9; ++r) {
            const int ny = mp.cy + (r % 3) - 1;
            const int nz = mp.cz + (r / 3) - 1;
            uint32_t mask = 0u;
            if (kMany ? (rows.flags >> r) & 1u
                      : ny >= 0 && ny < G.gy && nz >= 0 && nz < G.gz) {
                int begin, end;
                if constexpr (kMany)
                    tra_row_range(f, rows,
                                  rows.own + ((r % 3) - 1) * rows.sy + ((r / 3) - 1) * rows.sz,
                                  begin, end);
                else
                    row_range(f, G, G.cbase + mp.cx + G.gx * (ny + G.gy * nz), mp.cx, mp.lmx,
                              mp.lmx, begin, end);
                incomplete |= (end - begin > kMaskRowMax);
                uint32_t bit = 1u;
#pragma unroll 8
                for (int j = begin; j < end; ++j, bit <<= 1) {
                    const float4 q = f.pos[j];
                    const float dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
                    const float e = sq_dist_less_small(dx, dy, dz);
                    if (__float_as_uint(e) > cut_bits) continue;
                    const float t = cut - e;
                    sum += t * t * t;
                    mask |= bit;
                }
            }
            masks[r * 32] = mask;
            found += __popc(mask);
        }
        f.nbr_flag[idx] = incomplete ? -1 : found;
        write_density(f, P, self, sum, false);
    }
}

// The same for small scenes, with the nine rows of a work unit spread over
// 9 / kRows warps: a lane that walks its nine rows one after the other waits
// on some forty dependent loads, which is all the time there is when the GPU
// holds fewer units than warps. The row warps find the masks and leave the
// interacting candidates' h^2 - r^2 in shared memory (up to kRowTerms per
// row); the unit's first warp then adds the terms in the order, and with the
// operations, of k_density_tra, so both give the same bits.
constexpr int kRowTerms = 12;
template <int kRows>
__global__ void __launch_bounds__(288, kRows == 1 ? 5 : 3)
k_density_tra_rows(Frame f, DevParams P) {
    chain_wait();
    constexpr int kWarps = 9 / kRows;       // per unit
    constexpr int kUnits = 9 / kWarps;      // per block of 9 warps
    __shared__ float row_term[kUnits][9][kRowTerms][32];
    __shared__ uint32_t row_mask[kUnits][9][32];
    __shared__ int2 row_range_sh[kUnits][9][32];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int lu = warp / kWarps, part = warp % kWarps;
    const int middle = f.ctr->middle;
    const int u = blockIdx.x * kUnits + lu;
    const int idx = (u << 5) + lane;
    if (blockIdx.x * (kUnits << 5) >= middle) return;   // the whole block
    const bool active = idx < middle;
    const float cut = P.h2 - kFloatSmall;
    const uint32_t cut_bits = __float_as_uint(cut);
    int self = 0;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (active) {
        self = f.ctr->any_sms ? f.compact[idx] : idx;
        p = f.pos[self];
        const SceneGeom G = geom_of_particle(f.scenes, self);
        const MicroPos mp = micro_of(p, P, G);
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const int r = part * kRows + k;
            const int ny = mp.cy + (r % 3) - 1;
            const int nz = mp.cz + (r / 3) - 1;
            uint32_t mask = 0u;
            int begin = 0, end = 0;
            if (ny >= 0 && ny < G.gy && nz >= 0 && nz < G.gz) {
                row_range(f, G, G.cbase + mp.cx + G.gx * (ny + G.gy * nz), mp.cx, mp.lmx,
                          mp.lmx, begin, end);
                const int n = min(end - begin, kMaskRowMax);
                int terms = 0;
#pragma unroll 8
                for (int j = 0; j < n; ++j) {
                    const float4 q = f.pos[begin + j];
                    const float e = sq_dist_less_small(p.x - q.x, p.y - q.y, p.z - q.z);
                    if (__float_as_uint(e) > cut_bits) continue;
                    if (terms < kRowTerms) row_term[lu][r][terms][lane] = cut - e;
                    ++terms;
                    mask |= 1u << j;
                }
            }
            row_mask[lu][r][lane] = mask;
            row_range_sh[lu][r][lane] = make_int2(begin, end);
        }
    }
    __syncthreads();
    if (part != 0 || !active) return;
    uint32_t *masks = f.nbr_mask + size_t(u) * 9 * 32 + lane;
    int found = 0;
    bool incomplete = false;
    float sum = 0.f;
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        uint32_t mask = row_mask[lu][r][lane];
        const int2 range = row_range_sh[lu][r][lane];
        const int n = __popc(mask);
        masks[r * 32] = mask;
        found += n;
        for (int k = 0; k < min(n, kRowTerms); ++k) {
            const float t = row_term[lu][r][k][lane];
            sum += t * t * t;
        }
        auto add = [&](int j) {
            const float4 q = f.pos[j];
            const float e = sq_dist_less_small(p.x - q.x, p.y - q.y, p.z - q.z);
            if (__float_as_uint(e) > cut_bits) return;
            const float t = cut - e;
            sum += t * t * t;
        };
        if (n > kRowTerms) {
            for (int k = 0; k < kRowTerms; ++k) mask &= mask - 1u;
            for (; mask; mask &= mask - 1u) add(range.x + __ffs(mask) - 1);
        }
        if (range.y - range.x > kMaskRowMax) {
            incomplete = true;
            for (int j = range.x + kMaskRowMax; j < range.y; ++j) add(j);
        }
    }
    f.nbr_flag[idx] = incomplete ? -1 : found;
    write_density(f, P, self, sum, false);
}

// ------------------------------------------------------- SMS candidates --
// An SMS task's 32 particles are taken as clusters of C consecutive ones. A
// warp works on one cluster: lane = (group g = lane / C, particle i = lane %
// C), and the 32 / C groups share the cluster's candidates between them.
// Consecutive particles of a cell lie close together (the sort order is
// micro-x, micro-z, micro-y), so a small cluster's bounding box is small and
// most candidates within h of the box interact with a given particle of it:
// in the default scene (spacing 0.15 h, 1,237 neighbours per particle) 70 /
// 56 / 46 / 40% for clusters of 4 / 8 / 16 / 32, of 1,764 / 2,197 / 2,693 /
// 3,127 listed out of 4,155 / 4,481 / 4,861 / 5,343 tested. The pair
// arithmetic is bound by the FP32 pipe and wants small clusters, the testing
// by issue slots and wants large ones, and small scenes want many units:
// force, 3.94M particles 14.0 / 12.5 ms and 64,000 particles 260 / 277 us at
// C = 8 / 16 (with two packed operations a pair less than now: 12.8 ms at 16);
// density 6.8 / 5.2 / 4.8 ms and 146 / 154 / 165 us at 8 / 16 / 32. Whole tasks
// without the box test took 16.3 ms and 690 us (force), 6.7 ms and 230 us
// (density).
//
// Candidates are pruned twice before a pair is evaluated:
//  * by micro cells: micro-x slab s of a neighbour cell keeps only the
//    micro-z groups whose gap to the cluster's own micro cells, gx, gy, gz in
//    quarters of h (gy of the whole cell), has gx^2 + gy^2 + gz^2 < 16: a
//    particle beyond that is at least h away;
//  * by the box: a candidate is listed only if its distance from the
//    cluster's bounding box is at most h.
// Both leave every interacting candidate in, in increasing sorted index per
// row, rows z-major as in the reference.
struct ClusterBox {
    float cx, cy, cz, ex, ey, ez;       // a point inside, half extents from it
    int x0, x1, y0, y1, z0, z1;         // micro cells inside the cell, [0, 3]
};

// A position no farther than kFar, from where no squared distance overflows: a
// particle outside the grid may be anywhere, and a cluster's box with it. (Box
// widening, this and the position read again at the end: 3.94M dense particles
// 20.3 -> 20.1 ms a host step, 64,000 498 -> 485 us; the box test given its own margin
// instead 20.5 ms, stray clusters scanned apart 20.6.)
__device__ __forceinline__ float4 on_scale(float4 p) {
    p.x = fminf(fmaxf(p.x, -kFar), kFar);
    p.y = fminf(fmaxf(p.y, -kFar), kFar);
    p.z = fminf(fmaxf(p.z, -kFar), kFar);
    return p;
}

__device__ __forceinline__ float warp_max(float v) {   // v >= 0
    return __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(v)));
}

__device__ __forceinline__ ClusterBox cluster_box(const float4 &p, uint32_t key) {
    ClusterBox b;
    float l[3] = {p.x, p.y, p.z}, h[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            l[a] = fminf(l[a], __shfl_xor_sync(kFull, l[a], o));
            h[a] = fmaxf(h[a], __shfl_xor_sync(kFull, h[a], o));
        }
    b.cx = 0.5f * (l[0] + h[0]);
    b.cy = 0.5f * (l[1] + h[1]);
    b.cz = 0.5f * (l[2] + h[2]);
    // wider by four roundings: a particle outside the grid, clamped into the cell,
    // may stretch the box until its differences round by more than h
    const float wider = 1.f + 4.f / 16777216.f;
    b.ex = wider * warp_max(fabsf(p.x - b.cx));
    b.ey = wider * warp_max(fabsf(p.y - b.cy));
    b.ez = wider * warp_max(fabsf(p.z - b.cz));
    const uint32_t m = __reduce_or_sync(kFull, (1u << ((key >> 4) & 3u)) |
                                                   (16u << (key & 3u)) |
                                                   (256u << ((key >> 2) & 3u)));
    const uint32_t mx = m & 15u, my = (m >> 4) & 15u, mz = m >> 8;
    b.x0 = __ffs(mx) - 1;
    b.x1 = 31 - __clz(mx);
    b.y0 = __ffs(my) - 1;
    b.y1 = 31 - __clz(my);
    b.z0 = __ffs(mz) - 1;
    b.z1 = 31 - __clz(mz);
    return b;
}

// The clusters of one warp. Where there are fewer than warps, each block takes
// as many as the others (a queue would fill the first blocks to the last warp
// and leave later ones idle: density of 64,000 dense particles 146 us against
// 128); else they come from the queue. Negative: done.
struct ClusterUnits {
    int count, per, own;
    // blocks: those of the grid that run at once
    __device__ __forceinline__ ClusterUnits(int units, int warps, int blocks)
        : count(units) {
        per = (units + blocks - 1) / blocks;
        const int warp = threadIdx.x >> 5;
        own = per > warps ? -2
              : warp < per && int(blockIdx.x) < blocks ? int(blockIdx.x) * per + warp
                                                       : -1;
    }
    __device__ __forceinline__ int next(int *queue) {
        int u = own;
        if (u == -2)
            u = next_unit(queue);
        else
            own = -1;
        return u < count ? u : -1;
    }
};

// Shared memory of one warp's candidate stream.
constexpr int kSegMax = 27 * 4;    // a segment per neighbour cell and micro-x slab
constexpr int kBatch = 128;        // candidates staged and evaluated at a time
struct __align__(16) ClusterLists {
    int2 seg[kSegMax];             // candidate ranges [x, y)
    int idx[kBatch + 64];          // listed candidates
};
static_assert(kBatch % 64 == 0, "whole pairs per lane");

// The candidate ranges of a cluster after the micro-cell pruning, one
// neighbour cell per lane (27 of 32); returns their number.
__device__ __forceinline__ int cluster_segments(const Frame &f, const SceneGeom &G,
                                                const gsph_block_task &task,
                                                const ClusterBox &b, int lane,
                                                int2 *__restrict__ seg) {
    const int dx = lane % 3 - 1, dy = lane / 3 % 3 - 1, dz = lane / 9 - 1;
    const int x = task.cell_pos[0] + dx, y = task.cell_pos[1] + dy, z = task.cell_pos[2] + dz;
    int2 own[4];
    int n = 0;
    if (lane < 27 && x >= 0 && x < G.gx && y >= 0 && y < G.gy && z >= 0 && z < G.gz) {
        const int c = G.cbase + x + G.gx * (y + G.gy * z);
        const int cs = f.cell_start[c];
        const int cnt = f.cell_start[c + 1] - cs;
        if (cnt > 0) {
            const uint16_t *g = f.cell_grp + size_t(c) * 16;
            const int gy = dy < 0 ? b.y0 : dy > 0 ? 3 - b.y1 : 0;
            if (g[0] == kGroupsUnknown) {   // > 65,535 particles: taken whole
                own[0] = make_int2(cs, cs + cnt);
                n = 1;
            } else {
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const int rx = 4 * dx + s;
                    const int gx = max(0, max(rx - b.x1, b.x0 - rx) - 1);
                    const int room = 15 - gx * gx - gy * gy;   // gz^2 <= room
                    const int gz = room >= 9 ? 3 : room >= 4 ? 2 : room >= 1 ? 1 : 0;
                    const int zlo = max(0, b.z0 - 1 - gz - 4 * dz);
                    const int zhi = min(3, b.z1 + 1 + gz - 4 * dz);
                    const bool some = room >= 0 && zlo <= zhi;
                    const int lo = min(4 * s + zlo, 15), hi = 4 * s + zhi + 1;
                    const int first = cs + min(some ? int(g[lo]) : 0, cnt);
                    const int last =
                        cs + (some ? (hi < 16 ? min(int(g[max(hi, 0)]), cnt) : cnt) : 0);
                    own[s] = make_int2(first, some ? last : first);
                }
                // slabs that continue one another become one range
                int m = 0;
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const int2 v = own[s];
                    if (v.y <= v.x) continue;
                    if (m > 0 && own[0].y == v.x && m == 1) {
                        own[0].y = v.y;
                    } else if (m > 1 && own[1].y == v.x && m == 2) {
                        own[1].y = v.y;
                    } else if (m > 2 && own[2].y == v.x && m == 3) {
                        own[2].y = v.y;
                    } else {
                        if (m == 0) own[0] = v;
                        if (m == 1) own[1] = v;
                        if (m == 2) own[2] = v;
                        if (m == 3) own[3] = v;
                        ++m;
                    }
                }
                n = m;
            }
        }
    }
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
    }
    const int at = incl - n;
#pragma unroll
    for (int s = 0; s < 4; ++s)
        if (s < n) seg[at + s] = own[s];
    __syncwarp();
    return __shfl_sync(kFull, incl, 31);
}

// Streams a cluster's candidates: two runs of 32 positions are loaded
// together and tested against the box (one candidate per lane), the indices
// that pass are compacted into a list, and kBatch of them at a time are
// staged and evaluated. fill(k, a, b) stages the pair k (one pair per lane, so
// that the gathers are dense and in flight together) from the indices a and
// b, where -1 stands for a candidate that interacts with nothing; run(n)
// takes the first n * (32 / C) pairs, each group every (32 / C)-th of them.
// Control flow is warp-uniform.
template <int C, class Fill, class Run>
__device__ __forceinline__ void cluster_stream(const Frame &f, const SceneGeom &G,
                                               const gsph_block_task &task,
                                               const ClusterBox &box, float h2, int lane,
                                               ClusterLists &ls, Fill fill, Run run) {
    constexpr int kStep = 2 * (32 / C);   // candidates per iteration of run
    static_assert(kBatch % kStep == 0, "a batch is whole iterations");
    const int nseg = cluster_segments(f, G, task, box, lane, ls.seg);
    const unsigned lt = lanemask_lt();
    // differences of coordinates round to 2^-24 of themselves, so 1e-5 of h^2
    // covers the test's rounding (beside the box's own, see cluster_box)
    const float reach = h2 * 1.00001f;
    auto near = [&](const float4 &q) {
        const float ax = fmaxf(fabsf(q.x - box.cx) - box.ex, 0.f);
        const float ay = fmaxf(fabsf(q.y - box.cy) - box.ey, 0.f);
        const float az = fmaxf(fabsf(q.z - box.cz) - box.ez, 0.f);
        return sq_dist(ax, ay, az) <= reach;
    };
    int cnt = 0;
    auto batch = [&](int n) {   // stage and evaluate the first n listed
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kBatch / 2; q += 32) {
            const int2 ab = *reinterpret_cast<const int2 *>(ls.idx + 2 * (q + lane));
            fill(q + lane, 2 * (q + lane) < n ? ab.x : -1, 2 * (q + lane) + 1 < n ? ab.y : -1);
        }
        __syncwarp();
        run((n + kStep - 1) / kStep);
        __syncwarp();
    };
    for (int k = 0; k < nseg; ++k) {
        const int2 sg = ls.seg[k];
        for (int j0 = sg.x; j0 < sg.y; j0 += 64) {
            const int ja = j0 + lane, jb = ja + 32;
            const float4 qa = f.pos[min(ja, sg.y - 1)];
            const float4 qb = f.pos[min(jb, sg.y - 1)];
            const bool ina = ja < sg.y && near(qa);
            const bool inb = jb < sg.y && near(qb);
            const unsigned ha = __ballot_sync(kFull, ina);
            const unsigned hb = __ballot_sync(kFull, inb);
            const int na = cnt + __popc(ha);
            if (ina) ls.idx[cnt + __popc(ha & lt)] = ja;
            if (inb) ls.idx[na + __popc(hb & lt)] = jb;
            cnt = na + __popc(hb);
            if (cnt >= kBatch) {
                batch(kBatch);
                cnt -= kBatch;   // at most 63 stay
                int v0 = 0, v1 = 0;
                if (lane < cnt) v0 = ls.idx[kBatch + lane];
                if (lane + 32 < cnt) v1 = ls.idx[kBatch + lane + 32];
                __syncwarp();
                if (lane < cnt) ls.idx[lane] = v0;
                if (lane + 32 < cnt) ls.idx[lane + 32] = v1;
            }
        }
    }
    if (cnt > 0) batch(cnt);
    __syncwarp();
}

// ------------------------------------------------------------ density SMS --
// One cluster of kDenCluster particles per warp (density_kernels.cu:368-565).
// Bound by issue slots, about two fifths of them in the candidate tests
// and the staging.
// Candidates are staged as pairs (slots 2k, 2k+1), an (x, x, y, y) float4 and
// a (z, z) float2, and evaluated two at a time with packed FP32x2 arithmetic
// and the TRA pass's one-compare cut-off test; the groups' sums are added at
// the end.
constexpr int kDenCluster = 16;
template <int W>
__global__ void __launch_bounds__(W * 32, 4 * kWarpsPerBlock / W)
k_density_sms(Frame f, DevParams P) {
    constexpr int C = kDenCluster, kGroups = 32 / C;
    // candidate pair k (slots 2k, 2k+1): (x, x, y, y) and (z, z)
    __shared__ __align__(16) float4 sms_xy[W][kBatch / 2];
    __shared__ __align__(16) float2 sms_zz[W][kBatch / 2];
    __shared__ ClusterLists lists[W];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int task_count = f.ctr->task_count;
    if (task_count == 0) return;   // no SMS work: skip the queue atomics
    float4 *sxy = sms_xy[warp];
    float2 *szz = sms_zz[warp];
    const int i = lane % C, g = lane / C;
    ClusterUnits units(task_count * kGroups, W, gridDim.x);
    for (int u; (u = units.next(&f.ctr->work_density_sms)) >= 0;) {
        const gsph_block_task task = f.tasks[u / kGroups];
        const int first = task.cell_begin + task_offset(task) + (u % kGroups) * C;
        const int cend = task.cell_begin + task.cell_particle_count;
        if (first >= cend) continue;   // warp-uniform
        const int self = min(first + i, cend - 1);
        const float4 p = on_scale(f.pos[self]);
        const SceneGeom G = geom_of_cell(f.scenes, task.cellid);
        const ClusterBox box = cluster_box(p, f.key[self]);
        const float2 npx = make_float2(-p.x, -p.x);
        const float2 npy = make_float2(-p.y, -p.y);
        const float2 npz = make_float2(-p.z, -p.z);
        const float cut = P.h2 - kFloatSmall;
        const uint32_t cut_bits = __float_as_uint(cut);
        const float2 cutv = make_float2(cut, cut);
        const float2 msm = make_float2(-kFloatSmall, -kFloatSmall);
        const float2 m1 = make_float2(-1.f, -1.f);
        float2 acc = make_float2(0.f, 0.f);
        const float4 far = make_float4(kFar, kFar, kFar, 0.f);
        cluster_stream<C>(
            f, G, task, box, P.h2, lane, lists[warp],
            [&](int k, int ja, int jb) {
                const float4 a = ja < 0 ? far : f.pos[ja];
                const float4 b = jb < 0 ? far : f.pos[jb];
                sxy[k] = make_float4(a.x, b.x, a.y, b.y);
                szz[k] = make_float2(a.z, b.z);
            },
            [&](int n) {
#pragma unroll 8
                for (int k = 0; k < n; ++k) {
                    const float4 qa = sxy[k * kGroups + g];
                    const float2 dx = __fadd2_rn(make_float2(qa.x, qa.y), npx);
                    const float2 dy = __fadd2_rn(make_float2(qa.z, qa.w), npy);
                    const float2 dz = __fadd2_rn(szz[k * kGroups + g], npz);
                    // the cut-off test of sq_dist_less_small, per half
                    float2 e = __ffma2_rn(dx, dx, msm);
                    e = __ffma2_rn(dy, dy, e);
                    e = __ffma2_rn(dz, dz, e);
                    float2 t = __ffma2_rn(e, m1, cutv);
                    t.x = __float_as_uint(e.x) > cut_bits ? 0.f : t.x;
                    t.y = __float_as_uint(e.y) > cut_bits ? 0.f : t.y;
                    acc = __ffma2_rn(__fmul2_rn(t, t), t, acc);
                }
            });
        float sum = acc.x + acc.y;
#pragma unroll
        for (int o = C; o < 32; o <<= 1) sum += __shfl_xor_sync(kFull, sum, o);
        if (g == 0 && first + i < cend) write_density(f, P, self, sum, true);
    }
}

// -------------------------------------------------------------- force TRA --
// All candidates of a particle, tested as the reference does.
template <bool kArt>
__device__ __forceinline__ void force_scan(const Frame &f, const DevParams &P,
                                           const SceneGeom &G, const MicroPos &mp,
                                           const float4 &p, const float4 &pev, ForceAcc &a) {
    for (int r = 0; r < 9; ++r) {
        const int ny = mp.cy + (r % 3) - 1;
        const int nz = mp.cz + (r / 3) - 1;
        if (ny < 0 || ny >= G.gy || nz < 0 || nz >= G.gz) continue;
        const int m = G.cbase + mp.cx + G.gx * (ny + G.gy * nz);
        int begin, end;
        row_range(f, G, m, mp.cx, mp.lmx, mp.lmx, begin, end);
        for (int j = begin; j < end; ++j) {
            const float4 q = f.pos[j];
            const float rx = p.x - q.x, ry = p.y - q.y, rz = p.z - q.z;
            const float d2 = sq_dist(rx, ry, rz);
            if (P.h2 < d2 || kFloatSmall > d2) continue;
            force_pair<true, kArt>(p, pev, q, f.ev[j], P, a);
        }
    }
}

// Start of row r's candidate range (tra_row_range's and row_range's begin), from
// the particle's own cell `own`; a row without neighbours reads the own cell.
__device__ __forceinline__ int row_begin(const Frame &f, const SceneGeom &G,
                                         const MicroPos &mp, int own, int r, uint32_t mask) {
    const int left = mp.cx > 0 ? 1 : 0;
    const int m = mask ? own + G.gx * ((r % 3) - 1 + G.gy * ((r / 3) - 1)) : own;
    const int s0 = f.cell_start[m - left];
    const int s1 = f.cell_start[m];
    const uint32_t xs = f.cell_xslab[m - left];
    if (left && mp.lmx > 0 && xs != kXslabUnknown)
        return s0 + min(int((xs >> (10 * (mp.lmx - 1))) & 1023u), s1 - s0);
    return s0;
}

// The neighbours the density pass found, in the same order (rows in sequence,
// set bits in increasing candidate index). Each lane stages its 9 (row start,
// mask) pairs in shared memory and walks all its neighbours in one loop, so
// lanes stay converged across rows. Without masks (or with a row longer than
// 32 candidates) the lane scans its candidates as the reference does.
//
// kSmall: the build for scenes with fewer work units than the GPU holds
// warps. Each warp takes the unit of its index (no queue: thousands of idle
// warps taking turns on one counter cost more than the work), and four
// neighbours' loads instead of two are in flight before the first of them is
// evaluated (the order of the sums is unchanged).
//
// kPart: only the units of `part`.
template <bool kArt, int W, bool kSmall = false, bool kPart = false>
__global__ void __launch_bounds__(W * 32, kSmall ? 1 : 4 * kWarpsPerBlock / W)
k_force_tra(Frame f, DevParams P, bool fresh, ForcePart part) {
    __shared__ uint32_t row_mask[9][W * 32];
    __shared__ int row_start[9][W * 32];
    const int lane = threadIdx.x & 31;
    const int middle = f.ctr->middle;
    const int units = (middle + 31) >> 5;
    const bool ident = !f.ctr->any_sms;   // all TRA: compact is the identity
    if (units == 0) return;        // no TRA work: skip the queue atomics
    for (bool first = true;; first = false) {
        if (kSmall && !first) break;
        const int u = kSmall  ? int(blockIdx.x * W + (threadIdx.x >> 5))
                      : kPart ? part.begin + next_unit(&f.ctr->work_force_part[part.queue])
                              : next_unit(&f.ctr->work_force);
        if (u >= (kPart ? min(units, part.end) : units)) break;
        const int idx = (u << 5) + lane;
        if (idx >= middle) continue;
        const int self = ident ? idx : f.compact[idx];
        const float4 p = f.pos[self];
        const float4 pev = f.ev[self];
        const SceneGeom G = geom_of_particle(f.scenes, self);
        const MicroPos mp = micro_of(p, P, G);
        ForceAcc a = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const int found = fresh ? f.nbr_flag[idx] : -1;
        if (found >= 0) {
            // all nine masks, then every row's offsets and slab word, loaded
            // without conditions (a row without neighbours reads the
            // particle's own cell) so that the loads are in flight together
            const uint32_t *masks = f.nbr_mask + size_t(u) * 9 * 32 + lane;
            uint32_t mk[9];
#pragma unroll
            for (int r = 0; r < 9; ++r) mk[r] = masks[r * 32];
            const int own = G.cbase + mp.cx + G.gx * (mp.cy + G.gy * mp.cz);
#pragma unroll
            for (int r = 0; r < 9; ++r) {
                const int start = row_begin(f, G, mp, own, r, mk[r]);
                row_mask[r][threadIdx.x] = mk[r];
                row_start[r][threadIdx.x] = start;
            }
            int r = 0;
            uint32_t mask = row_mask[0][threadIdx.x];
            int base = row_start[0][threadIdx.x];
            // two (kSmall: four) neighbours per iteration: their loads are in
            // flight before the first pair is evaluated (the order of the sums
            // is unchanged)
            if constexpr (kSmall) {
                for (int k = 0; k < found; k += 4) {
                    float4 q[4], e[4];
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        int j = self;
                        if (k + s < found) {
                            while (!mask) {
                                ++r;
                                mask = row_mask[r][threadIdx.x];
                                base = row_start[r][threadIdx.x];
                            }
                            j = base + __ffs(mask) - 1;
                            mask &= mask - 1u;
                        }
                        q[s] = f.pos[j];
                        e[s] = f.ev[j];
                    }
#pragma unroll
                    for (int s = 0; s < 4; ++s)
                        if (k + s < found) force_pair<false, kArt>(p, pev, q[s], e[s], P, a);
                }
            } else {
                int k = 0;
                for (; k + 1 < found; k += 2) {
                    while (!mask) {
                        ++r;
                        mask = row_mask[r][threadIdx.x];
                        base = row_start[r][threadIdx.x];
                    }
                    const int j0 = base + __ffs(mask) - 1;
                    mask &= mask - 1u;
                    while (!mask) {
                        ++r;
                        mask = row_mask[r][threadIdx.x];
                        base = row_start[r][threadIdx.x];
                    }
                    const int j1 = base + __ffs(mask) - 1;
                    mask &= mask - 1u;
                    const float4 q0 = f.pos[j0], e0 = f.ev[j0];
                    const float4 q1 = f.pos[j1], e1 = f.ev[j1];
                    force_pair<false, kArt>(p, pev, q0, e0, P, a);
                    force_pair<false, kArt>(p, pev, q1, e1, P, a);
                }
                if (k < found) {
                    while (!mask) {
                        ++r;
                        mask = row_mask[r][threadIdx.x];
                        base = row_start[r][threadIdx.x];
                    }
                    const int j = base + __ffs(mask) - 1;
                    force_pair<false, kArt>(p, pev, f.pos[j], f.ev[j], P, a);
                }
            }
        } else {
            force_scan<kArt>(f, P, G, mp, p, pev, a);
        }
        write_force(f, P, self, p, pev, G, a, false);
    }
}

// The same for the smallest scenes, four lanes per particle: with one lane, a
// warp alone on its scheduler spends the pass in rounds of neighbour loads.
// The lanes list the particle's neighbours together, each evaluates every
// fourth of them (the next round's loads in flight), and the terms change
// hands through shared memory so that each lane keeps one of the four sums
// (pressure, viscosity, gradient, laplacian) and adds its terms in neighbour
// order with k_force_tra's operations: the same bits.
constexpr int kQuadList = 64;   // neighbours listed; with more the first lane walks all
template <bool kArt>
__global__ void __launch_bounds__(128)
k_force_tra_quad(Frame f, DevParams P, bool fresh) {
    __shared__ int list[4][8][kQuadList];
    __shared__ __align__(16) float terms[4][8][4][12];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pl = lane >> 2, s = lane & 3;
    const int middle = f.ctr->middle;
    const int base = blockIdx.x * 32 + warp * 8;
    if (base >= middle) return;   // the whole warp
    const int idx = base + pl;
    const bool active = idx < middle;
    const int at = active ? idx : base;   // idle lanes follow a live particle
    const int self = f.ctr->any_sms ? f.compact[at] : at;
    const float4 p = f.pos[self];
    const float4 pev = f.ev[self];
    const SceneGeom G = geom_of_particle(f.scenes, self);
    const MicroPos mp = micro_of(p, P, G);
    int found = fresh ? f.nbr_flag[at] : -1;
    const bool listed = found >= 0 && found <= kQuadList;
    // lane s of the particle lists rows s, s + 4 and s + 8
    const uint32_t *masks = f.nbr_mask + (size_t(at >> 5) * 9) * 32 + (at & 31);
    uint32_t mk[3];
    int start[3], cnt[3];
    const int own = G.cbase + mp.cx + G.gx * (mp.cy + G.gy * mp.cz);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int r = s + 4 * k;
        mk[k] = listed && r < 9 ? masks[r * 32] : 0u;
        cnt[k] = __popc(mk[k]);
        start[k] = row_begin(f, G, mp, own, r, mk[k]);
    }
    int ahead = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int incl = cnt[k];
        int v = __shfl_up_sync(kFull, incl, 1, 4);
        if (s >= 1) incl += v;
        v = __shfl_up_sync(kFull, incl, 2, 4);
        if (s >= 2) incl += v;
        int o = ahead + incl - cnt[k];
        ahead += __shfl_sync(kFull, incl, 3, 4);
        for (uint32_t m = mk[k]; m; m &= m - 1u)
            list[warp][pl][o++] = start[k] + __ffs(m) - 1;
    }
    __syncwarp();
    const int n = listed ? found : 0;
    const int rounds = (int(__reduce_max_sync(kFull, unsigned(n))) + 3) >> 2;
    float *mine = terms[warp][pl][s];
    // the lane's sum: which vector and which factor of a pair's terms
    const float *vec = terms[warp][pl][0] + (s == 1 ? 4 : s == 3 ? 8 : 0);
    const float *fac = terms[warp][pl][0] + (s == 0 ? 3 : s == 1 ? 7 : s == 2 ? 9 : 10);
    float ax = 0.f, ay = 0.f, az = 0.f;
    int j = s < n ? list[warp][pl][s] : self;
    float4 q = f.pos[j], e = f.ev[j];
    for (int k = 0; k < rounds; ++k) {
        const float4 cq = q, ce = e;
        const int next = 4 * (k + 1) + s;
        j = next < n ? list[warp][pl][next] : self;
        q = f.pos[j];
        e = f.ev[j];
        const PairTerms t = pair_terms<kArt>(p, pev, cq, ce, P);
        *reinterpret_cast<float4 *>(mine) = make_float4(t.rx, t.ry, t.rz, -t.ps);
        *reinterpret_cast<float4 *>(mine + 4) = make_float4(t.ux, t.uy, t.uz, t.wk);
        *reinterpret_cast<float4 *>(mine + 8) = make_float4(t.lf, t.gw, t.wh, 0.f);
        __syncwarp();
        // terms past the particle's neighbours (of a lane paired with itself) are
        // skipped, not weighted by zero: the velocity may not be finite
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (4 * k + i >= n) continue;
            const float4 v = *reinterpret_cast<const float4 *>(vec + 12 * i);
            const float w = fac[12 * i];
            ax = __fmaf_rn(v.x, w, ax);
            ay = __fmaf_rn(v.y, w, ay);
            az = __fmaf_rn(v.z, w, az);
        }
        __syncwarp();
    }
    ForceAcc a;
    a.px = ax;
    a.py = ay;
    a.pz = az;
    a.vx = __shfl_down_sync(kFull, ax, 1);
    a.vy = __shfl_down_sync(kFull, ay, 1);
    a.vz = __shfl_down_sync(kFull, az, 1);
    a.gx = __shfl_down_sync(kFull, ax, 2);
    a.gy = __shfl_down_sync(kFull, ay, 2);
    a.gz = __shfl_down_sync(kFull, az, 2);
    a.lap = __shfl_down_sync(kFull, ax, 3);
    if (s != 0 || !active) return;
    if (!listed) {   // (the sums are zero)
        if (found < 0) {
            force_scan<kArt>(f, P, G, mp, p, pev, a);
        } else {   // the masks decide, as in k_force_tra: the scan's test rounds otherwise
            for (int r = 0; r < 9; ++r) {
                const uint32_t mask = masks[r * 32];
                const int from = row_begin(f, G, mp, own, r, mask);
                for (uint32_t m = mask; m; m &= m - 1u) {
                    const int at_j = from + __ffs(m) - 1;
                    force_pair<false, kArt>(p, pev, f.pos[at_j], f.ev[at_j], P, a);
                }
            }
        }
    }
    write_force(f, P, self, p, pev, G, a, false);
}

// -------------------------------------------------------------- force SMS --
// One cluster of kForceCluster particles per warp (force_kernels.cu:830-1054),
// over the density pass's candidates. Bound by the FP32 pipe (67% busy with 3.94M
// dense particles, 12.8 ms; most instructions of a pair step are packed and hold
// it for two cycles) and, beside it, by the candidate tests. Three blocks per SM,
// 80 registers: 228 bytes a thread are spilled and 92 loaded again (208 and 76
// with artificial viscosity; the position is read again at the end, which saved
// some); at four blocks, 64 registers, the pass was slower (13.3 ms against 12.5,
// before the velocities' differences were taken per pair).
// Each candidate pair is staged as four float4s (one 16-byte load per pair and
// quantity group) and evaluated with packed FP32x2 arithmetic. Each term rounds as
// the reference's scalar expression; the two halves of every accumulator and then
// the groups' sums are added at the end.
constexpr int kForceCluster = 16;
static_assert(kForceCluster == kDenCluster, "sms_blocks counts one cluster size");
// Resident blocks per SM. The grid may hold a fourth (kMaxShape), which starts
// when another leaves and finds the queue empty; a grid of three is no faster in
// dense scenes and slower where there is no SMS work (46,656 particles all TRA
// 50.0 us a frame against 46.7, from 110,592 on the same).
constexpr int kForceSmsCtas = 3;
template <bool kArt, int W>
__global__ void __launch_bounds__(W * 32, kForceSmsCtas * kWarpsPerBlock / W)
k_force_sms(Frame f, DevParams P, int resident) {
    constexpr int C = kForceCluster, kGroups = 32 / C;
    // candidate pair k (slots 2k, 2k+1) as four float4s: (x, x, y, y),
    // (z, z, 1/rho, 1/rho), (vx, vx, vy, vy), (vz, vz, p, p)
    __shared__ __align__(16) float4 sm[4][W][kBatch / 2];
    __shared__ ClusterLists lists[W];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int task_count = f.ctr->task_count;
    if (task_count == 0) return;   // no SMS work: skip the queue atomics
    float4 *sa = sm[0][warp], *sb4 = sm[1][warp], *sc = sm[2][warp], *sd = sm[3][warp];
    const int i = lane % C, g = lane / C;
    ClusterUnits units(task_count * kGroups, W, min(int(gridDim.x), resident));
    for (int u; (u = units.next(&f.ctr->work_force_sms)) >= 0;) {
        const gsph_block_task task = f.tasks[u / kGroups];
        const int first = task.cell_begin + task_offset(task) + (u % kGroups) * C;
        const int cend = task.cell_begin + task.cell_particle_count;
        if (first >= cend) continue;   // warp-uniform
        const int self = min(first + i, cend - 1);
        const float4 p = on_scale(f.pos[self]);
        const float4 pev = f.ev[self];
        const SceneGeom G = geom_of_cell(f.scenes, task.cellid);
        const ClusterBox box = cluster_box(p, f.key[self]);
        const float2 npx = make_float2(-p.x, -p.x);
        const float2 npy = make_float2(-p.y, -p.y);
        const float2 npz = make_float2(-p.z, -p.z);
        // the velocities' differences are taken pair by pair. The sum of V_j v_j
        // (h - r) less v_i times the sum of V_j (h - r) is two packed operations
        // a pair cheaper (3.94M dense particles, a whole host step, 19.9 ms
        // against 20.3), but where differences are small against the velocities
        // it loses them: 1.4e-5 of a particle's pair terms against 5e-7 with
        // fast particles among slow ones
        const float2 nvx = make_float2(-pev.x, -pev.x);
        const float2 nvy = make_float2(-pev.y, -pev.y);
        const float2 nvz = make_float2(-pev.z, -pev.z);
        const float2 pi2 = make_float2(pev.w, pev.w);
        const float2 h2v = make_float2(P.h2, P.h2);
        const float2 hv = make_float2(P.h, P.h);
        const float2 m1 = make_float2(-1.f, -1.f);
        const float2 m075 = make_float2(-0.75f, -0.75f);
        const float2 zero = make_float2(0.f, 0.f);
        // pressure sum gets -r*ps = d*ps with d = q - p; the colour
        // gradient is accumulated with the opposite sign and negated at the end
        float2 Px = zero, Py = zero, Pz = zero, Vx = zero, Vy = zero, Vz = zero;
        float2 Gx = zero, Gy = zero, Gz = zero, L = zero;
        // artificial viscosity: V_i and 0.01 h^2
        const float2 viv = make_float2(p.w, p.w);
        const float2 epsv = make_float2(P.art_eps, P.art_eps);
        // added to r^2 so that 1/r stays finite for the particle itself, whose
        // terms are zeroed; far below a rounding of any interacting r^2
        const float2 tiny = make_float2(1e-30f, 1e-30f);
        const float4 far = make_float4(kFar, kFar, kFar, 0.f);
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        cluster_stream<C>(
            f, G, task, box, P.h2, lane, lists[warp],
            [&](int k, int ja, int jb) {
                const float4 a = ja < 0 ? far : f.pos[ja];
                const float4 b = jb < 0 ? far : f.pos[jb];
                const float4 va = ja < 0 ? none : f.ev[ja];
                const float4 vb = jb < 0 ? none : f.ev[jb];
                sa[k] = make_float4(a.x, b.x, a.y, b.y);
                sb4[k] = make_float4(a.z, b.z, a.w, b.w);
                sc[k] = make_float4(va.x, vb.x, va.y, vb.y);
                sd[k] = make_float4(va.z, vb.z, va.w, vb.w);
            },
            [&](int n) {
#pragma unroll 4
                for (int k = 0; k < n; ++k) {
                    const int s = k * kGroups + g;
                    const float4 qa = sa[s], qb = sb4[s];
                    const float2 dx = __fadd2_rn(make_float2(qa.x, qa.y), npx);
                    const float2 dy = __fadd2_rn(make_float2(qa.z, qa.w), npy);
                    const float2 dz = __fadd2_rn(make_float2(qb.x, qb.y), npz);
                    float2 d2 = __ffma2_rn(dx, dx, tiny);
                    d2 = __ffma2_rn(dy, dy, d2);
                    d2 = __ffma2_rn(dz, dz, d2);
                    const float2 t = __ffma2_rn(d2, m1, h2v);   // h^2 - r^2
                    const bool okx = t.x >= 0.f && d2.x >= kFloatSmall;
                    const bool oky = t.y >= 0.f && d2.y >= kFloatSmall;
                    const float2 inv = make_float2(rsqrtf(d2.x), rsqrtf(d2.y));
                    const float2 d = __fmul2_rn(d2, inv);
                    const float2 kk = __ffma2_rn(d, m1, hv);       // h - r
                    // 1/rho of the candidate, zero where it does not interact:
                    // the pressure, viscosity and colour terms vanish with it
                    const float2 V = make_float2(okx ? qb.z : 0.f, oky ? qb.w : 0.f);
                    const float4 qc = sc[s], qd = sd[s];
                    const float2 wk = __fmul2_rn(V, kk);
                    const float2 psum = __fadd2_rn(pi2, make_float2(qd.z, qd.w));
                    // V (h - r)^2 / r, which with kArt both sums share; the
                    // factor 2 alpha c0 h V_i waits for the end as well (350,000
                    // mixed particles, four stages: 1,893 -> 1,795 us)
                    const float2 sq = kArt ? __fmul2_rn(__fmul2_rn(wk, kk), inv) : zero;
                    const float2 ps =
                        kArt ? __fmul2_rn(sq, psum)
                             : __fmul2_rn(__fmul2_rn(__fmul2_rn(wk, psum), kk), inv);
                    Px = __ffma2_rn(dx, ps, Px);
                    Py = __ffma2_rn(dy, ps, Py);
                    Pz = __ffma2_rn(dz, ps, Pz);
                    const float2 dvx = __fadd2_rn(make_float2(qc.x, qc.y), nvx);
                    const float2 dvy = __fadd2_rn(make_float2(qc.z, qc.w), nvy);
                    const float2 dvz = __fadd2_rn(make_float2(qd.x, qd.y), nvz);
                    if (kArt) {
                        // v_ij . r_ij = (v_j - v_i) . (x_j - x_i); the sum is
                        // kept against d = x_j - x_i and negated at the end
                        float2 vr = __fmul2_rn(dvx, dx);
                        vr = __ffma2_rn(dvy, dy, vr);
                        vr = __ffma2_rn(dvz, dz, vr);
                        // artificial_pair, packed; V is zero where the pair
                        // does not interact
                        const float2 vn = make_float2(fminf(vr.x, 0.f), fminf(vr.y, 0.f));
                        const float2 den =
                            __fmul2_rn(__fadd2_rn(d2, epsv),
                                       __fadd2_rn(make_float2(qb.z, qb.w), viv));
                        const float2 rcp =
                            make_float2(__fdividef(1.f, den.x), __fdividef(1.f, den.y));
                        const float2 w = __fmul2_rn(__fmul2_rn(sq, vn), rcp);
                        Vx = __ffma2_rn(dx, w, Vx);
                        Vy = __ffma2_rn(dy, w, Vy);
                        Vz = __ffma2_rn(dz, w, Vz);
                    } else {
                        Vx = __ffma2_rn(dvx, wk, Vx);
                        Vy = __ffma2_rn(dvy, wk, Vy);
                        Vz = __ffma2_rn(dvz, wk, Vz);
                    }
                    const float2 wh = __fmul2_rn(V, t);
                    const float2 gw = __fmul2_rn(wh, t);
                    Gx = __ffma2_rn(dx, gw, Gx);
                    Gy = __ffma2_rn(dy, gw, Gy);
                    Gz = __ffma2_rn(dz, gw, Gz);
                    L = __ffma2_rn(wh, __ffma2_rn(t, m075, d2), L);
                }
            });
        float s[10] = {Px.x + Px.y, Py.x + Py.y, Pz.x + Pz.y,
                       Vx.x + Vx.y, Vy.x + Vy.y, Vz.x + Vz.y,
                       Gx.x + Gx.y, Gy.x + Gy.y, Gz.x + Gz.y, L.x + L.y};
#pragma unroll
        for (int k = 0; k < 10; ++k)
#pragma unroll
            for (int o = C; o < 32; o <<= 1) s[k] += __shfl_xor_sync(kFull, s[k], o);
        if (g == 0 && first + i < cend) {
            ForceAcc a;
            a.px = s[0];
            a.py = s[1];
            a.pz = s[2];
            // artificial viscosity: the sums times 2 alpha c0 h V_i
            const float art = kArt ? 2.f * P.art_coef * P.h * p.w : 1.f;
            a.vx = art * s[3];
            a.vy = art * s[4];
            a.vz = art * s[5];
            a.gx = -s[6];
            a.gy = -s[7];
            a.gz = -s[8];
            a.lap = s[9];
            write_force(f, P, self, f.pos[self], pev, G, a, true);
        }
    }
}

// -------------------------------------------------------------- integrate --
__global__ void __launch_bounds__(256)
k_integrate(Frame f, DevParams P) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= f.n) return;
    const float4 tp = f.pos[i];
    const float4 ev = f.ev[i];
    const SceneGeom G = geom_of_particle(f.scenes, i);
    const float4 v4 = f.vel[i];
    const float4 a4 = f.acc[i];
    float4 po, vo, eo;
    integrate_one(tp, v4, ev, a4.x, a4.y, a4.z, P, G, po, vo, eo);
    f.pos[i] = po;
    f.vel[i] = vo;
    f.ev[i] = eo;
}

// ---------------------------------------------------------------- render --
// COLORA (kernel_common.cuh:58): a * 255 << 24 | b << 16 | g << 8 | r, each
// channel clamped to [0, 255] (the device conversion of the reference
// saturates the same way).
__device__ __forceinline__ uint32_t colora(float r, float g, float b, float a) {
    auto ch = [](float v) { return uint32_t(fminf(fmaxf(v * 255.0f, 0.f), 255.f)); };
    return (ch(a) << 24) | (ch(b) << 16) | (ch(g) << 8) | ch(r);
}

__device__ __forceinline__ float density_color(const Frame &f, int i) {
    return (5000.f - 1.0f / f.pos[i].w) / 6000.f;
}

__global__ void __launch_bounds__(256)
k_render_tra(Frame f, uint32_t *color) {
    const int middle = f.ctr->middle;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < middle;
         k += gridDim.x * blockDim.x) {
        const int i = f.ctr->any_sms ? f.compact[k] : k;
        const float c = density_color(f, i);
        color[i] = colora(c, 0.f, c, 1.f);
    }
}

__global__ void __launch_bounds__(256)
k_render_sms(Frame f, uint32_t *color) {
    const int tasks = f.ctr->task_count;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < tasks * kSmsTaskParticles;
         k += gridDim.x * blockDim.x) {
        const gsph_block_task t = f.tasks[k / kSmsTaskParticles];
        const int i = t.cell_begin + task_offset(t) + k % kSmsTaskParticles;
        if (i >= t.cell_begin + t.cell_particle_count) continue;
        const float c = density_color(f, i);
        color[i] = t.is_same ? colora(0.f, c, c, 1.f) : colora(c, c, 0.f, 1.f);
    }
}

__global__ void __launch_bounds__(256)
k_final_position(Frame f, float3 ratio, float3 origin, float4 *out) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < f.n;
         i += gridDim.x * blockDim.x) {
        const float4 p = f.pos[i];
        out[i] = make_float4(p.x * ratio.x + origin.x, p.y * ratio.y + origin.y,
                             p.z * ratio.z + origin.z, 1.f);
    }
}

// ------------------------------------------------------- FP64 reductions --
// Deterministic two-level tree: fixed per-block partials, then one block.
constexpr int kRedThreads = 256;
constexpr int kRedBlocks = 512;

template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K], double *out) {
    __shared__ double sh[K][kRedThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double x = v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(kFull, x, o);
        if (lane == 0) sh[k][warp] = x;
    }
    __syncthreads();
    if (threadIdx.x < K) {
        double t = 0.0;
        for (int w = 0; w < kRedThreads / 32; ++w) t += sh[threadIdx.x][w];
        out[threadIdx.x] = t;
    }
}

__global__ void __launch_bounds__(kRedThreads)
k_checksum_partial(const float4 *__restrict__ pos, int n,
                   double *__restrict__ part) {
    double v[5] = {0, 0, 0, 0, 0};
    for (int i = blockIdx.x * kRedThreads + threadIdx.x; i < n;
         i += gridDim.x * kRedThreads) {
        const float4 p = pos[i];
        v[0] += p.x;
        v[1] += p.y;
        v[2] += p.z;
        v[3] += p.w;
        v[4] += double((unsigned(i) & 1023u) + 1u) *
                (double(p.x) + 3.0 * double(p.y) + 7.0 * double(p.z));
    }
    block_sum<5>(v, part + 5 * blockIdx.x);
}

__global__ void __launch_bounds__(kRedThreads)
k_reduce_partial(const float4 *__restrict__ pos, const float4 *__restrict__ vel,
                 int n, double mass, double *__restrict__ part) {
    double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int i = blockIdx.x * kRedThreads + threadIdx.x; i < n;
         i += gridDim.x * kRedThreads) {
        const float4 p = pos[i];
        const float4 u = vel[i];
        v[0] += mass;
        v[1] += mass * u.x;
        v[2] += mass * u.y;
        v[3] += mass * u.z;
        v[4] += 0.5 * mass * (double(u.x) * u.x + double(u.y) * u.y +
                              double(u.z) * u.z);
        v[5] += p.x;
        v[6] += p.y;
        v[7] += p.z;
    }
    block_sum<8>(v, part + 8 * blockIdx.x);
}

template <int K>
__global__ void __launch_bounds__(kRedThreads)
k_final_sum(const double *__restrict__ part, int nparts, double *__restrict__ out) {
    double v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = 0.0;
    for (int b = threadIdx.x; b < nparts; b += kRedThreads)
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] += part[K * b + k];
    block_sum<K>(v, out);
}

// Shared-memory carveout of one kernel: what `ctas` resident CTAs of it need
// (static shared memory plus the 1 KB the SM reserves per CTA), so that the
// rest of the SM's unified L1/shared storage stays L1 for candidate reads.
template <class Kernel>
cudaError_t set_carveout(Kernel kernel, int ctas, int smem_per_sm, int threads) {
    cudaFuncAttributes a{};
    cudaError_t e = cudaFuncGetAttributes(&a, kernel);
    if (e != cudaSuccess) return e;
    int pct = 0;
    if (a.sharedSizeBytes > 0 && smem_per_sm > 0) {
        const long long need = (long long)(a.sharedSizeBytes + 1024) * ctas;
        pct = int(std::min<long long>(100, (need * 100 + smem_per_sm - 1) / smem_per_sm));
    }
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
    if (e != cudaSuccess) return e;
    // the hint is rounded to a supported split; keep the default if the
    // rounded one would hold fewer CTAs
    int fit = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kernel, threads, 0);
    if (e != cudaSuccess) return e;
    if (fit < ctas)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 int(cudaSharedmemCarveoutDefault));
    return e;
}

template <int W>
cudaError_t configure_shape(int smem) {
    const int k = kWarpsPerBlock / W;   // CTAs per SM scale with the block size
    cudaError_t e;
    for (auto kernel : {k_density_tra<W, false, false>, k_density_tra<W, false, true>,
                        k_density_tra<W, true, false>, k_density_tra<W, true, true>})
        if ((e = set_carveout(kernel, kMaxShape.density_tra * k, smem, W * 32))) return e;
    if ((e = set_carveout(k_density_sms<W>, kMaxShape.density_sms * k, smem, W * 32)))
        return e;
    for (auto kernel : {k_force_tra<false, W>, k_force_tra<true, W>,
                        k_force_tra<false, W, false, true>, k_force_tra<true, W, false, true>})
        if ((e = set_carveout(kernel, kMaxShape.force_tra * k, smem, W * 32))) return e;
    if ((e = set_carveout(k_force_sms<false, W>, kForceSmsCtas * k, smem, W * 32)))
        return e;
    return set_carveout(k_force_sms<true, W>, kForceSmsCtas * k, smem, W * 32);
}

// Blocks of an SMS pass: `ctas` per SM, but one or two where the scene's
// clusters cannot fill more. (All-TRA frames, whose SMS blocks only look and
// leave, feel the difference: 13,824 particles 33.7 us a frame with four per
// SM, 32.6 with one. Three, which fill the SMs' shared memory to the last
// block, hold the TRA blocks back: 39.9.)
int sms_blocks(const Frame &f, int num_sms, int ctas, int warps) {
    const int clusters = f.n / kDenCluster + 1;
    const int need = (clusters + num_sms * warps - 1) / (num_sms * warps);
    return num_sms * (need <= 2 ? std::min(need, ctas) : ctas);
}

// Which build the TRA passes of a scene of f.n particles run (kRowsMax1 and the
// following lines). All but the general ones have a fixed shape.
enum class DensityTra { kRow1, kRow3, kGeneral };
DensityTra density_build(const Frame &f, int num_sms) {
    const int units = (f.n + 31) / 32;
    if (units <= num_sms * kRowsMax1 ||
        (units > num_sms * kRowsAgain1 && units <= num_sms * kRowsAgainMax1))
        return DensityTra::kRow1;
    return units <= num_sms * kRowsMax3 ? DensityTra::kRow3 : DensityTra::kGeneral;
}
enum class ForceTra { kQuad, kSmall, kGeneral };
ForceTra force_build(const Frame &f, int num_sms) {
    const int units = (f.n + 31) / 32;
    if (units <= num_sms * kForceQuadMax) return ForceTra::kQuad;
    return units <= num_sms * kForceSmallMax ||
                   (units > num_sms * kForceSmallAgain && units <= num_sms * kForceSmallAgainMax)
               ? ForceTra::kSmall
               : ForceTra::kGeneral;
}

template <int W>
void launch_density_w(const Frame &f, const DevParams &P, int num_sms,
                      const LaunchShape &shape, cudaStream_t s, cudaStream_t s_sms,
                      bool row_prefetch) {
    k_density_sms<W><<<sms_blocks(f, num_sms, shape.density_sms, W), W * 32, 0, s_sms>>>(f, P);
    const int units = (f.n + 31) / 32;
    const DensityTra build = density_build(f, num_sms);
    if (build == DensityTra::kRow1)
        launch_after(k_density_tra_rows<1>, units, 288, s, f, P);
    else if (build == DensityTra::kRow3)
        launch_after(k_density_tra_rows<3>, (units + 2) / 3, 288, s, f, P);
    else {
        const bool many = f.scenes.count > 1;
        auto kernel = row_prefetch ? (many ? k_density_tra<W, true, true>
                                           : k_density_tra<W, true, false>)
                                   : (many ? k_density_tra<W, false, true>
                                           : k_density_tra<W, false, false>);
        if (tra_fills(f, num_sms))
            kernel<<<num_sms * shape.density_tra, W * 32, 0, s>>>(f, P);
        else
            launch_after(kernel, num_sms * shape.density_tra, W * 32, s, f, P);
    }
}

template <bool kArt, int W>
void launch_force_sms_w(const Frame &f, const DevParams &P, int num_sms,
                        const LaunchShape &shape, cudaStream_t s) {
    k_force_sms<kArt, W><<<sms_blocks(f, num_sms, shape.force_sms, W), W * 32, 0, s>>>(
        f, P, num_sms * kForceSmsCtas * kWarpsPerBlock / W);
}

// part: null for all units.
template <bool kArt, int W>
void launch_force_tra_w(const Frame &f, const DevParams &P, int num_sms, bool fresh,
                        const LaunchShape &shape, const ForcePart *part, cudaStream_t s) {
    const int units = (f.n + 31) / 32;
    const ForceTra build = force_build(f, num_sms);
    if (part)
        k_force_tra<kArt, W, false, true>
            <<<num_sms * shape.force_tra, W * 32, 0, s>>>(f, P, fresh, *part);
    else if (build == ForceTra::kQuad)
        k_force_tra_quad<kArt><<<units, 128, 0, s>>>(f, P, fresh);
    else if (build == ForceTra::kSmall)
        k_force_tra<kArt, 2, true><<<(units + 1) / 2, 64, 0, s>>>(f, P, fresh, ForcePart{});
    else
        k_force_tra<kArt, W>
            <<<num_sms * shape.force_tra, W * 32, 0, s>>>(f, P, fresh, ForcePart{});
}

// Calls run(viscosity model, block shape) with both as compile-time constants.
template <class Run>
void with_build(const DevParams &P, const LaunchShape &shape, Run run) {
    using Full = std::integral_constant<int, kWarpsPerBlock>;
    using Half = std::integral_constant<int, kWarpsPerBlock / 2>;
    const bool half = shape.warps == kWarpsPerBlock / 2;
    if (P.visc_artificial)
        half ? run(std::true_type{}, Half{}) : run(std::true_type{}, Full{});
    else
        half ? run(std::false_type{}, Half{}) : run(std::false_type{}, Full{});
}

}  // namespace

cudaError_t configure_physics_kernels(int device) {
    int smem = 0;
    cudaError_t e = cudaDeviceGetAttribute(
        &smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
    if (e != cudaSuccess) return e;
    if ((e = configure_shape<kWarpsPerBlock>(smem))) return e;
    return configure_shape<kWarpsPerBlock / 2>(smem);
}

void launch_density(const Frame &f, const DevParams &P, int num_sms,
                    const LaunchShape &shape, cudaStream_t s, cudaStream_t s_sms) {
    if (f.n <= 0) return;
    // cell offsets and slab words: 8 bytes per cell
    const bool row_prefetch = size_t(P.numc) * 8 > kRowPrefetchCellBytes;
    if (shape.warps == kWarpsPerBlock / 2)
        launch_density_w<kWarpsPerBlock / 2>(f, P, num_sms, shape, s, s_sms, row_prefetch);
    else
        launch_density_w<kWarpsPerBlock>(f, P, num_sms, shape, s, s_sms, row_prefetch);
}

LaunchShape launched_shape(const Frame &f, int num_sms, LaunchShape shape) {
    if (density_build(f, num_sms) != DensityTra::kGeneral) shape.density_tra = 0;
    if (force_build(f, num_sms) != ForceTra::kGeneral) shape.force_tra = 0;
    shape.density_sms = sms_blocks(f, num_sms, shape.density_sms, shape.warps);
    shape.force_sms = sms_blocks(f, num_sms, shape.force_sms, shape.warps);
    return shape;
}

bool tra_fills(const Frame &f, int num_sms) {
    return (f.n + 31) / 32 > num_sms * kTraFills;
}
bool force_in_parts(const Frame &f, int num_sms) {
    return (f.n + 31) / 32 > num_sms * kForcePartsMin;
}

void launch_force_sms(const Frame &f, const DevParams &P, int num_sms,
                      const LaunchShape &shape, cudaStream_t s) {
    if (f.n <= 0) return;
    with_build(P, shape, [&](auto art, auto warps) {
        launch_force_sms_w<art.value, warps.value>(f, P, num_sms, shape, s);
    });
}

void launch_force_tra_part(const Frame &f, const DevParams &P, int num_sms, bool fresh,
                           const LaunchShape &shape, const ForcePart &part, cudaStream_t s) {
    if (f.n <= 0) return;
    with_build(P, shape, [&](auto art, auto warps) {
        launch_force_tra_w<art.value, warps.value>(f, P, num_sms, fresh, shape, &part, s);
    });
}

void launch_force(const Frame &f, const DevParams &P, int num_sms, bool fresh,
                  const LaunchShape &shape, cudaStream_t s, cudaStream_t s_sms) {
    if (f.n <= 0) return;
    launch_force_sms(f, P, num_sms, shape, s_sms);
    with_build(P, shape, [&](auto art, auto warps) {
        launch_force_tra_w<art.value, warps.value>(f, P, num_sms, fresh, shape, nullptr, s);
    });
}

void launch_integrate(const Frame &f, const DevParams &P, cudaStream_t s) {
    if (f.n <= 0) return;
    k_integrate<<<(f.n + 255) / 256, 256, 0, s>>>(f, P);
}

// out5 must hold 5 + 5*kRedBlocks doubles (partials follow the result).
void launch_checksum(const float4 *pos, int n, double *out5, cudaStream_t s) {
    k_checksum_partial<<<kRedBlocks, kRedThreads, 0, s>>>(pos, n, out5 + 8);
    k_final_sum<5><<<1, kRedThreads, 0, s>>>(out5 + 8, kRedBlocks, out5);
}

// out8 must hold 8 + 8*kRedBlocks doubles.
void launch_render(const Frame &f, float3 ratio, float3 origin, uint32_t *color,
                   float4 *final_pos, cudaStream_t s) {
    if (f.n <= 0) return;
    const int blocks = std::min((f.n + 255) / 256, 4096);
    if (color) {
        k_render_tra<<<blocks, 256, 0, s>>>(f, color);
        k_render_sms<<<blocks, 256, 0, s>>>(f, color);
    }
    if (final_pos) k_final_position<<<blocks, 256, 0, s>>>(f, ratio, origin, final_pos);
}

void launch_reductions(const float4 *pos, const float4 *vel, int n, float mass,
                       double *out8, cudaStream_t s) {
    k_reduce_partial<<<kRedBlocks, kRedThreads, 0, s>>>(pos, vel, n, mass,
                                                        out8 + 8);
    k_final_sum<8><<<1, kRedThreads, 0, s>>>(out8 + 8, kRedBlocks, out8);
}

}  // namespace gsph
