// Device data layout and kernel interfaces of the soft-force library.
//
// HBM layout (one copy per process, grown on demand, never shrunk):
//   EpjMix[n_epj_tot]    32 B: FP64 position, FP32 mass, FP32 r_search^2
//   epj_m64[n_epj_tot]    8 B: FP64 mass       (plain FP64 kernel)
//   epj_rs64[n_epj_tot]   8 B: FP64 r_search   (plain FP64 kernel, exact re-tests)
//   SpjMix[n_spj_tot]    64 B: FP64 position, FP32 mass, FP32 traceless
//                              quadrupole Q = 3q - tr(q) I and tr(q)
//   SpjQ64[n_spj_tot]    64 B: FP64 mass and raw quadrupole (plain FP64 kernel)
//   EpjF32[n_epj_tot]    32 B: position as an FP32 (hi, lo) pair, FP32 mass
//                              and r_search^2 (warp-specialised kernels)
//   SpjF32[n_spj_tot]    64 B: position as an FP32 (hi, lo) pair, FP32 mass,
//                              traceless quadrupole and tr(q)
//   EpiDev[ni_tot]       32 B: FP64 position and r_search
//   id_epj / id_spj      int32 per list entry, walks concatenated
//   WalkDesc[n_walk]    160 B: list offsets, walk centre (FP64 and FP32), box
//                              half-extents, largest i r_search, r_out^2
//   order[n_walk]        walks sorted by descending work (the work queue)
//   EpiRel[ni_tot]       32 B: FP32 (hi, lo) position about the walk centre,
//                              r_search^2, guard band (warp-specialised kernels)
//   out_accp[ni_tot]     Accp (32 B): acc.xyz, pot (G applied)
//   out_nnb[ni_tot]      int32 neighbour count
// The j arrays of a 1.5M-particle problem (about 50 MB EPJ + 18 MB SPJ for the
// mixed kernel) stay resident in the 129 MB L2 while the id lists stream from
// HBM once per force evaluation.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace pgf {

struct __align__(32) EpjMix {
    double x, y, z;
    float m;
    float rs2;  // (float)(r_search * r_search), the square taken in FP64
};
static_assert(sizeof(EpjMix) == 32, "EpjMix layout");

struct __align__(32) SpjMix {
    double x, y, z;
    float m;
    float pad0;
    float Q[6];  // traceless 3q - tr(q) I: xx, yy, zz, xy, xz, yz
    float tr;    // tr(q)
    float pad1;
};
static_assert(sizeof(SpjMix) == 64, "SpjMix layout");

// Positions split into FP32 hi = fl(x) and lo = fl(x - hi), so hi + lo holds x
// to about 2^-48 |x|.  Built on the device from EpjMix / SpjMix; they let the
// warp-specialised kernels form walk-relative coordinates in FP32 arithmetic
// (the FP64 pipe of GB300 runs at 1/64 of the FP32 rate).
struct __align__(32) EpjF32 {
    float xh, yh, zh, m;
    float xl, yl, zl, rs2;
};
static_assert(sizeof(EpjF32) == 32, "EpjF32 layout");

struct __align__(32) SpjF32 {
    float xh, yh, zh, m;
    float xl, yl, zl, tr;
    float Q[6];  // traceless 3q - tr(q) I
    float pad[2];
};
static_assert(sizeof(SpjF32) == 64, "SpjF32 layout");

// Acceleration of one particle as an FP32 (hi, lo) pair (KDKDK_4TH gradient mode):
// differences a_j - a_i are formed from both halves, accurate to an ulp of
// the difference itself.
struct __align__(32) AccF32 {
    float xh, yh, zh, pad0;
    float xl, yl, zl, pad1;
};
static_assert(sizeof(AccF32) == 32, "AccF32 layout");

// Changeover data of one particle for the fused changeover mode: the
// ChangeOver members of src/changeover.hpp:8-14 (r_in, r_out, norm =
// 1/(r_out - r_in), coff = (r_out - r_in)/(r_out + r_in), pot_off =
// (1 + coff)/r_out), computed in FP64 and rounded; the particle id; and a mass:
// for EPJ the mass its neighbours' potentials use (m for singles, mass_backup
// for members, 0 otherwise), for EPI the mass of its self-potential term.
struct __align__(32) CoRec {
    float r_in, r_out, norm, coff;
    float pot_off, mass;
    int64_t id;
};
static_assert(sizeof(CoRec) == 32, "CoRec layout");

struct __align__(16) SpjQ64 {
    double m;
    double q[6];  // raw second moment: xx, yy, zz, xy, xz, yz (zero for monopoles)
    double pad;
};
static_assert(sizeof(SpjQ64) == 64, "SpjQ64 layout");

struct __align__(32) EpiDev {
    double x, y, z, rs;
};
static_assert(sizeof(EpiDev) == 32, "EpiDev layout");

// An i-particle as the warp-specialised kernels read it: x - c of its walk as
// an FP32 (hi, lo) pair, r_search^2 and the guard band of its neighbour test
// in ulps.  Formed in FP64 once per dispatch (a split walk's parts and every
// pass share it): GB300's FP64 pipe holds a warp instruction for 64 cycles.
struct __align__(32) EpiRel {
    float hx, hy, hz, rs2;
    float lx, ly, lz;
    int32_t kb;
};
static_assert(sizeof(EpiRel) == 32, "EpiRel layout");

constexpr int kKMax = 1 << 22;

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Guard band in ulps of rs2 for the near-pair neighbour test of one i at
// distance D (max norm) from the walk centre; see kband_near64 in
// pgf_kernels_mixed.cu for the derivation: the FP32 test is off by less than
// 8 + 1.3e-6 D / r_ref ulps, r_ref = sqrt(rs^2 - eps2), and the band is
// 48 + 1e-5 D / r_ref.  Evaluated here in FP32; the few ulps of rounding of
// the FP32 form are far inside the factor of six between the band and the
// bound, and a larger band only adds exact re-tests.
__device__ __forceinline__ int kband_near(float D, float rs2, float eps2) {
    const float r2ref = rs2 - eps2;
    if (!(r2ref > 0.f)) return kKMax;
    const float k = 48.f + 1e-5f * D * rsqrt_approx(r2ref) * 1.001f;
    return k >= float(kKMax) ? kKMax : int(k) + 1;
}

// (float)x and the rest x - (float)x as a float, on the integer pipe where both
// are normal numbers: the same roundings (to nearest, ties to even) as the FP64
// pipe's conversions and subtraction, at a dozen instructions instead of 64
// cycles of that pipe each.
__device__ __forceinline__ float2 split_rn(double x) {
    const unsigned lo = (unsigned)__double2loint(x), hi = (unsigned)__double2hiint(x);
    const unsigned e = (hi >> 20) & 0x7ffu, sign = hi & 0x80000000u;
    if (e - 949u >= 1150u - 949u) {  // 0, too small for either part, too large, infinite, NaN
        if (!((hi << 1) | lo)) return make_float2(__uint_as_float(sign), 0.f);
        const float h = (float)x;
        return make_float2(h, (float)(x - (double)h));
    }
    const unsigned m = ((hi & 0xfffffu) << 3) | (lo >> 29), r = lo & 0x1fffffffu;
    const unsigned up = r + (m & 1u) > 0x10000000u;
    const float h = __uint_as_float((sign | ((e - 896u) << 23) | m) + up);
    const float scale = __uint_as_float(sign | ((e - 948u) << 23));
    return make_float2(h, scale * (float)(int)(r - (up << 29)));
}
__device__ __forceinline__ float f32_rn(double x) { return split_rn(x).x; }

__device__ __forceinline__ AccF32 make_acc32(double x, double y, double z) {
    const float2 u = split_rn(x), v = split_rn(y), w = split_rn(z);
    return AccF32{u.x, v.x, w.x, 0.f, u.y, v.y, w.y, 0.f};
}

__device__ __forceinline__ EpiRel make_epi_rel(const EpiDev& e, double cx, double cy, double cz, float eps2) {
    const float2 dx = split_rn(__dsub_rn(e.x, cx)), dy = split_rn(__dsub_rn(e.y, cy)), dz = split_rn(__dsub_rn(e.z, cz));
    EpiRel r;
    r.hx = dx.x;
    r.hy = dy.x;
    r.hz = dz.x;
    r.rs2 = f32_rn(__dmul_rn(e.rs, e.rs));
    r.lx = dx.y;
    r.ly = dy.y;
    r.lz = dz.y;
    r.kb = kband_near(fmaxf(fabsf(r.hx), fmaxf(fabsf(r.hy), fabsf(r.hz))), r.rs2, eps2);
    return r;
}

// Error-free sum: s + e == a + b exactly (round-to-nearest, no reassociation).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// Sum of two (hi, lo) pairs.
__device__ __forceinline__ float2 add_pair(float2 a, float2 b) {
    float s, e;
    two_sum(a.x, b.x, s, e);
    return make_float2(s, e + (a.y + b.y));
}

struct __align__(32) WalkDesc {
    int64_t epj_begin;  // offset of the walk's EPJ ids in id_epj
    int64_t spj_begin;  // offset of the walk's SPJ ids in id_spj
    int32_t i_begin;    // first EPI row of the walk
    int32_t n_i;
    int32_t n_epj;
    int32_t n_spj;
    double cx, cy, cz;  // walk centre: centre of the EPI bounding box
    double rcut2;       // r_out^2 of the walk
    float hx, hy, hz;   // EPI box half-extents, rounded up
    float rs_max;       // largest r_search of the walk's EPI, rounded up
    uint16_t part;      // 0, or k >= 1 for part k of a split walk (adds no per-i terms)
    uint16_t n_parts;   // 1, or the parts of a split walk
    int32_t root;       // descriptor of part 0 (this one when not split)
    int32_t n_spj_all;  // SPJ of the whole walk
    int32_t i_root;     // first EPI row of the walk; i_begin is the first result row
    // FP32 forms of the above for the kernels' passes (set_walk_f32).
    float ch[3], cl[3];      // walk centre, hi and lo
    float rcut2f;
    float gr_kh, gr_kl;      // 3 / r_out^2, hi and lo (gradient mode)
    float gr_r3;             // r_out^-3 (gradient mode)
    float pad[6];
};
static_assert(sizeof(WalkDesc) == 160, "WalkDesc layout");

__host__ __device__ inline void set_walk_f32(WalkDesc& d, bool gradient) {
    const double c[3] = {d.cx, d.cy, d.cz};
    for (int k = 0; k < 3; ++k) {
        d.ch[k] = (float)c[k];
        d.cl[k] = (float)(c[k] - (double)d.ch[k]);
    }
    d.rcut2f = (float)d.rcut2;
    d.gr_kh = d.gr_kl = d.gr_r3 = 0.f;
    if (gradient) {
        const double kd = 3.0 / d.rcut2;
        d.gr_kh = (float)kd;
        d.gr_kl = (float)(kd - (double)d.gr_kh);
        d.gr_r3 = (float)(1.0 / (d.rcut2 * sqrt(d.rcut2)));
    }
    for (int k = 0; k < 6; ++k) d.pad[k] = 0.f;
}

// Result of one i-particle: acceleration and potential with G applied.
struct __align__(32) Accp {
    double x, y, z, w;
};
static_assert(sizeof(Accp) == 32, "Accp layout");

// An (i, EPJ tile) whose FP32 neighbour test came within rounding distance of
// r_search for some pair: the retest kernel recounts the tile in FP64.
struct Retest {
    int64_t j_begin;  // offset in id_epj
    int32_t i;        // EPI row
    int32_t n;        // number of list entries
    int32_t row;      // result row
    int32_t pad;
};

// Superparticles of one walk left to the pair kernels by the far-field pass:
// the entries in each quarter of the walk's list (n[0] < 0: the list as it
// is), and whether out_accp of the walk's rows holds the sums of the others
// (load_pairs) for the pair kernels to
// add.
struct __align__(32) SpjNear {
    int32_t n[4];
    int32_t add_far;
    int32_t pad[3];
};

struct Params {
    const EpiDev* epi;
    const EpiRel* epi_rel;  // of the same rows (launch_epi_rel or the walk gather)
    const EpjMix* epj;
    const double* epj_m64;
    const double* epj_rs64;
    const SpjMix* spj;
    const SpjQ64* spj_q64;
    const EpjF32* epj32;
    const SpjF32* spj32;
    const CoRec* epj_co;   // fused changeover mode only (else null)
    const CoRec* epi_co;
    double* out_pot_soft;  // fused changeover mode: soft potential (G applied)
    const AccF32* epj_acc32;  // gradient mode: EPJ accelerations (hi, lo)
    const Accp* epi_acc64;    // gradient mode: EPI accelerations (x, y, z; w unused)
    const AccF32* epi_acc32;  // and as (hi, lo) pairs
    Accp* out_acorr;          // gradient mode: acorr (no G; w unused)
    const int32_t* id_epj;
    const int32_t* id_spj;
    const WalkDesc* walks;
    const int32_t* order;
    int32_t n_walk;
    int32_t pad0;
    double eps2;
    double G;
    Accp* out_accp;
    int32_t* out_nnb;
    // Bases of the result rows of parts >= 1 of split walks (null: out_accp,
    // out_nnb).
    Accp* part_accp;
    int32_t* part_nnb;
    // Part 0 writes rows of its own there too: the walks' rows may overlap
    // (only the combine kernel writes those of a split walk, whole results).
    int32_t part0_rows;
    int32_t pad1;
    // scratch
    // Launch counters, kLaunchCounters ints that lie together and are zeroed
    // before each launch (reset_counters): the work-queue cursor, the number
    // of re-test records pushed (n_retest, may exceed the capacity) and the
    // far-field pass's cursor.
    int32_t* queue_head;
    int32_t* n_retest;     // queue_head + 1
    int32_t* far_queue;    // queue_head + 2
    Retest* retest;        // FP64 re-test records
    int32_t retest_cap;
    int32_t pad2;
    int32_t* err;          // device error word (0 = ok)
    int32_t* retest_total; // records re-tested since the host last read it (optional)
    // Walk count written by an earlier kernel on the same stream (the device
    // list builder), or null: the kernels then run min(*n_walk_dev, n_walk)
    // walks, n_walk being the capacity of walks and order.
    const int32_t* n_walk_dev;
    // Limit of every bounded wait in the warp-specialised kernels (0: 1 s).
    uint64_t wait_limit_ns;
    // Test hook: > 0 makes their producer stop after that many ring items.
    int32_t stall_after_items;
    int32_t gr_compensated;  // gradient pass: r^2 and 1/r of far pairs to about 2^-40 (pgf_set_gradient_accuracy)
    // Far-field pass (pgf_kernels_far.cu), or null: the ids of the
    // superparticles left to the pair kernels (same offsets as id_spj), and
    // per walk (by root descriptor) what they hold.
    int32_t* id_spj_near;
    SpjNear* spj_near;
    // Parts of split walks start at multiples of this many entries of the
    // compacted list (0: 1).
    int32_t part_align;
    // Partial sums are flushed at every tile's end, so that whole walks and
    // walks in parts of whole tiles add the same FP32 terms.
    int32_t flush_tiles;
    // Walks without their further parts: when some are split (n_root <
    // n_walk) the roots are descriptors 0 .. n_root - 1 by descending cost.
    int32_t n_root;
    int32_t far_wide;  // far-field pass with eight warps per walk (kFarWideRows)
    // Result of the device-side check of a host-direct dispatch's ids, or
    // null: when it is non-zero the force kernels run nothing.
    const int32_t* input_err;
    // The CTA-synchronous kernel runs only when this word is non-zero (null:
    // always).  A null order is the walks as they lie.
    const int32_t* run_if;
};

// Limit of the bounded waits and the stall test hook, as set through the C ABI.
struct WaitHooks {
    uint64_t wait_limit_ns;  // 0: 1 s
    int stall_after_items;   // 0: none
};
WaitHooks wait_hooks();

// Number of walks of this launch.
__device__ __forceinline__ int walk_count(const Params& p) {
    return p.n_walk_dev ? min(*p.n_walk_dev, p.n_walk) : p.n_walk;
}

// Exact FP64 neighbour test of one pair, in the oracle's evaluation order
// (src/force_gpu_cuda.cu:62-64 semantics, src/soft_force.hpp:58-64 order):
// r2 = ((dx*dx) + (dy*dy)) + (dz*dz); (r2 + eps2) < max(rs_i, rs_j)^2.
__device__ __forceinline__ int exact_neighbour(double xi, double yi, double zi, double rsi, double xj,
                                               double yj, double zj, double rsj, double eps2) {
    const double dx = __dsub_rn(xi, xj);
    const double dy = __dsub_rn(yi, yj);
    const double dz = __dsub_rn(zi, zj);
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    const double rs = rsi > rsj ? rsi : rsj;
    return __dadd_rn(r2, eps2) < __dmul_rn(rs, rs) ? 1 : 0;
}

// FP64 difference between the changeover pair terms and the linear-cutoff
// pair terms of one neighbour pair (the fused mode's correction for pairs
// whose neighbour status only the FP64 re-test decides): acceleration x, y,
// z, pot_tot and pot_soft, without G.  Same formulas as the FP32 pair path.
__device__ __forceinline__ void co_pair_diff(const EpiDev& ei, const CoRec& ci, const EpjMix& ej, float mj, const CoRec& cj,
                                    double eps2, double rcut2, double out[5]) {
    const double dx = ej.x - ei.x, dy = ej.y - ei.y, dz = ej.z - ei.z;
    const double r2 = dx * dx + dy * dy + dz * dz + eps2;
    const double r = sqrt(r2), ri = 1.0 / r;
    const double rimax = 1.0 / sqrt(r2 > rcut2 ? r2 : rcut2);
    const CoRec& c = ci.r_out > cj.r_out ? ci : cj;
    const double x = (r - (double)c.r_in) * (double)c.norm;
    const double xa = x < 0.0 ? 0.0 : (x > 1.0 ? 1.0 : x);
    const double x_1 = xa - 1.0, x_2 = x_1 * x_1, xa2 = xa * xa;
    const double wacc = (x_2 * x_2) * (1.0 + 4.0 * xa + 10.0 * xa2 + 20.0 * xa2 * xa + 35.0 * (double)c.coff * xa2 * xa2);
    double wpot = 1.0;
    if (x >= 1.0) {
        wpot = (double)c.pot_off * r;
    } else if (x > 0.0) {
        const double x2 = x * x, x3 = x2 * x;
        wpot = 1.0 - (double)c.coff * (x2 * x3) * (5.0 * x3 - 20.0 * x2 + 28.0 * x - 14.0);
    }
    const double f = (double)mj * ((1.0 - wacc) * ri * ri * ri - rimax * rimax * rimax);
    out[0] = f * dx;
    out[1] = f * dy;
    out[2] = f * dz;
    const double meff = (double)cj.mass;
    out[3] = -meff * ri + (double)mj * rimax;
    out[4] = -meff * (1.0 - wpot) * ri + (double)mj * rimax;
}

// A walk whose list was split into n_parts parts (small dispatches, to spread
// the largest walks over several CTAs): every part reads the walk's EPI rows;
// part 0 writes the walk's own result rows from row0, part k >= 1 rows of its
// own from rows1 + (k - 1) n_i.
struct SplitRec {
    int32_t row0, rows1, n_i, n_parts;
};

// ---- Host-direct data movement (pgf_hostdirect.cu) ----
// The GPU reads the caller's records in host memory through the host page
// tables and writes results into them; these tables and arguments describe
// where.

// One walk of a host-direct dispatch, in layout order.
struct WalkSrc {
    const char* epi;        // the caller's EPI records of the walk
    const int32_t* id_epj;  // the caller's id lists of the walk
    const int32_t* id_spj;
    int64_t i_off, e_off, s_off;  // first EPI row and list entries in the device arrays
    int64_t rows1;          // split walks: first result row of part 1
    double rcut2;           // r_out^2 of the walk
    int32_t n_i, n_epj, n_spj;
    int32_t walk;           // the caller's walk index (error reports)
    int32_t parts;          // 1, or the parts of a split walk
    int32_t desc1;          // split walks: descriptor index of part 1
    int32_t split;          // split walks: index of its SplitRec
    int32_t pad;
};

// Where retrieve writes walk k's results.
struct ForceDst {
    char* base;   // the caller's Force records of the walk
    int64_t row;  // first result row of the walk
    int32_t n;
    int32_t pad;
};

struct HdSendArgs {
    const char* epj;
    int64_t n_epj;
    size_t epj_size, epj_off_mass, epj_off_pos, epj_off_rs;
    const char* spj;
    int64_t n_spj;
    size_t spj_size, spj_off_mass, spj_off_pos, spj_off_quad;
    int spj_has_quad;
    // fused changeover mode (out_epj_co non-null)
    size_t co_epj_off_id, co_epj_off_r_in, co_epj_off_r_out, co_epj_off_mass_backup, co_epj_off_status;
    // gradient mode (out_epj_acc32 non-null)
    size_t gr_epj_off_acc;
    EpjMix* out_epj;
    double* out_epj_m64;
    double* out_epj_rs64;
    EpjF32* out_epj32;
    CoRec* out_epj_co;
    AccF32* out_epj_acc32;
    SpjMix* out_spj;
    SpjQ64* out_spj_q64;
    SpjF32* out_spj32;
};

struct HdWalkArgs {
    const WalkSrc* src;         // pinned host table, read in place
    int n_walk;
    int n_desc;                 // work-queue entries (walks and parts)
    const int32_t* order_src;   // pinned host work-queue order, copied to order_dst
    int32_t* order_dst;
    SplitRec* out_splits;       // split walks' records (combine kernel)
    size_t epi_size, epi_off_pos, epi_off_rs;
    size_t gr_epi_off_acc;  // gradient mode (out_epi_acc non-null)
    size_t co_epi_off_id, co_epi_off_r_in, co_epi_off_r_out, co_epi_off_self_mass;  // changeover (out_epi_co)
    int64_t n_epj_tot, n_spj_tot;
    EpiDev* out_epi;
    EpiRel* out_epi_rel;
    float eps2;  // of the kernels' neighbour test (guard bands)
    AccF32* out_epi_acc32;
    Accp* out_epi_acc;
    CoRec* out_epi_co;
    int32_t* out_id_epj;
    int32_t* out_id_spj;
    WalkDesc* out_walks;
    // [0] set when an id is out of range, [1] the largest such caller walk
    // index, [2] finished CTAs, [3] the outcome the force kernels read.  The
    // last CTA moves [0], [1] into err_host[0], [1] (pinned) and [3], and
    // clears [0..2] for the next dispatch.
    int32_t* err;
    int32_t* err_host;
};

struct HdScatterArgs {
    const ForceDst* dst;
    int n_walk;
    int counts_only;  // neighbour search: n_ngb only
    size_t size, off_acc, off_pot, off_nnb;
    int nnb_bytes;
    int pad;
    size_t off_pot_soft, off_acorr;
    const Accp* accp;
    const int32_t* nnb;
    const double* pot_soft;  // changeover mode, else null
    const Accp* acorr;       // gradient mode, else null
    // Status words of the evaluation (the device error word and the re-test
    // total at [2], [3]): copied to flags_host and cleared by the kernel.
    int32_t* flags_dev;
    int32_t* flags_host;
};

cudaError_t launch_gather_j(const HdSendArgs& a, int num_sms, cudaStream_t s);
cudaError_t launch_gather_walks(const HdWalkArgs& a, int num_sms, cudaStream_t s);
cudaError_t launch_scatter_results(const HdScatterArgs& a, int num_sms, cudaStream_t s);

constexpr int kLaunchCounters = 3;
inline void bind_counters(Params& p, int32_t* c) {
    p.queue_head = c;
    p.n_retest = c + 1;
    p.far_queue = c + 2;
}
inline cudaError_t reset_counters(const Params& p, cudaStream_t s) {
    return cudaMemsetAsync(p.queue_head, 0, kLaunchCounters * sizeof(int32_t), s);
}

// The far-field pass pays where enough superparticles are distant: where lists
// are long (few walks of a large cluster do), or fairly long in launches that
// fill the GPU.  With the pass and without it: Plummer models at theta = 0.3 of
// 33,333 stars (2,200 EP-SP pairs per i) 0.54 and 0.51 ms a call, 65,536 (3,500)
// 0.99 and 0.97, 98,304 (4,300) 1.40 and 1.43, 196,608 (5,700) 2.75 and 2.91;
// 200-walk calls on 65,536 stars (3,500) 1.47 and 1.39 ms in all, on 393,216
// (6,900) 8.47 and 8.82; 230,253 stars in five clusters (2,900) 2.58 and 2.42,
// 112,126 in three (3,800) 1.48 and 1.52; King models at theta = 0.4: 131,072
// (2,850) 1.205 and 1.218, 180,000 (3,000) 1.60 and 1.66.  It expands
// unsoftened gravity only.
constexpr int64_t kFarMinRows = 8192, kFarPairs = 4000;   // EP-SP pairs per i
constexpr int64_t kFarRows = 80000, kFarRowsPairs = 3000;
constexpr int64_t kFarWideRows = 40000;
inline bool far_applies(double eps2, int64_t n_i, double sp_pairs) {
    return eps2 == 0.0 && n_i >= kFarMinRows &&
           sp_pairs >= (double)n_i * (double)(n_i >= kFarRows ? kFarRowsPairs : kFarPairs);
}
// The device-resident step, which knows its lists only on the device: King
// models, 65,536 particles 0.97 ms with the pass and 0.95 without, 131,072 1.50
// and 1.52, 262,144 2.41 and 2.52.
inline bool far_applies_step(double eps2, int64_t n) { return eps2 == 0.0 && n >= kFarRows; }

// Tile of the default pair kernel: the parts of a device plan start at
// multiples of it.
constexpr int kPartAlign = 256;
// Launches with more i-particles than this run their walks whole in the
// device-resident step (in groups of 512 they have enough of them: a King model
// of 1M has 7,000 walks for 456 CTAs); up to it, whole walks flush at tile ends.
// Step split and whole: King models of 262,144 2.40 and 2.64 ms, 400,000 3.35 and
// 3.45, 524,288 4.27 and 4.27, 700,000 5.42 and 5.37, 1M 8.00 and 7.81.  Larger
// groups leave fewer walks (600,000 particles in groups of 4,096: 7.9 and 31.7).
constexpr int64_t kPlanRows = 400000;

// First entry of part j of n entries in n_parts parts.
__host__ __device__ inline int part_begin(int64_t n, int j, int n_parts, int align) {
    const int64_t units = (n + align - 1) / align, b = units * j / n_parts * align;
    return (int)(b < n ? b : n);
}

// A result row as four (hi, lo) FP32 pairs, without G: the far-field sums
// (acceleration x, y, z and potential) and the sums of a split walk's parts.
__device__ __forceinline__ void load_pairs(const Accp* row, float2 f[4]) {
    const float4* r = reinterpret_cast<const float4*>(row);
    const float4 a = r[0], b = r[1];
    f[0] = make_float2(a.x, a.y);
    f[1] = make_float2(a.z, a.w);
    f[2] = make_float2(b.x, b.y);
    f[3] = make_float2(b.z, b.w);
}
__device__ __forceinline__ void store_pairs(Accp* row, const float2 f[4]) {
    float4* r = reinterpret_cast<float4*>(row);
    r[0] = make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
    r[1] = make_float4(f[2].x, f[2].y, f[3].x, f[3].y);
}
__device__ __forceinline__ double pair_value(float2 v) { return (double)v.x + (double)v.y; }

// The superparticle list the pair kernels run for one descriptor: entries
// [begin, begin + n) of the walk's own list, or of its compacted one, whose
// quarter q starts where quarter q of the walk's list does and follows the
// others in the numbering.  A part of a split walk takes its share of the
// compacted list.  Part 0 adds the far-field sums.
struct SpjList {
    const int32_t* ids;
    int n;
    int begin;
    int after1, after2, after3;  // entries before quarters 1, 2, 3
    int gap1, gap2, gap3;        // id offset minus entry number in those quarters
    bool add_far;
    __device__ __forceinline__ const int32_t* at(int k) const {
        const int e = begin + k;
        return ids + e + (e < after2 ? (e < after1 ? 0 : gap1) : (e < after3 ? gap2 : gap3));
    }
};
__device__ __forceinline__ SpjList spj_list(const Params& p, const WalkDesc& wd) {
    SpjList l;
    if (p.spj_near) {
        const SpjNear c = p.spj_near[wd.root];
        if (c.n[0] >= 0) {
            const int64_t all = wd.n_spj_all;
            const int align = p.part_align ? p.part_align : 1;
            l.ids = p.id_spj_near + (wd.spj_begin - part_begin(all, wd.part, wd.n_parts, align));
            l.after1 = c.n[0];
            l.after2 = l.after1 + c.n[1];
            l.after3 = l.after2 + c.n[2];
            l.gap1 = (int)(all / 4) - l.after1;
            l.gap2 = (int)(all * 2 / 4) - l.after2;
            l.gap3 = (int)(all * 3 / 4) - l.after3;
            const int64_t total = l.after3 + c.n[3];
            l.begin = part_begin(total, wd.part, wd.n_parts, align);
            l.n = part_begin(total, wd.part + 1, wd.n_parts, align) - l.begin;
            l.add_far = c.add_far != 0 && wd.part == 0;
            return l;
        }
    }
    l.ids = p.id_spj + wd.spj_begin;
    l.n = wd.n_spj;
    l.begin = 0;
    l.after1 = l.after2 = l.after3 = 0x7fffffff;
    l.gap1 = l.gap2 = l.gap3 = 0;
    l.add_far = false;
    return l;
}

// Launchers (stream-ordered, asynchronous).
// Far-field pass of a launch; nothing when p.spj_near is null.  Runs after
// reset_counters, before the pair kernel.
cudaError_t launch_far(const Params& p, cudaStream_t s, int num_sms);
cudaError_t launch_fp64(const Params& p, cudaStream_t s, int num_sms);
cudaError_t launch_mixed(const Params& p, cudaStream_t s, int num_sms);
cudaError_t launch_retest(const Params& p, cudaStream_t s, int num_sms);
// Split plan made on the device (pgf_plan.cu).  cap_splits bounds the further
// parts, row0 is the first of cap_rows result rows for them (in part_accp).
struct PlanArgs {
    const WalkDesc* roots;
    int n_root;
    const int32_t* n_root_dev;  // walk count on the device (at most n_root), or null
    const SpjNear* spj_near;    // far-field pass, or null
    int num_sms;
    WalkDesc* walks;
    int32_t* order;
    SplitRec* splits;
    int32_t* n_desc;
    int32_t* n_split;
    int cap_desc, cap_splits, row0;
    int part0_rows;  // Params::part0_rows
    int64_t cap_rows;
};
cudaError_t launch_plan(const PlanArgs& a, cudaStream_t s);
cudaError_t launch_combine_plan(const PlanArgs& a, const Params& p, cudaStream_t s);
// Adds the results of every split walk's parts into its own rows, parts in
// order (deterministic).
// pot_soft and acorr (optional) are the changeover and gradient modes'
// outputs.  pairs: the parts' rows are (hi, lo) pairs without G (the
// warp-specialised and gradient kernels; epi_acc: the latter's a_i, added
// here), else FP64 with G applied.
cudaError_t launch_combine_parts(const SplitRec* recs, int n_recs, Accp* accp, int32_t* nnb, double* pot_soft,
                                 Accp* acorr, const Accp* epi_acc, bool pairs, double G, cudaStream_t s);
// EpiRel rows of every walk of a launch (its roots), and the AccF32 forms of
// epi_acc64 (gradient mode; null otherwise).
cudaError_t launch_epi_rel(const Params& p, EpiRel* out, AccF32* out_acc, cudaStream_t s, int num_sms);
// Builds the (hi, lo) FP32 copies of the EPJ / SPJ arrays.
cudaError_t launch_split_j(const EpjMix* epj, int64_t n_epj, EpjF32* epj32, const SpjMix* spj, int64_t n_spj,
                           SpjF32* spj32, cudaStream_t s);
// Warp-specialised kernel, variants 0..kNumWsVariants-1 (see pgf_kernels_ws.cu).
constexpr int kNumWsVariants = 8;
// TMA descriptors of the (hi, lo) EPJ and SPJ arrays (rows of 32 and 64
// bytes, boxes one row high), rebuilt at every send.
struct TensorMaps {
    CUtensorMap epj;
    CUtensorMap spj;
    bool valid = false;
};
cudaError_t launch_ws(const Params& p, cudaStream_t s, int num_sms, int variant, const TensorMaps* tm);
// The default variant on FP64 records alone (epi, EpjMix, SpjMix), for callers
// whose data has no FP32 forms.
cudaError_t launch_ws_fp64_records(const Params& p, cudaStream_t s, int num_sms);
// Whether warp-specialised variant v stages its tiles with TMA (needs TensorMaps).
bool ws_variant_uses_tma(int variant);
// Neighbour search (counts only, SPJ lists ignored) with the warp-specialised kernel.
cudaError_t launch_ws_search(const Params& p, cudaStream_t s, int num_sms);
// Soft force with the changeover correction of neighbours fused in.
cudaError_t launch_ws_changeover(const Params& p, cudaStream_t s, int num_sms);
// KDKDK_4TH gradient-correction pass (pgf_kernels_gradient.cu).
cudaError_t launch_gradient(const Params& p, cudaStream_t s, int num_sms);

}  // namespace pgf
