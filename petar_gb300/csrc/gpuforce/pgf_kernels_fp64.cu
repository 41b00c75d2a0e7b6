// Plain FP64 soft-force kernel: FP64 throughout, the option for verification
// and the baseline the mixed-precision kernel is measured against.
//
// The reference's FP64 functors (src/soft_force.hpp:53-71 for EP-EP with the
// linear cutoff, :174-195 for the EP-SP quadrupole) over the work queue.
// GB300 issues an FP64 instruction per warp and SM quadrant once in 64
// cycles, so the time is the number of FP64 warp instructions:
// * EPJ farther than any neighbour or cutoff radius from the walk's box
//   (classified once per staged entry, in FP32 with a margin) are plain
//   gravity, 18 FP64 operations a pair instead of 28; the others keep the
//   cutoff and the oracle's exact neighbour expression, so counts are
//   bit-exact;
// * 1/r is one third-order Householder step (Householder, The Numerical
//   Treatment of a Single Nonlinear Equation, 1970) from the hardware's
//   reciprocal square root estimate: its error, a few 2^-20 of the result,
//   is cubed;
// * the quadrupole in its traceless form, 38 operations a pair from 48;
// * a pass holds up to 256 i, one per thread, and as many j-slices as fit,
//   so that small walks and remainders leave few lanes idle.
// Measured on GB300 (kernel, event-timed): 65,536 stars 55 -> 34.3 ms, 10,000
// stars 9.5 -> 3.2 ms; the operations above take 27.5 ms at 65,536.
#include "pgf_internal.cuh"

namespace pgf {
namespace {

constexpr int kT = 256;  // threads per block = i per pass = j per tile
constexpr int kW = kT / 32;

struct Smem64 {
    double x[kT], y[kT], z[kT], m[kT];
    double q[6][kT];  // EP tiles: r_search in q[0]
    double c[kT];
    double red[4][kT];
    int cnt[kT];
    int wn[kW];
    int w;
};

// 1/sqrt(a).  The step from the estimate is for normal a; r^2 that underflowed
// or overflowed (a source 1e154 away: 1/r is 0) takes the library's function.
__device__ __forceinline__ double rsqrt_fp64(double a) {
    if ((((unsigned)__double2hiint(a) >> 20) - 1u) >= 0x7feu) return rsqrt(a);
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// j-slices of a pass of n i: the count (of those that fit) whose threads
// issue the fewest warp instructions per j.
__device__ __forceinline__ int slices64(int n) {
    int best = 1, cost = (n + 31) / 32;  // warps per slice, as cost / best
    for (int k = 2; k * n <= kT; ++k) {
        const int c = (k * n + 31) / 32;
        if (c * best <= cost * k) {
            best = k;
            cost = c;
        }
    }
    return best;
}

__global__ __launch_bounds__(kT, 2) void fp64_kernel(Params p) {
    if (p.input_err && *p.input_err) return;  // the inputs failed their check: run nothing
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem64& s = *reinterpret_cast<Smem64*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double eps2 = p.eps2;
    const int n_walk = walk_count(p);
    for (;;) {
        __syncthreads();
        if (tid == 0) s.w = atomicAdd(p.queue_head, 1);
        __syncthreads();
        const int wq = s.w;
        if (wq >= n_walk) break;
        const WalkDesc wd = p.walks[p.order[wq]];
        const double rcut2 = wd.rcut2;
        const float rc2 = __double2float_ru(rcut2), rsmax2 = wd.rs_max * wd.rs_max * 1.000001f;
        const float chx = wd.ch[0], chy = wd.ch[1], chz = wd.ch[2];
        const float hmax = fmaxf(wd.hx, fmaxf(wd.hy, wd.hz));
        const float cmax = fmaxf(fabsf(chx), fmaxf(fabsf(chy), fabsf(chz)));
        const int n_pass = (wd.n_i + kT - 1) / kT, per_pass = n_pass ? (wd.n_i + n_pass - 1) / n_pass : 0;
        for (int ic = 0; ic < wd.n_i; ic += per_pass) {
            const int S = min(per_pass, wd.n_i - ic);
            const int n_js = slices64(S);
            const int js = tid / S, li = ic + tid - js * S;
            const bool valid = js < n_js;
            double xi = 0, yi = 0, zi = 0, rsi = 0;
            if (valid) {
                const EpiDev e = p.epi[wd.i_root + li];
                xi = e.x;
                yi = e.y;
                zi = e.z;
                rsi = e.rs;
            }
            double ax = 0, ay = 0, az = 0, pe = 0;  // pe: minus the potential
            int nnb = 0;
            for (int t0 = 0; t0 < wd.n_epj; t0 += kT) {
                const int nt = min(kT, wd.n_epj - t0);
                bool near = false;
                EpjMix j{};
                double m = 0, rs = 0;
                if (tid < nt) {
                    const int id = p.id_epj[wd.epj_begin + t0 + tid];
                    j = p.epj[id];
                    m = p.epj_m64[id];
                    rs = p.epj_rs64[id];
                    // Conservative: 0.1% over the radii and the FP32 rounding
                    // of the absolute coordinates.  A NaN among them (which
                    // fmaxf hides in d2) makes the entry near.
                    const EpjF32 f = p.epj32[id];
                    const float dx = fabsf(f.xh - chx), dy = fabsf(f.yh - chy), dz = fabsf(f.zh - chz);
                    const float ex = fmaxf(dx - wd.hx, 0.f), ey = fmaxf(dy - wd.hy, 0.f), ez = fmaxf(dz - wd.hz, 0.f);
                    const float d2 = fmaf(ex, ex, fmaf(ey, ey, ez * ez));
                    const float R = sqrtf(fmaxf(fmaxf(rsmax2, f.rs2), rc2));
                    const float Rm = R * 1.001f + 1e-6f * ((dx + dy + dz) + hmax + cmax);
                    near = !(d2 > Rm * Rm);
                }
                const unsigned bn = __ballot_sync(0xffffffffu, near);
                __syncthreads();  // the previous tile is done with
                if (lane == 0) s.wn[warp] = __popc(bn);
                __syncthreads();
                int before = 0, nn = 0;
#pragma unroll
                for (int k = 0; k < kW; ++k) {
                    before += k < warp ? s.wn[k] : 0;
                    nn += s.wn[k];
                }
                // far entries from the front, near ones from the back
                if (tid < nt) {
                    before += __popc(bn & ((1u << lane) - 1u));
                    const int e = near ? kT - 1 - before : tid - before;
                    s.x[e] = j.x;
                    s.y[e] = j.y;
                    s.z[e] = j.z;
                    s.m[e] = m;
                    s.q[0][e] = rs;
                }
                __syncthreads();
                if (valid) {
                    const int nf = nt - nn;
                    const int pf = (nf + n_js - 1) / n_js;
                    const int f1 = min(nf, (js + 1) * pf);
#pragma unroll 4
                    for (int k = js * pf; k < f1; ++k) {
                        const double dx = s.x[k] - xi, dy = s.y[k] - yi, dz = s.z[k] - zi;
                        const double ri = rsqrt_fp64(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
                        const double mr = s.m[k] * ri;
                        const double mr3 = mr * (ri * ri);
                        ax = fma(mr3, dx, ax);
                        ay = fma(mr3, dy, ay);
                        az = fma(mr3, dz, az);
                        pe += mr;
                    }
                    const int pn = (nn + n_js - 1) / n_js;
                    const int k1 = min(nn, (js + 1) * pn);
                    for (int q = js * pn; q < k1; ++q) {
                        const int k = kT - 1 - q;
                        const double dx = __dsub_rn(xi, s.x[k]);
                        const double dy = __dsub_rn(yi, s.y[k]);
                        const double dz = __dsub_rn(zi, s.z[k]);
                        const double r2 =
                            __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
                        const double r2e = __dadd_rn(r2, eps2);
                        const double rs = rsi > s.q[0][k] ? rsi : s.q[0][k];
                        nnb += r2e < __dmul_rn(rs, rs) ? 1 : 0;
                        const double r2c = r2e > rcut2 ? r2e : rcut2;
                        const double ri = rsqrt(r2c);
                        const double mr = s.m[k] * ri;
                        const double mr3 = mr * ri * ri;
                        ax -= mr3 * dx;
                        ay -= mr3 * dy;
                        az -= mr3 * dz;
                        pe += mr;
                    }
                }
            }
            for (int t0 = 0; t0 < wd.n_spj; t0 += kT) {
                const int nt = min(kT, wd.n_spj - t0);
                __syncthreads();
                if (tid < nt) {
                    const int id = p.id_spj[wd.spj_begin + t0 + tid];
                    const SpjMix j = p.spj[id];
                    const SpjQ64 q = p.spj_q64[id];
                    s.x[tid] = j.x;
                    s.y[tid] = j.y;
                    s.z[tid] = j.z;
                    s.m[tid] = q.m;
                    // -Q = tr(q) I - 3 q and -c = tr(q) eps^2
                    const double tr = q.q[0] + q.q[1] + q.q[2];
                    for (int c = 0; c < 3; ++c) s.q[c][tid] = fma(-3.0, q.q[c], tr);
                    for (int c = 3; c < 6; ++c) s.q[c][tid] = -3.0 * q.q[c];
                    s.c[tid] = tr * eps2;
                }
                __syncthreads();
                if (valid) {
                    const int ps = (nt + n_js - 1) / n_js;
                    const int k1 = min(nt, (js + 1) * ps);
#pragma unroll 2
                    for (int k = js * ps; k < k1; ++k) {
                        // with u = d.(-Q).d - c and t = u / r^5:
                        // acc += (m/r^3 - 2.5 t/r^2) d + (-Q).d / r^5, -pot += m/r - 0.5 t
                        const double dx = s.x[k] - xi, dy = s.y[k] - yi, dz = s.z[k] - zi;
                        const double ri = rsqrt_fp64(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
                        const double qxy = s.q[3][k], qxz = s.q[4][k], qyz = s.q[5][k], m = s.m[k];
                        const double qx = fma(s.q[0][k], dx, fma(qxy, dy, qxz * dz));
                        const double qy = fma(qxy, dx, fma(s.q[1][k], dy, qyz * dz));
                        const double qz = fma(qxz, dx, fma(qyz, dy, s.q[2][k] * dz));
                        const double u = fma(qx, dx, fma(qy, dy, fma(qz, dz, s.c[k])));
                        const double ri2 = ri * ri, ri3 = ri2 * ri, ri5 = ri3 * ri2;
                        const double t = u * ri5;
                        const double A = fma(t * ri2, -2.5, m * ri3);
                        ax = fma(A, dx, fma(ri5, qx, ax));
                        ay = fma(A, dy, fma(ri5, qy, ay));
                        az = fma(A, dz, fma(ri5, qz, az));
                        pe = fma(t, -0.5, fma(m, ri, pe));
                    }
                }
            }
            // Sum the slices.
            __syncthreads();
            s.red[0][tid] = ax;
            s.red[1][tid] = ay;
            s.red[2][tid] = az;
            s.red[3][tid] = pe;
            s.cnt[tid] = nnb;
            __syncthreads();
            if (valid && js == 0) {
                for (int k = 1; k < n_js; ++k) {
                    const int src = k * S + tid;
                    ax += s.red[0][src];
                    ay += s.red[1][src];
                    az += s.red[2][src];
                    pe += s.red[3][src];
                    nnb += s.cnt[src];
                }
                const double G = p.G;
                const int gi = wd.i_begin + li;
                p.out_accp[gi] = Accp{G * ax, G * ay, G * az, -(G * pe)};
                p.out_nnb[gi] = nnb;
            }
        }
    }
}

}  // namespace

cudaError_t launch_fp64(const Params& p, cudaStream_t s, int num_sms) {
    if (p.n_walk <= 0) return cudaSuccess;
    static int per_sm = 0;
    if (per_sm == 0) {
        cudaError_t e = cudaFuncSetAttribute(fp64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem64));
        if (e != cudaSuccess) return e;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fp64_kernel, kT, sizeof(Smem64));
        if (e != cudaSuccess) return e;
        if (per_sm < 1) per_sm = 1;
    }
    int grid = num_sms * per_sm;
    if (grid > p.n_walk) grid = p.n_walk;
    fp64_kernel<<<grid, kT, sizeof(Smem64), s>>>(p);
    return cudaGetLastError();
}

}  // namespace pgf
