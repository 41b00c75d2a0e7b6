// Far-field pass: the force of distant superparticles on a walk's i-particles
// through a local expansion about the walk centre (pgf_localexp.cuh), run
// before the interaction kernel of the same launch.
//
// An EP-SP pair costs the interaction kernel 33 FP32 operations, and that
// kernel is FP32-pipe bound.  A superparticle at distance D from a walk of
// radius R (the farthest i from the walk centre) with R / D small acts on
// all n_i particles through the same few derivatives of its field: expanding
// it costs about 700 operations once, however many i there are.  On the 1M
// binary Plummer workload 51% of the EP-SP pairs pass the test below (16% at
// 65k stars, 34% in a King 1M model with theta = 0.4).
//
// Test.  A source is expanded when the dropped terms, bounded for an i at
// distance R straight towards it, stay below 2^-23 of the source's own force,
// half the FP32 rounding of a pair (2e-7 over sources on one side):
// 10.8 rho^8 for the monopole (rho = R / D) and 105 rho^6 |Q| / (m D^2) for the
// quadrupole, whose terms end two orders earlier; these are the first dropped
// terms, 9 and 84, and at rho = 0.14 a fifth and a quarter of them for the rest.
// The bound holds source by source because nothing averages truncation out
// where a walk's distant sources lie on one side: with 2e-6 for each of the two
// terms (64% of the pairs at the 1M workload) such a walk's force was off by
// 1.3e-6 where its pairs are off by 2.4e-7.  The leading terms (potential and
// uniform force) are summed as (hi, lo) FP32 pairs.
//
// One CTA per walk, from the same queue order as the interaction kernel (a
// split walk is handled whole; its parts share the compacted list).  Each of
// its four or eight warps takes a quarter of the list, or half of one, by itself: the near
// ids are appended to the compacted list that the interaction kernel reads
// instead, the far sources go to a ring in shared memory, and whenever 32 are
// there every lane expands one into 81 coefficients in its registers.  The
// lanes' coefficients are summed by a shuffle reduce-scatter, and each i
// evaluates the polynomial; the sums go to the i's result row, to which the
// interaction kernel adds its pairs.  The order of every sum is fixed by the
// list, so results do not depend on the grid.
//
// Measured on GB300 at the 1M binary workload (all walks in one launch): the
// pair kernel alone 22.7 ms; this pass 2.6 ms and the pair kernel 13.6 ms
// after it, with the force error against FP64 at median 6.4e-8 / p99.9 4.9e-7
// from 7.3e-8 / 5.5e-7.  FP64 instructions are what costs here (the FP64 pipe
// issues one per warp in 64 cycles): with the leading sums and the results in
// FP64 the pass took 1 ms more.
#include "pgf_internal.cuh"
#include "pgf_localexp.cuh"

namespace pgf {
namespace {

constexpr int kRing = 64;      // per warp: 32 sources arrive while fewer than 32 wait
constexpr int kMinI = 32;      // fewer i: direct pairs (33 n_i operations) cost about as much
constexpr float kTrunc = 1.f / 8388608.f;  // truncation of a source as a share of its force
constexpr float kRhoMax = 0.1f;            // 10.8 rho^8 < kTrunc, without quadrupole
constexpr float kMonoErr = 10.8f, kQuadErr = 105.f;
constexpr int kPad = 96;  // coefficients padded to 3 per lane

constexpr int kStage = 2048;  // list entries of half a quarter

template <int W>
struct FarSmem {
    float src[W][9][kRing];  // x, y, z, m, and the five quadrupole moments (QuadOp), scaled
    float red[W][kPad];
    float2 lead[W][4];  // rows 0 and 1 as (hi, lo)
    float L[kFarCoefs + 3];
    float4 ev[kFarCoefs + 3];  // phi and gradient coefficients
    float rmax[W];
    int n_near[W], n_far[W];
    int32_t stage[W == 8 ? 4 : 1][W == 8 ? kStage : 1];  // near ids of a quarter's second half
    int w;
};

struct SpjRec {
    float4 a, b, c;
    float2 d;
};
__device__ __forceinline__ SpjRec load_spj(const SpjF32* __restrict__ spj, int id) {
    SpjRec r{};
    if (id >= 0) {
        const float4* src = reinterpret_cast<const float4*>(spj + id);
        r.a = __ldg(src);
        r.b = __ldg(src + 1);
        r.c = __ldg(src + 2);
        r.d = __ldg(reinterpret_cast<const float2*>(src + 3));
    }
    return r;
}

// A shared-memory load that keeps its place: hoisted to the front, the 80
// coefficients of the evaluation spill.
__device__ __forceinline__ float4 ld_in_order(const float4* a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(static_cast<unsigned>(__cvta_generic_to_shared(a))));
    return v;
}

// Rows N .. kFarOrder of the expansion at one i: adds phi and its gradient.
template <int N>
__device__ __forceinline__ void eval_rows(const float (&p1)[2 * kFarOrder + 1], const float (&p2)[2 * kFarOrder + 1],
                                          float x, float y, float z, float r2, const float4* __restrict__ ev,
                                          float4& o) {
    if constexpr (N <= kFarOrder) {
        float r[2 * kFarOrder + 1];
        regular_row<N>(p1, p2, x, y, z, r2, r);
#pragma unroll
        for (int k = 0; k < 2 * N + 1; ++k) {
            const float4 e = ld_in_order(ev + N * N + k);
            o.w = fmaf(e.x, r[k], o.w);
            if (N < kFarOrder) {
                o.x = fmaf(e.y, r[k], o.x);
                o.y = fmaf(e.z, r[k], o.y);
                o.z = fmaf(e.w, r[k], o.z);
            }
        }
        eval_rows<N + 1>(r, p1, x, y, z, r2, ev, o);
    }
}

// One step of the reduce-scatter over lanes: the first H values of v become
// this lane's half of the 2H summed with its partner's.
template <int H>
__device__ __forceinline__ void halve(float (&v)[kPad], int lane, int bit) {
    const bool up = lane & bit;
#pragma unroll
    for (int k = 0; k < H; ++k) {
        const float send = up ? v[k] : v[k + H];
        const float keep = up ? v[k + H] : v[k];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
}

template <int W>
__global__ __launch_bounds__(W * 32, W == 4 ? 3 : 1) void far_kernel(Params p) {
    constexpr int kT = W * 32;
    static_assert(W == 4 || W == 8, "a quarter of the list, or half of one, per warp");
    if (p.input_err && *p.input_err) return;  // the inputs failed their check: run nothing
    __shared__ FarSmem<W> s;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned lane_lt = (1u << lane) - 1u;
    const int n_walk = p.n_root < p.n_walk ? p.n_root : walk_count(p);
    for (;;) {
        __syncthreads();
        if (t == 0) s.w = atomicAdd(p.far_queue, 1);
        __syncthreads();
        if (s.w >= n_walk) break;
        const int w = p.n_root < p.n_walk ? s.w : p.order[s.w];
        const WalkDesc wd = p.walks[w];
        const int n_spj = wd.n_spj_all;
        if (wd.n_i < kMinI || n_spj == 0) {
            if (t == 0) p.spj_near[w].n[0] = -1;
            continue;
        }
        // Radius of the walk's particles.
        float r2m = 0.f;
        for (int i = t; i < wd.n_i; i += kT) {
            const float4 e = __ldg(reinterpret_cast<const float4*>(p.epi_rel + wd.i_root + i));
            r2m = fmaxf(r2m, fmaf(e.x, e.x, fmaf(e.y, e.y, e.z * e.z)));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) r2m = fmaxf(r2m, __shfl_xor_sync(0xffffffffu, r2m, o));
        if (lane == 0) s.rmax[warp] = r2m;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < W; ++k) r2m = fmaxf(r2m, s.rmax[k]);
        const float R = sqrtf(r2m) * 1.00001f;
        if (!(R > 1e-18f && R < 1e18f)) {
            if (t == 0) p.spj_near[w].n[0] = -1;
            continue;
        }
        // Lengths in units of a power of two at the nearest distance expanded,
        // so that the powers of D and x stay in FP32's range.
        int ex;
        (void)frexpf(R / kRhoMax, &ex);
        const float inv = ldexpf(1.f, -ex);
        const float Rs = R * inv;  // in (0.05, 0.1]
        const float lim2 = (Rs / kRhoMax) * (Rs / kRhoMax);
        const float kq = (Rs * Rs * Rs) * (Rs * Rs * Rs) * (kQuadErr / kTrunc);
        const float km = (Rs * Rs) * ((Rs * Rs * Rs) * (Rs * Rs * Rs)) * (kMonoErr / kTrunc);
        const float chx = wd.ch[0], chy = wd.ch[1], chz = wd.ch[2];
        const float clx = wd.cl[0], cly = wd.cl[1], clz = wd.cl[2];

        float L[kFarCoefs], lo[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < kFarCoefs; ++k) L[k] = 0.f;
        // Each warp takes its quarter of the list, or half of it, by itself: 32
        // entries at a time, with the records loaded one chunk ahead and the
        // ids two.  The near ids of a second half wait in shared memory for
        // the number of those before them; quarters too long for that are
        // left to the first warp.
        const int quarter = W == 8 ? warp >> 1 : warp, half = W == 8 ? warp & 1 : 0;
        int b0 = (int)((int64_t)n_spj * quarter / 4), n_w = (int)((int64_t)n_spj * (quarter + 1) / 4) - b0;
        int32_t* const quarter_out = p.id_spj_near + wd.spj_begin + b0;
        if (W == 8) {
            const int first = n_w <= 2 * kStage ? (n_w + 1) >> 1 : n_w;
            if (half) b0 += first;
            n_w = half ? n_w - first : first;
        }
        int32_t* __restrict__ const near_out = half ? s.stage[W == 8 ? quarter : 0] : quarter_out;
        float (*const src)[kRing] = s.src[warp];
        int head = 0, waiting = 0, n_near = 0, n_far = 0;
        const int32_t* __restrict__ ids = p.id_spj + wd.spj_begin + b0;
        int id = lane < n_w ? __ldg(ids + lane) : -1;
        int id_next = 32 + lane < n_w ? __ldg(ids + 32 + lane) : -1;
        SpjRec rec = load_spj(p.spj32, id);
        for (int base = 0; base < n_w || waiting > 0; base += 32) {
            if (base < n_w) {
                const float hx = ((rec.a.x - chx) + (rec.b.x - clx)) * inv;
                const float hy = ((rec.a.y - chy) + (rec.b.y - cly)) * inv;
                const float hz = ((rec.a.z - chz) + (rec.b.z - clz)) * inv;
                const float m = rec.a.w;
                const float i2 = inv * inv;
                const QuadOp q = quad_op(rec.c.x * i2, rec.c.y * i2, rec.c.z * i2, rec.c.w * i2, rec.d.x * i2, rec.d.y * i2);
                const float qn = sqrtf(fmaf(rec.c.x, rec.c.x, fmaf(rec.c.y, rec.c.y, rec.c.z * rec.c.z)) +
                                       2.f * fmaf(rec.c.w, rec.c.w, fmaf(rec.d.x, rec.d.x, rec.d.y * rec.d.y))) * i2;
                const float d2 = fmaf(hx, hx, fmaf(hy, hy, hz * hz));
                const float d4 = d2 * d2;
                const bool valid = id >= 0;
                const bool far = valid && d2 >= lim2 && d2 < 1e16f && fabsf(m) < 1e30f &&
                                 fmaf(km, fabsf(m), kq * qn) <= fabsf(m) * (d4 * d4);
                const int id_cur = id;
                id = id_next;
                id_next = base + 64 + lane < n_w ? __ldg(ids + base + 64 + lane) : -1;
                rec = load_spj(p.spj32, id);
                const unsigned bf = __ballot_sync(0xffffffffu, far);
                const unsigned bn = __ballot_sync(0xffffffffu, valid && !far);
                if (far) {
                    const int e = (head + waiting + __popc(bf & lane_lt)) & (kRing - 1);
                    src[0][e] = hx;
                    src[1][e] = hy;
                    src[2][e] = hz;
                    src[3][e] = m;
                    src[4][e] = q.ppr;
                    src[5][e] = q.ppi;
                    src[6][e] = q.pzr;
                    src[7][e] = q.pzi;
                    src[8][e] = q.zz;
                } else if (valid) {
                    near_out[n_near + __popc(bn & lane_lt)] = id_cur;
                }
                const int nf = __popc(bf);
                waiting += nf;
                n_far += nf;
                n_near += __popc(bn);
                __syncwarp();
                if (waiting < 32 && base + 32 < n_w) continue;
            }
            if (waiting == 0) break;
            // One source per lane (fewer in the last batch).
            float hx = 1.f, hy = 0.f, hz = 0.f, m = 0.f;
            QuadOp q{};
            if (lane < waiting) {
                const int e = (head + lane) & (kRing - 1);
                hx = src[0][e];
                hy = src[1][e];
                hz = src[2][e];
                m = src[3][e];
                q.ppr = src[4][e];
                q.ppi = src[5][e];
                q.pzr = src[6][e];
                q.pzi = src[7][e];
                q.zz = src[8][e];
            }
            __syncwarp();  // the ring's slots may be written again
            const int take = min(32, waiting);
            head = (head + take) & (kRing - 1);
            waiting -= take;
            const float ri = rsqrt_approx(fmaf(hx, hx, fmaf(hy, hy, hz * hz)));
            add_source(hx, hy, hz, ri, m, q, L, lo);
        }
        if (lane == 0) {
            s.n_near[warp] = n_near;
            s.n_far[warp] = n_far;
        }
        __syncthreads();
        n_far = 0;
#pragma unroll
        for (int k = 0; k < W; ++k) n_far += s.n_far[k];
        if (half) {
            const int before = s.n_near[warp - 1], n = s.n_near[warp];
            for (int k = lane; k < n; k += 32) quarter_out[before + k] = near_out[k];
        }
        if (t == 0) {
            SpjNear r{};
#pragma unroll
            for (int q = 0; q < 4; ++q) r.n[q] = W == 8 ? s.n_near[(2 * q) % W] + s.n_near[(2 * q + 1) % W] : s.n_near[q];
            r.add_far = n_far > 0 ? 1 : 0;
            p.spj_near[w] = r;
        }
        if (n_far == 0) continue;

        // Sum over the threads: rows 0 and 1 as (hi, lo) pairs, the others by a
        // reduce-scatter (lane l ends with three coefficients).
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float2 v = make_float2(L[k], lo[k]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                v = add_pair(v, make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o)));
            if (lane == 0) s.lead[warp][k] = v;
        }
        {
            float v[kPad];
#pragma unroll
            for (int k = 0; k < kPad; ++k) v[k] = k < kFarCoefs ? L[k] : 0.f;
            halve<48>(v, lane, 16);
            halve<24>(v, lane, 8);
            halve<12>(v, lane, 4);
            halve<6>(v, lane, 2);
            halve<3>(v, lane, 1);
            const int b = (lane & 16 ? 48 : 0) + (lane & 8 ? 24 : 0) + (lane & 4 ? 12 : 0) + (lane & 2 ? 6 : 0) +
                          (lane & 1 ? 3 : 0);
#pragma unroll
            for (int k = 0; k < 3; ++k) s.red[warp][b + k] = v[k];
        }
        __syncthreads();
        if (t < kFarCoefs) {
            float v = 0.f;
#pragma unroll
            for (int k = 0; k < W; k += 2) v += s.red[k][t] + s.red[k + 1][t];
            s.L[t] = v;
        }
        __syncthreads();
        if (t < kFarCoefs) {
            int n = 0;
            while ((n + 1) * (n + 1) <= t) ++n;
            float4 e;
            eval_coef(n, t - n * n, [&](int i) { return s.L[i]; }, e.x, e.y, e.z, e.w);
            s.ev[t] = e;
        }
        float2 lead[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            lead[k] = s.lead[0][k];
#pragma unroll
            for (int q = 1; q < W; ++q) lead[k] = add_pair(lead[k], s.lead[q][k]);
        }
        __syncthreads();
        const float inv2 = inv * inv;  // powers of two: scaling the results is exact
#pragma unroll 1
        for (int i = t; i < wd.n_i; i += kT) {
            const int gi = wd.i_begin + i;
            const float4 e = __ldg(reinterpret_cast<const float4*>(p.epi_rel + wd.i_root + i));
            const float x = e.x * inv, y = e.y * inv, z = e.z * inv;
            float r0[2 * kFarOrder + 1] = {1.f}, rz[2 * kFarOrder + 1] = {};
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            eval_rows<1>(r0, rz, x, y, z, fmaf(x, x, fmaf(y, y, z * z)), s.ev, o);
            // rows 0: phi = L_00, gradient (Re L_11, Im L_11, L_10)
            const float2 ax = add_pair(lead[2], make_float2(o.x, 0.f)), ay = add_pair(lead[3], make_float2(o.y, 0.f));
            const float2 az = add_pair(lead[1], make_float2(o.z, 0.f)), ph = add_pair(lead[0], make_float2(o.w, 0.f));
            const float2 f[4] = {make_float2(ax.x * inv2, ax.y * inv2), make_float2(ay.x * inv2, ay.y * inv2),
                                 make_float2(az.x * inv2, az.y * inv2), make_float2(-ph.x * inv, -ph.y * inv)};
            store_pairs(p.out_accp + gi, f);
        }
    }
}

// EPI rows about their walk's centre, one warp per walk, more where walks are
// few (3,000 stars: 16 -> 6 us); conversions on the integer pipe (58 -> 24 us
// for 1M rows).
__global__ __launch_bounds__(256) void epi_rel_kernel(Params p, EpiRel* __restrict__ out, AccF32* __restrict__ out_acc) {
    const int n_walk = p.n_root < p.n_walk ? p.n_root : walk_count(p);
    if (n_walk <= 0) return;
    const int lane = threadIdx.x & 31;
    const int warps = (int)((gridDim.x * blockDim.x) >> 5), m = min(16, max(1, warps / n_walk));
    for (int k = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); k < n_walk * m; k += warps) {
        const WalkDesc wd = p.walks[p.n_root < p.n_walk ? k / m : p.order[k / m]];
        for (int i = (k % m) * 32 + lane; i < wd.n_i; i += 32 * m) {
            const int r = wd.i_root + i;
            out[r] = make_epi_rel(p.epi[r], wd.cx, wd.cy, wd.cz, (float)p.eps2);
            if (out_acc) out_acc[r] = make_acc32(p.epi_acc64[r].x, p.epi_acc64[r].y, p.epi_acc64[r].z);
        }
    }
}

}  // namespace

cudaError_t launch_epi_rel(const Params& p, EpiRel* out, AccF32* out_acc, cudaStream_t s, int num_sms) {
    if (p.n_walk <= 0) return cudaSuccess;
    const int64_t want = ((int64_t)(p.n_root < p.n_walk ? p.n_root : p.n_walk) + 7) / 8;
    const int grid = (int)(want < num_sms * 8 ? want : num_sms * 8);
    epi_rel_kernel<<<grid, 256, 0, s>>>(p, out, out_acc);
    return cudaGetLastError();
}

namespace {

template <int W>
cudaError_t launch_far_t(const Params& p, cudaStream_t s, int num_sms) {
    static int per_sm = 0;
    if (per_sm == 0) {
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, far_kernel<W>, W * 32, 0);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) per_sm = 1;
    }
    int grid = num_sms * per_sm;
    if (grid > p.n_walk) grid = p.n_walk;
    far_kernel<W><<<grid, W * 32, 0, s>>>(p);
    return cudaGetLastError();
}

}  // namespace

// Eight warps per walk where the walks leave SMs with one or none (200-walk
// calls on 262,144 binary stars: this kernel 96 -> 69 us a call, on 1M binaries
// 124 -> 94), else four.  The rule looks at the dispatch's i-particles, not at
// the launch, so that results do not depend on the pipeline stages.
cudaError_t launch_far(const Params& p, cudaStream_t s, int num_sms) {
    if (!p.spj_near || p.n_walk <= 0) return cudaSuccess;
    return p.far_wide ? launch_far_t<8>(p, s, num_sms) : launch_far_t<4>(p, s, num_sms);
}

}  // namespace pgf
