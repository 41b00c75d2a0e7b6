// Walk splitting on the device, for launches whose lists are built or checked
// there (the device-resident step and the allocation-free entry point): the
// counterpart of the host's split plan in pgf_api.cu.
//
// Few walks leave the GPU waiting for the most expensive one.  One CTA reads
// the walks, gives each that costs more than a sixteenth of one SM's even
// share (more where the result rows would not fit) up to 32 parts, and writes the descriptors, the work-queue order and
// the records of what to add up.  Parts are cut at multiples of 256 list
// entries, the pair kernel's tile: with partial sums flushed at every tile's
// end (Params::flush_tiles) a split walk adds the same FP32 terms as a whole
// one, and the results agree to the 2^-48 of the (hi, lo) sums.
#include "pgf_internal.cuh"

namespace pgf {
namespace {

constexpr int kPlanThreads = 1024;
constexpr int kPlanBuckets = 256;

struct PlanSmem {
    unsigned long long warp_tot[kPlanThreads / 32];
    longlong2 warp_scan[kPlanThreads / 32];  // further parts, their rows
    int hist[kPlanBuckets], start[kPlanBuckets];
    unsigned long long total;
    longlong2 all;
};

__device__ __forceinline__ int plan_bucket(unsigned long long cost) {
    if (cost < 2) return 0;
    const int b = (int)(log2f((float)cost) * 6.f);
    return b < kPlanBuckets ? b : kPlanBuckets - 1;
}

struct WalkCost {
    int n_spj;
    unsigned long long cost;
};

__device__ __forceinline__ WalkCost walk_cost(const PlanArgs& a, int k, const WalkDesc& d) {
    WalkCost c;
    c.n_spj = d.n_spj;
    if (a.spj_near) {
        const SpjNear n = a.spj_near[k];
        if (n.n[0] >= 0) c.n_spj = (n.n[0] + n.n[1]) + (n.n[2] + n.n[3]);
    }
    // An EP-SP pair costs about twice an EP-EP pair.
    c.cost = (unsigned long long)d.n_i * ((unsigned long long)d.n_epj + 2ull * (unsigned long long)c.n_spj);
    return c;
}

__device__ __forceinline__ int walk_parts(const WalkDesc& d, const WalkCost& c, unsigned long long target) {
    if (c.cost <= target) return 1;
    const int te = (d.n_epj + kPartAlign - 1) / kPartAlign, ts = (c.n_spj + kPartAlign - 1) / kPartAlign;
    const unsigned long long want = (c.cost + target - 1) / target;
    const int most = min(32, max(te, ts));
    return want < (unsigned long long)most ? (int)want : max(1, most);
}

__global__ __launch_bounds__(kPlanThreads) void plan_kernel(PlanArgs a) {
    __shared__ PlanSmem s;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int n_root = a.n_root_dev ? min(*a.n_root_dev, a.n_root) : a.n_root;
    const int chunk = (n_root + kPlanThreads - 1) / kPlanThreads;
    const int b = min(n_root, t * chunk), e = min(n_root, b + chunk);
    for (int k = t; k < kPlanBuckets; k += kPlanThreads) s.hist[k] = 0;
    unsigned long long sum = 0;
    for (int k = b; k < e; ++k) sum += walk_cost(a, k, a.roots[k]).cost;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) s.warp_tot[warp] = sum;
    __syncthreads();
    if (t == 0) {
        unsigned long long v = 0;
        for (int k = 0; k < kPlanThreads / 32; ++k) v += s.warp_tot[k];
        s.total = v;
    }
    __syncthreads();
    // Further parts and their result rows, scanned over the walks.  A plan
    // that does not fit its arrays is tried again with larger parts, down to
    // half an SM's share; then no walk is split.
    unsigned long long target = 0;
    long long parts = 0, rows = 0;
    longlong2 v = make_longlong2(0, 0);
    bool fits = false;
    for (int div = 16; div >= 2 && !fits; div >>= 1) {
        target = s.total / ((unsigned long long)div * (unsigned long long)a.num_sms) + 1;
        parts = rows = 0;
        for (int k = b; k < e; ++k) {
            const WalkDesc d = a.roots[k];
            const int p = walk_parts(d, walk_cost(a, k, d), target) - 1;
            parts += p;
            if (p > 0) rows += (long long)(p + a.part0_rows) * d.n_i;
        }
        v = make_longlong2(parts, rows);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long px = __shfl_up_sync(0xffffffffu, v.x, o), py = __shfl_up_sync(0xffffffffu, v.y, o);
            if (lane >= o) {
                v.x += px;
                v.y += py;
            }
        }
        __syncthreads();
        if (lane == 31) s.warp_scan[warp] = v;
        __syncthreads();
        if (t == 0) {
            longlong2 run = make_longlong2(0, 0);
            for (int k = 0; k < kPlanThreads / 32; ++k) {
                const longlong2 x = s.warp_scan[k];
                s.warp_scan[k] = run;
                run.x += x.x;
                run.y += x.y;
            }
            s.all = run;
        }
        __syncthreads();
        fits = n_root + s.all.x <= a.cap_desc && s.all.x <= a.cap_splits && s.all.y <= a.cap_rows;
    }
    const int desc = (int)(n_root + s.warp_scan[warp].x + v.x - parts);
    int row = (int)(s.warp_scan[warp].y + v.y - rows);  // used only when the plan fits
    for (int pass = 0; pass < 2; ++pass) {
        // pass 0: descriptors, records and the histogram; pass 1: the queue
        int dsc = desc;
        for (int k = b; k < e; ++k) {
            const WalkDesc d0 = a.roots[k];
            const WalkCost c = walk_cost(a, k, d0);
            const int np = fits ? walk_parts(d0, c, target) : 1;
            if (np == 1) {
                const int q = plan_bucket(c.cost);
                if (pass == 0) {
                    a.walks[k] = d0;
                    atomicAdd(&s.hist[q], 1);
                } else {
                    a.order[atomicAdd(&s.start[q], 1)] = k;
                }
                continue;
            }
            for (int j = 0; j < np; ++j) {
                const int e0 = part_begin(d0.n_epj, j, np, kPartAlign), e1 = part_begin(d0.n_epj, j + 1, np, kPartAlign);
                const int n0 = part_begin(c.n_spj, j, np, kPartAlign), n1 = part_begin(c.n_spj, j + 1, np, kPartAlign);
                const int q = plan_bucket((unsigned long long)d0.n_i * ((unsigned long long)(e1 - e0) + 2ull * (n1 - n0)));
                const int w = j == 0 ? k : dsc + j - 1;
                if (pass == 0) {
                    const int s0 = part_begin(d0.n_spj, j, np, kPartAlign), s1 = part_begin(d0.n_spj, j + 1, np, kPartAlign);
                    WalkDesc d = d0;
                    d.epj_begin = d0.epj_begin + e0;
                    d.n_epj = e1 - e0;
                    d.spj_begin = d0.spj_begin + s0;
                    d.n_spj = s1 - s0;
                    d.part = (uint16_t)j;
                    d.n_parts = (uint16_t)np;
                    if (j + a.part0_rows > 0) d.i_begin = a.row0 + row + (j + a.part0_rows - 1) * d0.n_i;
                    a.walks[w] = d;
                    atomicAdd(&s.hist[q], 1);
                } else {
                    a.order[atomicAdd(&s.start[q], 1)] = w;
                }
            }
            if (pass == 0) {
                const int r = atomicAdd(a.n_split, 1);
                a.splits[r] = SplitRec{d0.i_begin, a.row0 + row, d0.n_i, np};
                row += (np - 1 + a.part0_rows) * d0.n_i;
            }
            dsc += np - 1;
        }
        __syncthreads();
        if (pass == 0 && t == 0) {
            int run = 0;
            for (int q = kPlanBuckets - 1; q >= 0; --q) {
                s.start[q] = run;
                run += s.hist[q];
            }
            *a.n_desc = run;
        }
        __syncthreads();
    }
}

// Adds up the parts of every split walk of a device plan: as
// combine_parts_kernel, the number of records read on the device.
__global__ __launch_bounds__(128) void combine_plan_kernel(const SplitRec* __restrict__ recs, const int32_t* n_split,
                                                           Accp* accp, int32_t* nnb, const Accp* part_accp,
                                                           const int32_t* part_nnb, int part0_rows, double G) {
    const int n = *n_split;
    if (n == 0) return;
    // few walks: several CTAs each (3,000 stars: 22 -> 10 us)
    const int m = max(1, (int)gridDim.x / n);
    for (int q = blockIdx.x; q < n * m; q += gridDim.x) {
        const SplitRec r = recs[q / m];
        for (int i = (q % m) * blockDim.x + threadIdx.x; i < r.n_i; i += m * blockDim.x) {
            const int64_t r0 = (int64_t)r.row0 + i;
            float2 a[4];
            load_pairs(part0_rows ? part_accp + r.rows1 + i : accp + r0, a);
            int c = part0_rows ? part_nnb[r.rows1 + i] : nnb[r0];
#pragma unroll 8
            for (int k = 1; k < r.n_parts; ++k) {
                const int64_t row = (int64_t)r.rows1 + (int64_t)(k - 1 + part0_rows) * r.n_i + i;
                float2 b[4];
                load_pairs(part_accp + row, b);
#pragma unroll
                for (int u = 0; u < 4; ++u) a[u] = add_pair(a[u], b[u]);
                c += part_nnb[row];
            }
            accp[r0] = Accp{G * pair_value(a[0]), G * pair_value(a[1]), G * pair_value(a[2]), G * pair_value(a[3])};
            nnb[r0] = c;
        }
    }
}

}  // namespace

cudaError_t launch_plan(const PlanArgs& a, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(a.n_split, 0, sizeof(int32_t), s);
    if (e != cudaSuccess) return e;
    plan_kernel<<<1, kPlanThreads, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_combine_plan(const PlanArgs& a, const Params& p, cudaStream_t s) {
    combine_plan_kernel<<<a.num_sms * 4, 128, 0, s>>>(a.splits, a.n_split, p.out_accp, p.out_nnb,
                                                      p.part_accp ? p.part_accp : p.out_accp,
                                                      p.part_nnb ? p.part_nnb : p.out_nnb, a.part0_rows, p.G);
    return cudaGetLastError();
}

}  // namespace pgf
