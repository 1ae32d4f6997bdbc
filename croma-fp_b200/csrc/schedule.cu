// schedule.cu -- per-snapshot sub-step schedule on the device.
//
// Compiled with --fmad=false: the sub-step count is an integer decision
// (ceil of a quotient, a quantisation ladder) taken on floating-point loss
// rates, and the reference takes it with separately rounded multiplies and
// adds.  Keeping the same rounding sequence here makes nsub / n_on
// reproduce the reference's integers.
//
//   endpoint losses   tracer_fp_prepare_nsub_loss_endpoints, src/tracer_fp_nsub.c:242-282
//   nsub / n_on       compute_nsubsteps_core, src/tracer_fp_nsub.c:94-187
//   ladder            quantize_dt_sub / quantize_on_fraction, src/tracer_fp_nsub.c:37-92
//   segments          tracer_fp_choose_coeff_interp_segments, src/tracer_fp_setup.c:73-95
//   buckets           tracer_bucket_build_snapshot, src/tracer_fp_bucket.c:208-262
#include <cub/cub.cuh>

#include "croma_ctx.cuh"

namespace croma {

namespace {

__device__ double quantize_dt_sub(double t)
{
    const double ladder[10] = {1.0, 1.25, 1.6, 2.0, 2.5, 3.2, 4.0, 5.0, 6.4, 8.0};
    if (!(t > 0.0) || !isfinite(t)) return t;
    const double e10 = floor(log10(t));
    const double scale = pow(10.0, e10);
    const double norm = t / scale;
    double chosen = ladder[0];
    for (int i = 0; i < 10; i++) {
        if (ladder[i] <= norm) chosen = ladder[i];
        else break;
    }
    return chosen * scale;
}

__device__ double quantize_on_fraction(double f)
{
    const double bins[5] = {1.0 / 8.0, 1.0 / 4.0, 1.0 / 3.0, 1.0 / 2.0, 1.0};
    if (!(f > 0.0) || !isfinite(f)) return 1.0;
    if (f >= 1.0) return 1.0;
    double chosen = bins[0], best = fabs(f - chosen);
    for (int i = 1; i < 5; i++) {
        const double d = fabs(f - bins[i]);
        if (d < best) { chosen = bins[i]; best = d; }
    }
    return chosen;
}

__device__ int coeff_segments(const ModelParams &mp, int nsub, int allow)
{
    int seg = 1;
    int max_seg = mp.interp_max_segments;
    if (!allow || nsub <= 1) return 1;
    if (mp.interp_min_steps <= 0) return 1;
    if (max_seg < 1) max_seg = 1;
    const int max_allowed = nsub / mp.interp_min_steps;
    if (max_allowed < 1) return 1;
    while (seg <= 1073741823 && seg * 2 <= max_seg && seg * 2 <= max_allowed) seg *= 2;
    if (seg > nsub) seg = nsub;
    if (seg < 1) seg = 1;
    return seg;
}

__global__ void nsub_kernel(ModelParams mp, int ntracer, const double *bg, const double *ic_row,
                            double p_lo, double p_hi, double pe_lo, double pe_hi,
                            double dt_snap, int allow, Schedule s)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntracer) return;
    const double ng = bg[0 * (size_t)ntracer + t];
    const double kbt = bg[1 * (size_t)ntracer + t];
    const double bf = bg[2 * (size_t)ntracer + t];
    const double dvv = bg[3 * (size_t)ntracer + t];
    const double lt = bg[4 * (size_t)ntracer + t];
    const double dv = bg[5 * (size_t)ntracer + t];

    const double rp_lo = coulomb_p_from_p(ng, p_lo, kbt) + 1.0 / 3.0 * dvv * p_lo;
    const double rp_hi = coulomb_p_from_p(ng, p_hi, kbt) + 1.0 / 3.0 * dvv * p_hi;
    const double re_lo = b_synch(pe_lo, bf) + ic_row[0] + b_coulomb_e(ng, pe_lo) + 1.0 / 3.0 * dvv * pe_lo;
    const double re_hi = b_synch(pe_hi, bf) + ic_row[NB - 1] + b_coulomb_e(ng, pe_hi) + 1.0 / 3.0 * dvv * pe_hi;

    const double te0 = pe_lo / re_lo;
    const double tp0 = p_lo / rp_lo;
    const double teN = pe_hi / re_hi;
    const double tpN = p_hi / rp_hi;
    const double tmin = fmin(fabs(tp0), fmin(fabs(teN), fmin(fabs(te0), fabs(tpN))));

    double target = dt_snap / 10.0;
    if (isfinite(tmin) && tmin > 0.0) {
        const double stab = mp.nsub_safety * tmin;
        if (stab < target) target = stab;
    }
    if (target <= 0.0 || !isfinite(target)) target = dt_snap / 10.0;
    double tn = ceil(dt_snap / target);
    if (!isfinite(tn) || tn > 1000000.0) tn = 1000000.0;
    if (tn < 10.0) tn = 10.0;
    double used = quantize_dt_sub(target);
    if (!(used > 0.0) || !isfinite(used) || used > target) used = target;
    double raw = ceil(dt_snap / used);
    if (!isfinite(raw) || raw > 1000000.0) raw = 1000000.0;
    if (raw < 10.0) raw = 10.0;
    int nsub = (int)raw;
    unsigned char capped = 0;
    if (mp.nsub_max > 0 && nsub > mp.nsub_max) {
        nsub = mp.nsub_max;
        capped = 1;
    }
    double onf = 1.0;
    if (mp.window_centred && mp.f_eddy > 0.0 && dv > 0.0) {
        const double t_eddy = lt * 3.0857e24 / dv / 3.1536e16;
        if (mp.f_eddy * t_eddy < dt_snap) onf = quantize_on_fraction(mp.f_eddy * t_eddy / dt_snap);
    }
    int non = (int)floor((double)nsub * onf + 0.5);
    if (non < 1) non = 1;
    if (non > nsub) non = nsub;

    s.nsub[t] = nsub;
    s.non[t] = non;
    s.target[t] = (int)tn;
    s.capped[t] = capped;
    s.nseg[t] = coeff_segments(mp, nsub, allow);
}

// ---- bucket build: first-appearance order of the (nsub, n_on) key ----
__global__ void make_keys_kernel(int n, const int *nsub, const int *non, unsigned long long *keys,
                                 int *vals)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    // both at most 1e6: 20 bits each
    keys[t] = ((unsigned long long)(unsigned)nsub[t] << 20) | (unsigned)non[t];
    vals[t] = t;
}

// After a stable sort by key: head flags -> segment index per element.
__global__ void seg_heads_kernel(int n, const unsigned long long *keys, int *head)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    head[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

// seg_of[i] = inclusive-scan(head)[i] - 1.  For segment heads, record
// (first tracer, segment) pairs keyed by the first tracer index.
__global__ void seg_first_kernel(int n, const int *seg_incl, const int *sorted_t,
                                 unsigned long long *first_keys, int *first_seg)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int seg = seg_incl[i] - 1;
    if (i == 0 || seg_incl[i] != seg_incl[i - 1]) {
        first_keys[seg] = (unsigned long long)sorted_t[i];
        first_seg[seg] = seg;
    }
}

// bucket_of_seg[seg] = rank of the segment's first tracer (ranks beyond
// the segment count belong to the all-ones padding and are skipped).
__global__ void seg_rank_kernel(int n, const int *nseg_dev, const int *seg_by_first,
                                int *bucket_of_seg)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n || r >= *nseg_dev) return;
    bucket_of_seg[seg_by_first[r]] = r;
}

__global__ void assign_bucket_kernel(int n, const int *seg_incl, const int *sorted_t,
                                     const int *bucket_of_seg, int *bucket_ids)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = bucket_of_seg[seg_incl[i] - 1];
    bucket_ids[sorted_t[i]] = b;
}

// The same for a run of at most kBucketOneBlock tracers, by one block: the
// distinct keys in a hash table in shared memory (one insertion per key and
// warp), each with its first tracer; a bucket's number is the count of first
// tracers before its own; the members are placed in tracer order by one warp.
// Three radix sorts and their dozen small kernels took 30 us of GPU time and
// some 25 launches at 64 tracers, 33 us at 999; this takes 3.7 and 7.3 us and
// one.  The line: 4,096 tracers take one block 32 us (43 us with uneven counts),
// 4,097 take the sorts 145 (138).  The block's table would fit for 8,192, where it
// is still ahead of the sorts, 58 us (74) against 145 (143), a snapshot alone 641 us
// against 770, but the snapshot's own kernels cover less of it: uneven snapshots
// in a row, of which the build is the longest chain, 362 us against 351.  Above that
// the table outgrows a block's shared memory.
constexpr int kBucketOneBlock = 4096;
constexpr int kBucketThreads = 1024;

__host__ __device__ constexpr int bucket_table(int n)   // a power of two, at least 2 n
{
    int h = 64;
    while (h < 2 * n) h <<= 1;
    return h;
}

constexpr size_t bucket_smem(int n)   // keys and first tracers of the table, slots of the tracers
{
    return (size_t)bucket_table(n) * (sizeof(unsigned long long) + sizeof(int)) + (size_t)n * sizeof(int);
}

static_assert(bucket_smem(kBucketOneBlock) + 256 <= 227 * 1024, "a block's shared memory");

// exclusive prefix sum of v over the block, and its total
__device__ __forceinline__ int block_prefix(int v, int *warp_sums, int &total)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int s = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, s, off);
        if (lane >= off) s += o;
    }
    if (lane == 31) warp_sums[w] = s;
    __syncthreads();
    if (w == 0) {
        const int ws = warp_sums[lane];
        int x = ws;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += o;
        }
        warp_sums[lane] = x - ws;
        if (lane == 31) warp_sums[32] = x;
    }
    __syncthreads();
    const int before = warp_sums[w] + s - v;
    total = warp_sums[32];
    __syncthreads();
    return before;
}

__global__ void __launch_bounds__(kBucketThreads) bucket_small_kernel(int n, const int *nsub, const int *non,
                                                                      int *bucket_ids, int *bucket_indices, int *nbuckets)
{
    extern __shared__ unsigned long long bk_smem[];
    __shared__ int warp_sums[33];
    constexpr unsigned long long kEmpty = ~0ull;
    const int H = bucket_table(n), lane = threadIdx.x & 31;
    unsigned long long *keys = bk_smem;                  // [H]
    int *first = reinterpret_cast<int *>(keys + H);      // [H] first tracer of the slot's key
    int *slot = first + H;                               // [n] slot of each tracer
    int *id = reinterpret_cast<int *>(keys);             // [H] bucket of each slot, once the keys are done
    int *start = id + H;                                 // [n] next place of each bucket (2 H ints in keys, H >= 2 n)
    const int top = (n + 31) & ~31;
    for (int h = threadIdx.x; h < H; h += blockDim.x) {
        keys[h] = kEmpty;
        first[h] = 0x7fffffff;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < top; t += blockDim.x) {
        const bool on = t < n;
        const unsigned long long key = on ? ((unsigned long long)(unsigned)nsub[t] << 32) | (unsigned)non[t] : kEmpty;
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        const int leader = __ffs(peers) - 1;
        int h = 0;
        if (on && lane == leader) {
            h = (int)((key * 0x9e3779b97f4a7c15ull) >> 40) & (H - 1);
            for (int probe = 0; probe < H; probe++, h = (h + 1) & (H - 1)) {   // a free slot is always met
                unsigned long long at = *(volatile unsigned long long *)(keys + h);
                if (at == kEmpty) at = atomicCAS(keys + h, kEmpty, key);
                if (at == kEmpty || at == key) break;
            }
            atomicMin(first + h, t);   // the lowest lane of the warp's equals
        }
        h = __shfl_sync(0xffffffffu, h, leader);
        if (on) slot[t] = h;
    }
    __syncthreads();
    // bucket numbers in the order of the first tracers
    int total = 0;
    for (int t0 = 0; t0 < n; t0 += blockDim.x) {
        const int t = t0 + threadIdx.x;
        const bool lead = t < n && first[slot[t]] == t;
        int here;
        const int before = block_prefix(lead ? 1 : 0, warp_sums, here);
        if (lead) id[slot[t]] = total + before;
        total += here;
    }
    if (threadIdx.x == 0) *nbuckets = total;
    for (int b = threadIdx.x; b < n; b += blockDim.x) start[b] = 0;
    __syncthreads();
    for (int t = threadIdx.x; t < top; t += blockDim.x) {
        const bool on = t < n;
        const int b = on ? id[slot[t]] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, b);
        if (on) {
            bucket_ids[t] = b;
            slot[t] = b;
            if (lane == __ffs(peers) - 1) atomicAdd(start + b, __popc(peers));
        }
    }
    __syncthreads();
    int base = 0;
    for (int b0 = 0; b0 < total; b0 += blockDim.x) {
        const int b = b0 + threadIdx.x, c = b < total ? start[b] : 0;
        int here;
        const int before = block_prefix(c, warp_sums, here);
        if (b < total) start[b] = base + before;
        base += here;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        for (int t = lane; t < top; t += 32) {
            const bool on = t < n;
            const int b = on ? slot[t] : -1;
            const unsigned peers = __match_any_sync(0xffffffffu, b);
            const int at = on ? start[b] : 0;
            __syncwarp();
            if (on) {
                bucket_indices[at + __popc(peers & ((1u << lane) - 1u))] = t;
                if (lane == __ffs(peers) - 1) start[b] = at + __popc(peers);
            }
            __syncwarp();
        }
    }
}

// Members listed bucket by bucket in ascending tracer order: a stable
// pass over tracers in index order within each bucket is a stable sort
// of (bucket, tracer) by bucket, which the radix sort below provides.
__global__ void bucket_keys_kernel(int n, const int *bucket_ids, unsigned long long *keys, int *vals)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    keys[t] = (unsigned long long)(unsigned)bucket_ids[t];
    vals[t] = t;
}

}  // namespace

int schedule_reserve(Context &ctx, int cap)
{
    // ints: nsub, non, target, nseg, bucket_ids, bucket_indices, nbuckets(+pad), and aux
    if (ctx.d_sched_int) {
        dev_free(ctx, ctx.d_sched_int);
        dev_free(ctx, ctx.d_capped);
        dev_free(ctx, ctx.d_cub_tmp);
        dev_free(ctx, ctx.d_keys);
        dev_free(ctx, ctx.d_vals);
        ctx.d_sched_int = nullptr;
    }
    const size_t n = (size_t)cap;
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_sched_int, (n * 6 + 32) * sizeof(int)));
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_capped, n));
    int *p = ctx.d_sched_int;
    ctx.sched.nsub = p;
    ctx.sched.non = p + n;
    ctx.sched.target = p + 2 * n;
    ctx.sched.nseg = p + 3 * n;
    ctx.sched.bucket_ids = p + 4 * n;
    ctx.sched.bucket_indices = p + 5 * n;
    ctx.sched.nbuckets = p + 6 * n;
    ctx.sched.capped = ctx.d_capped;
    // keys/vals double buffers + aux (head/scan, first segments, bucket_of_seg, segments by first tracer)
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_keys, n * 3 * sizeof(unsigned long long)));
    ctx.d_keys_alt = ctx.d_keys + n;
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_vals, n * 6 * sizeof(int)));
    ctx.d_vals_alt = ctx.d_vals + n;
    ctx.d_seg_aux = ctx.d_vals + 2 * n;
    size_t b1 = 0, b2 = 0;
    cub::DoubleBuffer<unsigned long long> kb(ctx.d_keys, ctx.d_keys_alt);
    cub::DoubleBuffer<int> vb(ctx.d_vals, ctx.d_vals_alt);
    CROMA_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b1, kb, vb, cap, 0, 64, ctx.stream));
    CROMA_CUDA(cub::DeviceScan::InclusiveSum(nullptr, b2, ctx.d_seg_aux, ctx.d_seg_aux, cap, ctx.stream));
    ctx.cub_tmp_bytes = (b1 > b2 ? b1 : b2) + 256;
    CROMA_CUDA(dev_alloc(ctx, &ctx.d_cub_tmp, ctx.cub_tmp_bytes));
    // above the default 48 KB for runs of more than 1,024 tracers; per device, so here
    CROMA_CUDA(cudaFuncSetAttribute(bucket_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)bucket_smem(kBucketOneBlock)));
    if (!ctx.side_stream) {   // of the context stream's priority: the snapshot ends with it
        int priority = 0;
        CROMA_CUDA(cudaStreamGetPriority(ctx.stream, &priority));
        CROMA_CUDA(cudaStreamCreateWithPriority(&ctx.side_stream, cudaStreamNonBlocking, priority));
    }
    if (!ctx.side_begin) CROMA_CUDA(cudaEventCreateWithFlags(&ctx.side_begin, cudaEventDisableTiming));
    if (!ctx.side_end) CROMA_CUDA(cudaEventCreateWithFlags(&ctx.side_end, cudaEventDisableTiming));
    return 0;
}

// Buckets are for the caller (get_schedule); nothing of the snapshot reads
// them.  So they are built on a stream of their own from the sub-step counts
// on, beside the snapshot's kernels, which wait on FP64 latency most of the
// time.  A snapshot of 64 tracers: 118 to 98 us; GPU time of one of 999 629 to
// 579 us, of 30,011 814 to 741 us, the bucket kernels overlapping the rest.
static int run_buckets(Context &ctx, const SnapArgs &a, cudaStream_t st)
{
    const int n = a.ntracer;
    if (n <= kBucketOneBlock) {
        bucket_small_kernel<<<1, kBucketThreads, bucket_smem(n), st>>>(n, a.sched.nsub, a.sched.non, a.sched.bucket_ids,
                                                             a.sched.bucket_indices, a.sched.nbuckets);
        CROMA_CUDA(cudaGetLastError());
        ctx.last_launches += 1;
        return 0;
    }
    const int blk = 256, grd = (n + blk - 1) / blk;
    int bits = 1;   // all ones in them is no tracer's index
    while ((1LL << bits) - 1 < n) bits++;
    const size_t N = (size_t)n;
    int *head = ctx.d_seg_aux;              // [n] head flags, scanned in place
    int *first_seg = ctx.d_seg_aux + N;     // [n]
    int *bucket_of_seg = ctx.d_seg_aux + 2 * N;
    int *seg_by_first = ctx.d_seg_aux + 3 * N;
    unsigned long long *first_keys = ctx.d_keys + 2 * N;
    size_t tmp = ctx.cub_tmp_bytes;

    make_keys_kernel<<<grd, blk, 0, st>>>(n, a.sched.nsub, a.sched.non, ctx.d_keys, ctx.d_vals);
    cub::DoubleBuffer<unsigned long long> kb(ctx.d_keys, ctx.d_keys_alt);
    cub::DoubleBuffer<int> vb(ctx.d_vals, ctx.d_vals_alt);
    CROMA_CUDA(cub::DeviceRadixSort::SortPairs(ctx.d_cub_tmp, tmp, kb, vb, n, 0, 40, st));
    const unsigned long long *skeys = kb.Current();
    const int *sorted_t = vb.Current();
    seg_heads_kernel<<<grd, blk, 0, st>>>(n, skeys, head);
    tmp = ctx.cub_tmp_bytes;
    CROMA_CUDA(cub::DeviceScan::InclusiveSum(ctx.d_cub_tmp, tmp, head, head, n, st));
    // sorted_t lives in one of the two value buffers; keep it intact while the
    // segment-first pairs are sorted through the other key buffer and aux ints.
    // (first tracer, segment) pairs; unused tail entries carry all-ones keys
    // so that they sort last.
    CROMA_CUDA(cudaMemsetAsync(first_keys, 0xFF, N * sizeof(unsigned long long), st));
    seg_first_kernel<<<grd, blk, 0, st>>>(n, head, sorted_t, first_keys, first_seg);
    {
        unsigned long long *fk_alt = (kb.Current() == ctx.d_keys) ? ctx.d_keys_alt : ctx.d_keys;
        cub::DoubleBuffer<unsigned long long> fkb(first_keys, fk_alt);
        cub::DoubleBuffer<int> fvb(first_seg, seg_by_first);
        tmp = ctx.cub_tmp_bytes;
        CROMA_CUDA(cub::DeviceRadixSort::SortPairs(ctx.d_cub_tmp, tmp, fkb, fvb, n, 0, bits, st));
        seg_rank_kernel<<<grd, blk, 0, st>>>(n, head + (n - 1), fvb.Current(), bucket_of_seg);
        assign_bucket_kernel<<<grd, blk, 0, st>>>(n, head, sorted_t, bucket_of_seg, a.sched.bucket_ids);
        CROMA_CUDA(cudaMemcpyAsync(a.sched.nbuckets, head + (n - 1), sizeof(int),
                                   cudaMemcpyDeviceToDevice, st));
    }
    CROMA_CUDA(cudaGetLastError());
    ctx.last_launches += 6;

    // member lists: stable sort of (bucket id, tracer) by bucket id
    {
        unsigned long long *k0 = ctx.d_keys, *k1 = ctx.d_keys_alt;
        int *v0 = ctx.d_vals, *v1 = ctx.d_vals_alt;
        bucket_keys_kernel<<<grd, blk, 0, st>>>(n, a.sched.bucket_ids, k0, v0);
        cub::DoubleBuffer<unsigned long long> bkb(k0, k1);
        cub::DoubleBuffer<int> bvb(v0, v1);
        tmp = ctx.cub_tmp_bytes;
        CROMA_CUDA(cub::DeviceRadixSort::SortPairs(ctx.d_cub_tmp, tmp, bkb, bvb, n, 0, bits, st));
        CROMA_CUDA(cudaMemcpyAsync(a.sched.bucket_indices, bvb.Current(), N * sizeof(int),
                                   cudaMemcpyDeviceToDevice, st));
    }
    CROMA_CUDA(cudaGetLastError());
    ctx.last_launches += 6;
    return 0;
}

int run_schedule(Context &ctx, const SnapArgs &a)
{
    const int n = a.ntracer;
    nsub_kernel<<<(n + 255) / 256, 256, 0, ctx.stream>>>(ctx.mp, n, a.bg_curr, a.ic_curr, ctx.h_p[0][0],
                                                         ctx.h_p[0][NB - 1], ctx.h_p[1][0], ctx.h_p[1][NB - 1],
                                                         a.dt_snap, a.allow_interp, a.sched);
    CROMA_CUDA(cudaGetLastError());
    ctx.last_launches += 1;
    CROMA_CUDA(cudaEventRecord(ctx.side_begin, ctx.stream));
    CROMA_CUDA(cudaStreamWaitEvent(ctx.side_stream, ctx.side_begin, 0));
    const int rc = run_buckets(ctx, a, ctx.side_stream);
    CROMA_CUDA(cudaEventRecord(ctx.side_end, ctx.side_stream));
    ctx.side_open = 1;
    return rc;
}

int join_schedule(Context &ctx)
{
    if (!ctx.side_open) return 0;
    ctx.side_open = 0;
    CROMA_CUDA(cudaStreamWaitEvent(ctx.stream, ctx.side_end, 0));
    return 0;
}

}  // namespace croma
