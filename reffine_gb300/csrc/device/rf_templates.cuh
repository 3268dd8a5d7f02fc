// Kernel templates of the GB300 backend.  Included by a generated query source AFTER the
// query's fragment (the templates use the fragment's types and functions), once per source.
#pragma once

// loads a lane issues ahead of its combines in the last unit's fold over all units' partials
#ifndef RF_FOLD
#define RF_FOLD 16
#endif
#ifndef RF_FOLD_ACC
#define RF_FOLD_ACC 4
#endif

// Batched form: one persistent launch runs the work units of many queries of this shape.  work
// names the shape's queries and where their units begin: work[0] = {units, queries}, work[1] =
// {units taken beyond each block's first, 0}, then per query {index of its parameter block, its
// first unit}, in unit order; a block finds the query of its next unit by bisection.  (A list of
// every unit, 15 000 of them for 64 queries, took the host and its copy longer than the kernels.)  A
// query's units are the ones its stand-alone launch would run, folded in the same order: same bits
// either way.
// Blocks take units as they come free: the kernels of a batch's shapes share the SMs, and with every
// gridDim.x-th unit the blocks that started last, or had the costlier queries, finished alone.  (64
// queries of three shapes, from the launch to its end: 426 -> 381 us with tables of 1M rows, 96 -> 98
// of 150K.  Runs of consecutive units, an eighth, a quarter or half of a block's share, took 388, 387
// and 402 us, and 2264, 2354 and 2675 us with tables of 8M rows against 2217 unit by unit.)  The next
// unit is asked for before the one at hand is run, which hides the atomic's way.
RF_DEV int2 rf_batch_unit(const int2* work, int w)
{
    int lo = 0, hi = work[0].y;  // the last query whose first unit is not after w
    while (hi - lo > 1) {
        const int m = (lo + hi) >> 1;
        if (__ldg(&work[2 + m].y) <= w) lo = m;
        else hi = m;
    }
    const int2 q = __ldg(work + 2 + lo);
    return make_int2(q.x, w - q.y);
}

// F(parameters, unit) for every unit that this block gets
template <class F>
RF_DEV void rf_batch_units(const RfParams* params, int2* work, F f)
{
    __shared__ unsigned taken;
    const unsigned n = (unsigned)work[0].x;
#pragma unroll 1
    for (unsigned w = blockIdx.x; w < n;) {
        unsigned next = 0;
        if (threadIdx.x == 0) next = atomicAdd((unsigned*)&work[1].x, 1u);
        const int2 it = rf_batch_unit(work, (int)w);
        const RfParams& P = params[it.x];
        if (it.y < 0 || it.y >= P.nunits) {  // a malformed work item: report, skip
            if (threadIdx.x == 0) atomicExch(P.err, RF_DEVERR_RANGE);
        } else {
            f(P, it.y);
        }
        if (threadIdx.x == 0) taken = next;
        __syncthreads();
        w = gridDim.x + taken;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------------------
// Template 1: fused scan-filter-project-reduce.
//   The fragment defines: struct RfAcc (8-byte aligned fields, size a multiple of 8),
//   rf_acc_init(P, A), rf_acc_combine(A, B) (A <- A op B), rf_acc_shfl(A, off),
//   rf_row(P, r, A) (one row) and rf_finish(P, A, out).
// Work is split into fixed tiles of P.tile_rows rows; unit u takes the contiguous tiles
// [u*ntiles/nunits, (u+1)*ntiles/nunits).  Each unit's accumulator goes to P.partials[u]; the
// last unit to finish folds the partials in a fixed order.  So the result depends only on (rows,
// tile_rows, nunits, threads), not on scheduling: a query gives the same bits alone, batched with
// others, or launched a range of units at a time as its rows arrive (P.unit0).
// ---------------------------------------------------------------------------------------
#ifdef RF_SCAN_REDUCE
template <int T>
RF_DEV void rf_scan_reduce_rows(const RfParams& P, int unit, int nunits, RfAcc& acc)
{
    long long lo = P.row_lo, hi = P.row_hi;
    if (P.range) {
        long long b = P.range[0], e = P.range[1];
        lo = b > lo ? b : lo;
        hi = e < hi ? e : hi;
    }
    const long long tr = P.tile_rows;
    const long long ntiles = (P.row_hi - P.row_lo + tr - 1) / tr;
    const long long t_end = (long long)(unit + 1) * ntiles / nunits;
    for (long long tile = (long long)unit * ntiles / nunits; tile < t_end; tile++) {
        long long r0 = P.row_lo + tile * tr, r1 = r0 + tr;
        if (r1 > hi) r1 = hi;
        if (r0 < lo) r0 = lo;
#ifdef RF_VEC4
        if ((P.flags & RF_FLAG_VEC4) && r0 >= 0) {
            // a thread takes 4 consecutive rows per step (one 16-byte load per column), in row
            // order; the rows before the first multiple of 4 and after the last go one by one
            long long a = (r0 + 3) & ~3LL;
            if (a > r1) a = r1;
            const long long b = a + ((r1 - a) & ~3LL);
            for (long long r = r0 + threadIdx.x; r < a; r += T) rf_row(P, r, acc);
#pragma unroll 2
            for (long long r = a + 4 * (long long)threadIdx.x; r < b; r += 4LL * T) rf_row4(P, r, acc);
            for (long long r = b + threadIdx.x; r < r1; r += T) rf_row(P, r, acc);
            continue;
        }
#endif
#pragma unroll 4
        for (long long r = r0 + threadIdx.x; r < r1; r += T) rf_row(P, r, acc);
    }
}

template <int T>
RF_DEV void rf_scan_reduce_merge(const RfParams& P, int unit, int nunits, RfAcc& acc)
{
    __shared__ RfAcc warp_acc[T / 32];
    __shared__ int last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        RfAcc o = rf_acc_shfl(acc, off);
        rf_acc_combine(acc, o);
    }
    if (lane == 0) warp_acc[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        RfAcc tot = warp_acc[0];
        for (int w = 1; w < T / 32; w++) rf_acc_combine(tot, warp_acc[w]);
        rf_st_words((RfAcc*)P.partials + unit, &tot, (int)sizeof(RfAcc));
        __threadfence();
        unsigned int ticket = atomicAdd(P.counter, 1u);
        last = (ticket == (unsigned int)nunits - 1u);
    }
    __syncthreads();
    if (last) {
        __threadfence();
        // the whole block folds the units' partials: thread t takes units t, t+T, t+2T, ... in
        // that order (their loads issued RF_FOLD_ACC at a time ahead of the combines), then the
        // lanes of each warp by shuffles and the warps in order - a fixed order on every path
        RfAcc tot;
        rf_acc_init(P, tot);
        int u = threadIdx.x;
        for (; u + T * (RF_FOLD_ACC - 1) < nunits; u += T * RF_FOLD_ACC) {
            RfAcc v[RF_FOLD_ACC];
#pragma unroll
            for (int k = 0; k < RF_FOLD_ACC; k++)
                rf_ld_words(&v[k], (const RfAcc*)P.partials + u + T * k, (int)sizeof(RfAcc));
#pragma unroll
            for (int k = 0; k < RF_FOLD_ACC; k++) rf_acc_combine(tot, v[k]);
        }
        for (; u < nunits; u += T) {
            RfAcc p;
            rf_ld_words(&p, (const RfAcc*)P.partials + u, (int)sizeof(RfAcc));
            rf_acc_combine(tot, p);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            RfAcc o = rf_acc_shfl(tot, off);
            rf_acc_combine(tot, o);
        }
        if (lane == 0) warp_acc[warp] = tot;
        __syncthreads();
        if (threadIdx.x == 0) {
            RfAcc all = warp_acc[0];
            for (int w = 1; w < T / 32; w++) rf_acc_combine(all, warp_acc[w]);
            rf_finish(P, all, P.out);
            *P.counter = 0u;
        }
    }
    __syncthreads();  // shared state is reused by the next work item of a persistent block
}

// (rf_batch: the registers for 768 threads an SM, 80 each; left alone the compiler takes 118)
#define RF_SCAN_REDUCE_KERNEL(NAME, T)                                                      \
    extern "C" __global__ void __launch_bounds__(T) NAME(const __grid_constant__ RfParams P) \
    {                                                                                       \
        RfAcc acc;                                                                          \
        rf_acc_init(P, acc);                                                                \
        rf_scan_reduce_rows<T>(P, P.unit0 + (int)blockIdx.x, P.nunits, acc);                \
        rf_scan_reduce_merge<T>(P, P.unit0 + (int)blockIdx.x, P.nunits, acc);               \
    }                                                                                       \
    extern "C" __global__ void __launch_bounds__(T, T > 768 ? 1 : 768 / T)                  \
        rf_batch(const RfParams* __restrict__ params, int2* work)                          \
    {                                                                                       \
        rf_batch_units(params, work, [](const RfParams& Q, int unit) {                     \
            RfAcc acc;                                                                      \
            rf_acc_init(Q, acc);                                                            \
            rf_scan_reduce_rows<T>(Q, unit, Q.nunits, acc);                                 \
            rf_scan_reduce_merge<T>(Q, unit, Q.nunits, acc);                                \
        });                                                                                 \
    }
#endif  // RF_SCAN_REDUCE

// ---------------------------------------------------------------------------------------
// Template 2: grouped scan-reduce with shared-memory privatised accumulators.
//   The fragment defines RF_G groups x RF_M aggregates, struct RfVals, rf_group(P, r, V)
//   (group id or -1, and the row's aggregate inputs), rf_slot_init(m) (64-bit identity),
//   rf_slot_combine(m, a, b), rf_slot_at(q, t) (where thread t keeps slot q: S[q * T + t], or side
//   by side with its neighbour's), rf_slot_add(S, g, t, V, df), rf_slots_done(S, t, df) (df: the
//   thread keeps its FP64 sums as double-floats, see rf_device.cuh; RF_GROUP_DF: it can, and
//   rf_slot_kind(m) - 1: alone, 2: with the next slot, 3: with the one before -, rf_slot_df(S, q, t,
//   kind) {hi, hi of the next, lo, lo of the next} and rf_df_task(i), the RF_DF_TASKS aggregates of
//   kinds 1 and 2, read them) and
//   rf_finish_groups(P, tot, out, part, parts) (the output fields part, part + parts, ...).  With RF_GROUP_SPLIT it also defines the row's loads apart,
//   struct RfRowLd, rf_group_ld(P, r, L) and rf_group_v(P, r, L, V) (rf_group is the two in turn).
// Each thread owns a private column of G*M 64-bit slots in shared memory: no atomics and no bank
// conflicts on the per-row update.  At the end every slot column is folded over the block in a fixed
// order, then over units by the last unit, whose warps compute the output fields between them (a
// field may divide, and one thread doing all 18 quotients of the 6-group group-by in turn took 6 us).
// ---------------------------------------------------------------------------------------
#ifdef RF_GROUP_REDUCE
template <int T>
RF_DEV void rf_group_reduce(const RfParams& P, int unit, int nunits)
{
    extern __shared__ unsigned long long S[];
    __shared__ int last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Q = RF_G * RF_M;
    for (int q = 0; q < Q; q++) S[rf_slot_at(q, tid)] = rf_slot_init(P, q % RF_M);
    bool df = true;  // the thread's FP64 sum slots hold double-floats (rf_slot_add, rf_slots_done)
    long long lo = P.row_lo, hi = P.row_hi;
    if (P.range) {
        long long b = P.range[0], e = P.range[1];
        lo = b > lo ? b : lo;
        hi = e < hi ? e : hi;
    }
    const long long tr = P.tile_rows;
    const long long ntiles = (P.row_hi - P.row_lo + tr - 1) / tr;
#ifdef RF_COMPACT
    // per-warp queue (64 rows) behind the slots: rows passing the cheap prefix of the condition
    long long* q = (long long*)(S + (size_t)Q * T) + (size_t)warp * 64;
#endif
    const long long t_end = (long long)(unit + 1) * ntiles / nunits;
    for (long long tile = (long long)unit * ntiles / nunits; tile < t_end; tile++) {
        long long r0 = P.row_lo + tile * tr, r1 = r0 + tr;
        if (r1 > hi) r1 = hi;
        if (r0 < lo) r0 = lo;
#ifdef RF_PREFETCH
        // the next tile's rows of the row's columns into L2 while this one is read
        if (tid == 0 && tile + 1 < t_end) {
            const long long n0 = P.row_lo + (tile + 1) * tr;
            long long n1 = n0 + tr;
            if (n1 > hi) n1 = hi;
            rf_prefetch_rows(P, n0, n1);
        }
#endif
#ifdef RF_COMPACT
        // warp-uniform steps of 8 chunks of 32 rows: the cheap tests of all 8 are issued together
        constexpr int U = 8;
        int qn = 0;
        for (long long b = r0 + 32 * U * warp; b < r1; b += (long long)T * U) {
            bool c[U];
#pragma unroll
            for (int j = 0; j < U; j++) {
                const long long r = b + 32 * j + lane;
                c[j] = r < r1 && rf_cheap(P, r);
            }
#pragma unroll
            for (int j = 0; j < U; j++) {
                const unsigned m = __ballot_sync(0xffffffffu, c[j]);
                if (c[j]) q[qn + __popc(m & ((1u << lane) - 1u))] = b + 32 * j + lane;
                qn += __popc(m);
                __syncwarp();
                if (qn >= 32) {
                    RfVals V;
                    const int g = rf_group(P, q[lane], V);
                    if (g >= 0) rf_slot_add(S, g, tid, V, df);
                    __syncwarp();
                    if (lane < qn - 32) q[lane] = q[32 + lane];
                    __syncwarp();
                    qn -= 32;
                }
            }
        }
        if (lane < qn) {
            RfVals V;
            const int g = rf_group(P, q[lane], V);
            if (g >= 0) rf_slot_add(S, g, tid, V, df);
        }
        __syncwarp();
#else
#if defined(RF_GROUP_ROWS) && defined(RF_GROUP_SPLIT)
        // RF_GROUP_ROWS rows a thread per iteration: all their loads (rf_group_ld) issued before
        // any row is evaluated (rf_group_v), so a warp has that many rows' loads in flight
#pragma unroll 1
        for (long long r = r0 + tid; r < r1; r += (long long)RF_GROUP_ROWS * T) {
            RfRowLd L[RF_GROUP_ROWS];
#pragma unroll
            for (int k = 0; k < RF_GROUP_ROWS; k++)
                if (r + (long long)k * T < r1) rf_group_ld(P, r + (long long)k * T, L[k]);
#pragma unroll
            for (int k = 0; k < RF_GROUP_ROWS; k++) {
                if (r + (long long)k * T >= r1) break;
                RfVals V;
                const int g = rf_group_v(P, r + (long long)k * T, L[k], V);
                if (g >= 0) rf_slot_add(S, g, tid, V, df);
            }
        }
#else
        // RF_GROUP_UNROLL 1 (a fragment with double-float sums): one row per iteration - the slot
        // update is long, and unrolled rows (whose loads the compiler does not move above the
        // previous row's branches) cost registers the row's own latencies need (the 6-group
        // group-by, its value loads after its filter: 0.775 ms against 0.789 / 0.800 ms unrolled
        // 2 / 4)
#if defined(RF_GROUP_UNROLL) && RF_GROUP_UNROLL == 1
#pragma unroll 1
#else
#pragma unroll 4
#endif
        for (long long r = r0 + tid; r < r1; r += T) {
            RfVals V;
            int g = rf_group(P, r, V);
            if (g >= 0) rf_slot_add(S, g, tid, V, df);
        }
#endif
#endif
    }
#ifdef RF_GROUP_DF
    const bool sums_df = __syncthreads_and(df) != 0;  // every thread's FP64 sums are still double-floats
    if (!sums_df) {
        rf_slots_done(S, tid, df);
        __syncthreads();
    }
#else
    __syncthreads();
#endif
    unsigned long long* part = (unsigned long long*)P.partials;
#ifdef RF_GROUP_DF
    // Double-floats are summed as three floats, two neighbouring slots at once, and turned into doubles
    // last: a conversion and an addition of doubles for each thread's slot hold the FP64 pipe for 16
    // cycles a warp each (34K cycles for the 36 slots of 512 threads).  No bits are lost against sums in
    // doubles, which additions of double-floats would lose; they would be faster by the two additions'
    // errors (the 6-group group-by, those / these: 1M rows 26.7 / 26.8 us, 6M 73.1 / 74.1, 60M 523 / 526).
    if (sums_df)
        for (int i = warp; i < RF_G * RF_DF_TASKS; i += T / 32) {
            const int q = i / RF_DF_TASKS * RF_M + rf_df_task(i % RF_DF_TASKS), kind = rf_slot_kind(q % RF_M);
            constexpr int C = T / 32 < 4 ? T / 32 : 4;
            RfTf2 a[C];
#pragma unroll
            for (int k = 0; k < C; k++) {
                const float4 v = rf_slot_df(S, q, lane + 32 * k, kind);
                a[k] = RfTf2{rf_f2(v.x, v.y), rf_f2(v.z, v.w), 0ULL};
            }
#pragma unroll
            for (int k = C; k < T / 32; k++) {
                const float4 v = rf_slot_df(S, q, lane + 32 * k, kind);
                rf_tf_add2(a[k % C], rf_f2(v.x, v.y), rf_f2(v.z, v.w), 0ULL);
            }
#pragma unroll
            for (int w = C / 2; w > 0; w >>= 1)
#pragma unroll
                for (int k = 0; k < w; k++) rf_tf_add2(a[k], a[k + w].h, a[k + w].m, a[k + w].l);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                rf_tf_add2(a[0], __shfl_down_sync(0xffffffffu, a[0].h, off), __shfl_down_sync(0xffffffffu, a[0].m, off),
                           __shfl_down_sync(0xffffffffu, a[0].l, off));
            if (lane == 0) {
                const ulonglong2 d = rf_tf2_to_f64(a[0]);
                __stcg(part + (long long)unit * Q + q, d.x);
                if (kind == 2) __stcg(part + (long long)unit * Q + q + 1, d.y);
            }
        }
    // the other slots, from the last warp on (the first ones have most of the tasks above)
    for (int q = T / 32 - 1 - warp; q < Q; q += T / 32) {
        const int m = q % RF_M;
        if (sums_df && rf_slot_kind(m)) continue;
#else
    for (int q = warp; q < Q; q += T / 32) {
        const int m = q % RF_M;
#endif
        unsigned long long a = S[rf_slot_at(q, lane)];
        for (int k = 1; k < T / 32; k++) a = rf_slot_combine(m, a, S[rf_slot_at(q, lane + 32 * k)]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) a = rf_slot_combine(m, a, __shfl_down_sync(0xffffffffu, a, off));
        if (lane == 0) __stcg(part + (long long)unit * Q + q, a);
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        unsigned int ticket = atomicAdd(P.counter, 1u);
        last = (ticket == (unsigned int)nunits - 1u);
    }
    __syncthreads();
    if (last) {
        __threadfence();
        for (int q = warp; q < Q; q += T / 32) {
            const int m = q % RF_M;
            // units lane, lane+32, ... folded in that order; their loads are issued RF_FOLD at a
            // time ahead of the combines
            unsigned long long a = rf_slot_init(P, m);
#ifdef RF_GROUP_DF
            // (few units, large blocks: the last loads go out together too)
            for (int u = lane; u - lane < nunits; u += 32 * 8) {
                unsigned long long v[8];
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (u + 32 * k < nunits) v[k] = __ldcg(part + (long long)(u + 32 * k) * Q + q);
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (u + 32 * k < nunits) a = rf_slot_combine(m, a, v[k]);
            }
#else
            int u = lane;
            for (; u + 32 * (RF_FOLD - 1) < nunits; u += 32 * RF_FOLD) {
                unsigned long long v[RF_FOLD];
#pragma unroll
                for (int k = 0; k < RF_FOLD; k++) v[k] = __ldcg(part + (long long)(u + 32 * k) * Q + q);
#pragma unroll
                for (int k = 0; k < RF_FOLD; k++) a = rf_slot_combine(m, a, v[k]);
            }
            for (; u < nunits; u += 32) a = rf_slot_combine(m, a, __ldcg(part + (long long)u * Q + q));
#endif
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) a = rf_slot_combine(m, a, __shfl_down_sync(0xffffffffu, a, off));
            if (lane == 0) S[q] = a;
        }
        __syncthreads();
        // neighbouring fields to different warps, which then differ in what they compute
        rf_finish_groups(P, S, P.out, lane * (T / 32) + warp, T);
        if (tid == 0) *P.counter = 0u;
    }
    __syncthreads();  // shared state is reused by the next work item of a persistent block
}

// RF_MINB (set by the fragment): the blocks per SM the registers must allow; unset, the bound
// names the block size alone (a minimum of 1 block measured slower for the join's probe kernel:
// 1.11 -> 1.39 ms, as the compiler then takes registers freely)
#ifdef RF_MINB
#define RF_GROUP_BOUNDS(T) __launch_bounds__(T, RF_MINB)
#else
#define RF_GROUP_BOUNDS(T) __launch_bounds__(T)
#endif
#define RF_GROUP_REDUCE_KERNEL(NAME, T)                                                     \
    extern "C" __global__ void RF_GROUP_BOUNDS(T) NAME(const __grid_constant__ RfParams P) \
    {                                                                                       \
        rf_group_reduce<T>(P, P.unit0 + (int)blockIdx.x, P.nunits);                         \
    }                                                                                       \
    extern "C" __global__ void RF_GROUP_BOUNDS(T)                                           \
        rf_batch(const RfParams* __restrict__ params, int2* work)                          \
    {                                                                                       \
        rf_batch_units(params, work, [](const RfParams& Q, int unit) {                     \
            rf_group_reduce<T>(Q, unit, Q.nunits);                                          \
        });                                                                                 \
    }
#endif  // RF_GROUP_REDUCE


// ---------------------------------------------------------------------------------------
// Merge co-iteration of sorted key columns (InterSpace and UnionSpace, iter_space.cpp:217-364).
// A row's partner in another vector is the row (first row of the key there) + (the row's rank among
// its own vector's equal keys), as the two-pointer walk pairs duplicates.  Rows are taken in tiles
// of RF_MAT_TILE: rf_merge_bound finds, a warp to a tile, where the other vector's rows of the
// tile's keys begin (they end where the next tile's begin), and rf_merge_walk copies the tile's keys
// and that window into shared memory, where a thread searches once for its first row and walks on
// for the others.  A window larger than the buffer is searched in place.  The keys are so read
// once; the walk's shared-memory latency is covered by the other blocks of the SM.  (5M rows
// against 4M: 3836 us a call with two binary searches of the whole columns a row in each of two
// kernels on one block an SM, 580 us with the GPU full of them, 162 us so.)
// Keys out of order give other partners, never an access outside the columns.
// ---------------------------------------------------------------------------------------
#ifdef RF_MERGE
#define RF_MERGE_CAP 3328  // window keys of 8 bytes held (26 KiB beside the tile's 18 KiB)

template <class K>
RF_DEV K rf_key(const RfCol& c, long long i)
{
    return RfLd<K>::ldg(c.data, i);
}

// (whole warp) the rank of row x of `a` among the equal keys from row `lo` on
template <class K>
RF_DEV long long rf_merge_rank(const RfCol& a, long long lo, long long x, K key)
{
    if (x <= lo || rf_key<K>(a, x - 1) != key) return 0;
    return x - rf_warp_search(lo, x, [&](long long i) { return rf_key<K>(a, i) < key; });
}

// (whole warp) first row of `b` from row `lo` on whose key is not below `key`
template <class K>
RF_DEV long long rf_merge_bound(const RfCol& b, long long lo, K key)
{
    return rf_warp_search(lo, b.len, [&](long long i) { return rf_key<K>(b, i) < key; });
}

template <class K>
struct RfMergeBuf {
    K key[RF_MAT_TILE + RF_MAT_TILE / 8];
    long long win[RF_MERGE_CAP];  // the window's keys, then a value per row of the tile
};

// where the tile's row i is kept: a thread reads the rows after one another, so 8 rows are followed by
// a gap and the threads' rows lie in different banks
RF_DEV int rf_mp(int i) { return i + (i >> 3); }

// the tile's keys (n rows of `a` from row r0 on), for rf_merge_walk; the whole block
template <int T, class K>
RF_DEV void rf_merge_load(RfMergeBuf<K>& B, const RfCol& a, long long r0, int n)
{
    for (int i = threadIdx.x; i < n; i += T) B.key[rf_mp(i)] = rf_key<K>(a, r0 + i);
}

template <bool HELD>
struct RfMergeIndex {
    typedef long long t;
};
template <>
struct RfMergeIndex<true> {
    typedef int t;
};

// rf_merge_walk's rows, with the window held in shared memory (positions in it, and ranks, are ints
// then) or read in place
template <int T, bool HELD, class K, class F>
RF_DEV void rf_merge_rows(const RfMergeBuf<K>& B, long long r0, int n, int beg, long long rank0, const RfCol& b, long long w0,
                          long long wlen, F f)
{
    typedef typename RfMergeIndex<HELD>::t I;
    constexpr int R = RF_MAT_TILE / T;
    const K* win = (const K*)B.win;
    const I wn = (I)wlen;
    auto at = [&](I i) { return HELD ? win[i] : rf_key<K>(b, w0 + i); };
    const int i0 = (int)threadIdx.x * R;
    I p = 0, rank = 0;
    K prev = K(0);
    bool any = false;
#pragma unroll
    for (int j = 0; j < R; j++) {
        const int i = i0 + j;
        if (i < beg || i >= n) continue;
        const K key = B.key[rf_mp(i)];
        if (any && key == prev) {
            rank++;
        } else {
            I lo = p, hi = wn;
            rank = 0;
            if (any) {
                // the next key's rows are close by in most tables: a few steps, then a search
                for (int k = 0; k < 4 && lo < hi && at(lo) < key; k++) lo++;
                if (!(lo < hi && at(lo) < key)) hi = lo;
            } else if (i > beg && B.key[rf_mp(i - 1)] == key) {
                int l = beg, h = i - 1;  // the first row of the key in the tile
                while (l < h) {
                    const int m = (l + h) >> 1;
                    if (B.key[rf_mp(m)] < key) l = m + 1;
                    else h = m;
                }
                rank = (I)(i - l) + (l == 0 ? (I)rank0 : 0);
            } else if (i == 0) {
                rank = (I)rank0;
            }
            while (lo < hi) {
                const I m = (lo + hi) >> 1;
                if (at(m) < key) lo = m + 1;
                else hi = m;
            }
            p = lo;
        }
        any = true;
        prev = key;
        // whether the row `rank` after the first at or above the key holds it
        const I q = p + rank;
        const bool hit = q < wn ? at(q) == key : w0 + q < b.len && rf_key<K>(b, w0 + q) == key;
        f(j, r0 + i, key, w0 + p, (long long)rank, hit);
    }
}

// The thread's RF_MAT_TILE / T consecutive rows of the tile (from row `from` on): for the j-th,
// f(j, row, key, first row of b at or above the key, rank, whether b's row (that + rank) holds the key).
// rank0: the rank of the tile's first row; w0, w1: the window.  The whole block; ends with a barrier,
// after which B.win is free.
template <int T, class K, class F>
RF_DEV void rf_merge_walk(RfMergeBuf<K>& B, long long r0, int n, long long from, long long rank0, const RfCol& b,
                          long long w0, long long w1, F f)
{
    constexpr int CAP = RF_MERGE_CAP * 8 / (int)sizeof(K);
    if (w0 < 0) w0 = 0;
    if (w1 > b.len) w1 = b.len;
    const long long wn = w1 > w0 ? w1 - w0 : 0;
    const bool held = wn <= CAP && rank0 < (1 << 30);
    K* win = (K*)B.win;
    if (held)
        for (int i = threadIdx.x; i < (int)wn; i += T) win[i] = rf_key<K>(b, w0 + i);
    __syncthreads();
    const int beg = from > r0 ? (from - r0 < n ? (int)(from - r0) : n) : 0;
    if (held) rf_merge_rows<T, true>(B, r0, n, beg, rank0, b, w0, wn, f);
    else rf_merge_rows<T, false>(B, r0, n, beg, rank0, b, w0, wn, f);
    __syncthreads();
}
#endif  // RF_MERGE

// ---------------------------------------------------------------------------------------
// Template 3: Op materialisation (LoopGen::visit(Op), loopgen.cpp:113-204, and
// finalize_vector, vinstr.h:113-135).
//   The fragment defines rf_cond(P, r) (the iteration condition of element r) and
//   rf_emit(P, r, o) (computes the element's iterators and outputs, writes them at output row o),
//   and with RF_MAT_PREP rf_mat_prep<T>(P, tile), which a block runs before the tile's conditions.
//   Output columns: P.oc[c]; validity words: P.ov[c]; a bit per element that passes, 32 elements
//   from P.row_lo on to a word: (unsigned*)P.aux1; per-tile counts / offsets: (long long*)P.aux2;
//   the number that pass goes to *P.host_rows, the null count to *(long long*)P.aux3.
//   Compaction (vectorize off) keeps passing elements in loop order: rf_count evaluates the
//   condition once, writes its bits and each tile's count, and its last block turns the counts
//   into offsets; rf_scatter lists a tile's passing elements in shared memory and emits them 256
//   at a time, so every lane works and the output is written in order whatever share passes.
//   Vectorised (on): every visited element is written; its condition becomes the validity bit.
//   Both are bound by memory: a tile is RF_MAT_TILE elements and a block takes one tile at a time,
//   so that eight blocks an SM keep loads in flight through the few barriers of a tile.  (One
//   8192-element tile per SM with three barriers every 256 elements took 88 us to count and
//   945 us to scatter 37 % of 20M rows of 24 bytes.)
// ---------------------------------------------------------------------------------------
#ifdef RF_MATERIALIZE
RF_DEV void rf_mat_bounds(const RfParams& P, long long& lo, long long& hi)
{
    lo = P.row_lo;
    hi = P.row_hi;
    if (P.range) {
        long long b = P.range[0], e = P.range[1];
        lo = b > lo ? b : lo;
        hi = e < hi ? e : hi;
    }
}

RF_DEV long long rf_mat_ntiles(const RfParams& P)
{
    return (P.row_hi - P.row_lo + RF_MAT_TILE - 1) / RF_MAT_TILE;
}

// sum of v over the block, in every thread (sh: T / 32 words; ends with a barrier)
template <int T>
RF_DEV int rf_block_sum_int(int v, int* sh)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int w = 0; w < T / 32; w++) t += sh[w];
    __syncthreads();
    return t;
}

// exclusive scan of n tile counts in place by one block; returns the total
template <int T>
RF_DEV long long rf_mat_scan(long long* cnt, long long n)
{
    constexpr int K = 8;  // counts a thread scans in its registers per step
    __shared__ long long wsum[T / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long carry = 0;
    for (long long base = 0; base < n; base += (long long)T * K) {
        const long long i0 = base + (long long)threadIdx.x * K;
        long long v[K], x = 0;
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = i0 + k < n ? __ldcg(cnt + i0 + k) : 0;
#pragma unroll
        for (int k = 0; k < K; k++) x += v[k];
        long long incl = x;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        long long before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < T / 32; w++) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        long long o = carry + before + incl - x;
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (i0 + k < n) cnt[i0 + k] = o;
            o += v[k];
        }
        carry += all;
        __syncthreads();  // wsum is rewritten by the next step
    }
    return carry;
}

#ifndef RF_UNION  // (a union writes its visits itself)
template <int T>
RF_DEV void rf_mat_count(const RfParams& P)
{
    __shared__ int sh[T / 32];
    __shared__ int last;
    long long lo, hi;
    rf_mat_bounds(P, lo, hi);
    long long* cnt = (long long*)P.aux2;
    unsigned* bits = (unsigned*)P.aux1;
    const long long nt = rf_mat_ntiles(P);
    const int lane = threadIdx.x & 31;
    for (long long tile = blockIdx.x; tile < nt; tile += gridDim.x) {
        const long long t0 = tile * RF_MAT_TILE;  // relative to row_lo, a multiple of 32
        int c = 0;
#ifdef RF_MAT_PREP
        rf_mat_prep<T>(P, tile);
#endif
        // the conditions of all the thread's elements first: their loads are in flight together (no
        // test of the range between them in a tile that is whole)
        const long long r0 = P.row_lo + t0 + threadIdx.x;
        bool ok[RF_MAT_TILE / T];
        if (P.row_lo + t0 >= lo && P.row_lo + t0 + RF_MAT_TILE <= hi) {
#pragma unroll
            for (int j = 0; j < RF_MAT_TILE / T; j++) ok[j] = rf_cond(P, r0 + j * T);
        } else {
#pragma unroll
            for (int j = 0; j < RF_MAT_TILE / T; j++) ok[j] = r0 + j * T >= lo && r0 + j * T < hi && rf_cond(P, r0 + j * T);
        }
#pragma unroll
        for (int j = 0; j < RF_MAT_TILE / T; j++) {
            const unsigned m = __ballot_sync(0xffffffffu, ok[j]);
            if (lane == 0) {
                bits[(t0 + j * T + threadIdx.x) >> 5] = m;
                c += __popc(m);
            }
        }
        c = rf_block_sum_int<T>(c, sh);
        if (threadIdx.x == 0) __stcg(cnt + tile, (long long)c);
    }
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(P.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const long long total = rf_mat_scan<T>(cnt, nt);
    if (threadIdx.x == 0) {
        *P.host_rows = total;
        *P.counter = 0u;
    }
}

template <int T>
RF_DEV void rf_mat_scatter(const RfParams& P)
{
    constexpr int NW = RF_MAT_TILE / 32;  // words of a tile
    static_assert(NW == 64, "a warp scans a tile's words two to a lane");
    __shared__ unsigned short idx[RF_MAT_TILE];
    const long long* off = (const long long*)P.aux2;
    const unsigned* bits = (const unsigned*)P.aux1;
    const long long nt = rf_mat_ntiles(P);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long tile = blockIdx.x; tile < nt; tile += gridDim.x) {
        const long long base = __ldg(off + tile);
        // every warp scans the counts of all words, then lists its own share of them
        const unsigned a = __ldg(bits + tile * NW + 2 * lane), b = __ldg(bits + tile * NW + 2 * lane + 1);
        const int pa = __popc(a), pb = __popc(b);
        int incl = pa + pb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const int n = __shfl_sync(0xffffffffu, incl, 31);
        const int ea = incl - pa - pb;
#pragma unroll
        for (int k = 0; k < NW / (T / 32); k++) {
            const int w = warp * (NW / (T / 32)) + k;
            const unsigned m = __shfl_sync(0xffffffffu, (w & 1) ? b : a, w >> 1);
            const int o = __shfl_sync(0xffffffffu, (w & 1) ? ea + pa : ea, w >> 1);
            if ((m >> lane) & 1u) idx[o + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(w * 32 + lane);
        }
        __syncthreads();
        const long long r0 = P.row_lo + tile * RF_MAT_TILE;
        for (int i = threadIdx.x; i < n; i += T) rf_emit(P, r0 + idx[i], base + i);
        __syncthreads();  // the list is rewritten by the next tile
    }
}

template <int T>
RF_DEV void rf_mat_write_all(const RfParams& P, int ncols)
{
    long long lo, hi;
    rf_mat_bounds(P, lo, hi);
    const long long nt = rf_mat_ntiles(P);
    const int lane = threadIdx.x & 31;
    // the output starts at lo: where that is a whole number of words into the tiles, a warp's 32
    // elements are one word of their own, else they share two words with the neighbouring warps
    const bool whole = ((lo - P.row_lo) & 31) == 0;
    long long nulls = 0;
    for (long long tile = blockIdx.x; tile < nt; tile += gridDim.x) {
#ifdef RF_MAT_PREP
        rf_mat_prep<T>(P, tile);
#endif
#pragma unroll
        for (int j = 0; j < RF_MAT_TILE; j += T) {
            const long long r = P.row_lo + tile * RF_MAT_TILE + j + threadIdx.x;
            const bool in = r >= lo && r < hi;
            const bool c = in && rf_cond(P, r);
            if (in) rf_emit(P, r, r - lo);
            const unsigned m = __ballot_sync(0xffffffffu, c);
            const unsigned act = __ballot_sync(0xffffffffu, in);
            nulls += __popc(act & ~m);
            if (!act) continue;
            const int f = __ffs(act) - 1;  // the warp's first element in range
            const long long o0 = __shfl_sync(0xffffffffu, r - lo, f);
            for (int col = lane; col < ncols; col += 32) {
                unsigned* bm = P.ov[col] + (o0 >> 5);
                if (whole) {
                    *bm = m;
                } else {
                    const int sft = (int)(o0 & 31);
                    atomicOr(bm, (m >> f) << sft);
                    if (sft && ((m >> f) >> (32 - sft))) atomicOr(bm + 1, (m >> f) >> (32 - sft));
                }
            }
        }
    }
    if (lane == 0 && nulls) atomicAdd((unsigned long long*)P.aux3, (unsigned long long)nulls);
}

#define RF_MATERIALIZE_KERNELS(T, NCOLS)                                                                  \
    extern "C" __global__ void __launch_bounds__(T) rf_count(const __grid_constant__ RfParams P)         \
    {                                                                                                    \
        rf_mat_count<T>(P);                                                                              \
    }                                                                                                    \
    extern "C" __global__ void __launch_bounds__(T) rf_scatter(const __grid_constant__ RfParams P)       \
    {                                                                                                    \
        rf_mat_scatter<T>(P);                                                                            \
    }                                                                                                    \
    extern "C" __global__ void __launch_bounds__(T) rf_write_all(const __grid_constant__ RfParams P)     \
    {                                                                                                    \
        rf_mat_write_all<T>(P, NCOLS);                                                                   \
    }
#endif  // RF_UNION
#endif  // RF_MATERIALIZE

// ---------------------------------------------------------------------------------------
// Union merge of two sorted int64 key columns A and B (template 3's tiles over B, then over both).
//   The fragment defines rf_u_a(P), rf_u_b(P) (the key columns), rf_u_write(P, li, ri, v, o) (the
//   visit's outputs at output row o) and, vectorised, RF_UNION_VALID (output columns).
//   (long long*)P.aux4: {rank, window start} of each tile boundary of A (P.aux_n0 tiles + 1), then of
//   B (P.aux_n1 + 1); (long long*)P.aux5: of each B row, the A rows up to its key if it is unpaired,
//   else -1; (unsigned*)P.aux1: a bit per B row, unpaired; (unsigned short*)P.aux0: unpaired rows of
//   the tile before each word; (long long*)P.aux2: and of the tiles before each tile; visits: *P.host_rows, then P.out_rows.
// Both key columns are read twice (once to find what is unpaired, once to write); the rest of the
// traffic is the outputs.  (3M rows against 2.5M with 40 % of the keys shared: 1749 us a call with
// three binary searches a row in each of two kernels on one block an SM, 657 us with the GPU full of
// them, 210 us so.)
// ---------------------------------------------------------------------------------------
#ifdef RF_UNION
// the first row of c at or after lo with a key above `key`, knowing that row hi has one (or is the end)
RF_DEV long long rf_u_upper(const RfCol& c, long long lo, long long hi, long long key)
{
    if (hi > c.len) hi = c.len;
    while (lo < hi) {
        const long long m = (lo + hi) >> 1;
        if (rf_key<int64_t>(c, m) <= key) lo = m + 1;
        else hi = m;
    }
    return lo;
}

// (whole warp) {rank, window start} of boundary t of the tiles of `a`
RF_DEV void rf_u_bound(const RfCol& a, const RfCol& b, long long t, long long* out)
{
    const long long x = t * RF_MAT_TILE;
    long long rank = 0, lb = b.len;
    if (x < a.len) {
        const long long key = rf_key<int64_t>(a, x);
        rank = rf_merge_rank<int64_t>(a, 0, x, key);
        lb = rf_merge_bound<int64_t>(b, 0, key);
    }
    if ((threadIdx.x & 31) == 0) {
        out[2 * t] = rank;
        out[2 * t + 1] = lb;
    }
}

RF_DEV void rf_u_part_all(const RfParams& P)
{
    const long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    long long* out = (long long*)P.aux4;
    if (w <= P.aux_n0) rf_u_bound(rf_u_a(P), rf_u_b(P), w, out);
    else if (w - P.aux_n0 - 1 <= P.aux_n1) rf_u_bound(rf_u_b(P), rf_u_a(P), w - P.aux_n0 - 1, out + 2 * (P.aux_n0 + 1));
}

template <int T>
RF_DEV void rf_u_count_all(const RfParams& P)
{
    constexpr int R = RF_MAT_TILE / T;
    __shared__ RfMergeBuf<int64_t> B;
    __shared__ int sh[T / 32];
    __shared__ int last;
    const RfCol &a = rf_u_a(P), &b = rf_u_b(P);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long* cnt = (long long*)P.aux2;
    for (long long tile = blockIdx.x; tile < P.aux_n1; tile += gridDim.x) {
        const long long r0 = tile * RF_MAT_TILE;
        const int n = b.len - r0 < RF_MAT_TILE ? (int)(b.len - r0) : RF_MAT_TILE;
        const long long* part = (const long long*)P.aux4 + 2 * (P.aux_n0 + 1) + 2 * tile;
        rf_merge_load<T>(B, b, r0, n);
        long long j[R];
#pragma unroll
        for (int q = 0; q < R; q++) j[q] = -1;
        rf_merge_walk<T>(B, r0, n, 0, __ldg(part), a, __ldg(part + 1), __ldg(part + 3),
                         [&](int q, long long, long long key, long long lb, long long rank, bool hit) {
                             if (!hit) j[q] = rank ? rf_u_upper(a, lb, lb + rank, key) : lb;
                         });
#pragma unroll
        for (int q = 0; q < R; q++) B.win[rf_mp((int)threadIdx.x * R + q)] = j[q];
        __syncthreads();
        int c = 0;
#pragma unroll
        for (int q = 0; q < RF_MAT_TILE; q += T) {
            const int i = q + (int)threadIdx.x;
            const long long x = B.win[rf_mp(i)];
            if (i < n) ((long long*)P.aux5)[r0 + i] = x;
            const unsigned m = __ballot_sync(0xffffffffu, x >= 0);
            if (lane == 0) {
                ((unsigned*)P.aux1)[(r0 + i) >> 5] = m;
                B.key[i >> 5] = __popc(m);  // the keys are not read again
                c += __popc(m);
            }
        }
        c = rf_block_sum_int<T>(c, sh);
        if (threadIdx.x == 0) __stcg(cnt + tile, (long long)c);
        if (warp == 0) {  // words before each word, two words to a lane
            const int x = (int)B.key[2 * lane], y = (int)B.key[2 * lane + 1];
            int incl = x + y;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int z = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += z;
            }
            ((unsigned*)P.aux0)[tile * (RF_MAT_TILE / 64) + lane] = (unsigned)(incl - x - y) | (unsigned)(incl - y) << 16;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(P.counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const long long total = rf_mat_scan<T>(cnt, P.aux_n1);
    if (threadIdx.x == 0) {
        *P.host_rows = a.len + total;
        *P.counter = 0u;
    }
}

// writes a visit; false: a null row.  Keys out of order (the walk needs sorted iterator columns) can
// move a visit, never past the output: positions are checked against the visit count.
RF_DEV bool rf_u_visit(const RfParams& P, long long li, long long ri, long long v, long long pos, long long V)
{
    if (pos < 0 || pos >= V) {
        rf_set_err(P, RF_DEVERR_RANGE);
        return true;
    }
    rf_u_write(P, li, ri, v, pos);
#ifdef RF_UNION_VALID
    const RfCol &a = rf_u_a(P), &b = rf_u_b(P);
    if (!((li < a.len && rf_valid(a.valid, li)) || (ri < b.len && rf_valid(b.valid, ri)))) return false;
    for (int col = 0; col < RF_UNION_VALID; col++) atomicOr(P.ov[col] + (pos >> 5), 1u << (pos & 31));
#endif
    return true;
}

template <int T>
RF_DEV void rf_u_emit_all(const RfParams& P)
{
    constexpr int R = RF_MAT_TILE / T, NW = RF_MAT_TILE / 32;
    __shared__ RfMergeBuf<int64_t> B;
    const RfCol &a = rf_u_a(P), &b = rf_u_b(P);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long* off = (const long long*)P.aux2;
    const unsigned* bits = (const unsigned*)P.aux1;
    const unsigned short* before = (const unsigned short*)P.aux0;
    const long long V = P.out_rows;
    long long nulls = 0;
    // the tiles of both sides in turn, so that the visits of one stretch of keys are written at about the
    // same time: rows of the two sides share sectors of the outputs (B's tiles after all of A's: 378 MB
    // read, 243 MB written for 144 MB of outputs)
    const long long nt = P.aux_n0 + P.aux_n1;
    for (long long g = blockIdx.x; g < nt; g += gridDim.x) {
        const long long ta = g * P.aux_n0 / nt;
        if ((g + 1) * P.aux_n0 / nt > ta) {  // a tile of A: every row has a visit
            const long long tile = ta, r0 = tile * RF_MAT_TILE;
            const int n = a.len - r0 < RF_MAT_TILE ? (int)(a.len - r0) : RF_MAT_TILE;
            const long long* part = (const long long*)P.aux4 + 2 * tile;
            rf_merge_load<T>(B, a, r0, n);
            long long l[R], x[R];
#pragma unroll
            for (int q = 0; q < R; q++) l[q] = x[q] = 0;
            rf_merge_walk<T>(B, r0, n, 0, __ldg(part), b, __ldg(part + 1), __ldg(part + 3),
                             [&](int q, long long, long long key, long long lb, long long rank, bool hit) {
                                 l[q] = lb;
                                 x[q] = hit || rank == 0 ? lb + rank : rf_u_upper(b, lb, lb + rank, key);
                             });
#pragma unroll
            for (int q = 0; q < R; q++) {
                B.win[rf_mp((int)threadIdx.x * R + q)] = l[q];
                B.key[rf_mp((int)threadIdx.x * R + q)] = x[q];
            }
            __syncthreads();
            for (int i = threadIdx.x; i < n; i += T) {
                const long long lb = B.win[rf_mp(i)];
                long long u = V - a.len;  // unpaired rows of B before its row lb
                if (lb < b.len)
                    u = __ldg(off + (lb / RF_MAT_TILE)) + __ldg(before + (lb >> 5)) +
                        __popc(__ldg(bits + (lb >> 5)) & ((1u << (lb & 31)) - 1u));
                nulls += !rf_u_visit(P, r0 + i, B.key[rf_mp(i)], rf_key<int64_t>(a, r0 + i), r0 + i + u, V);
            }
        } else {  // a tile of B: its unpaired rows, listed in shared memory
            const long long t = g - ta, r0 = t * RF_MAT_TILE, base = __ldg(off + t);
            unsigned short* idx = (unsigned short*)B.win;
            int total = 0;
            for (int w = warp; w < NW; w += T / 32) {
                const unsigned m = __ldg(bits + t * NW + w);
                if ((m >> lane) & 1u)
                    idx[__ldg(before + t * NW + w) + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(w * 32 + lane);
            }
            total = __ldg(before + t * NW + NW - 1) + __popc(__ldg(bits + t * NW + NW - 1));
            __syncthreads();
            for (int i = threadIdx.x; i < total; i += T) {
                const long long j = r0 + idx[i], li = ((const long long*)P.aux5)[j];
                nulls += !rf_u_visit(P, li, j, rf_key<int64_t>(b, j), li + base + i, V);
            }
        }
        __syncthreads();
    }
    if (nulls) atomicAdd((unsigned long long*)P.aux3, (unsigned long long)nulls);
}

#define RF_UNION_KERNELS(T)                                                                               \
    extern "C" __global__ void __launch_bounds__(256) rf_u_part(const __grid_constant__ RfParams P)      \
    {                                                                                                    \
        rf_u_part_all(P);                                                                                \
    }                                                                                                    \
    extern "C" __global__ void __launch_bounds__(T) rf_u_count(const __grid_constant__ RfParams P)       \
    {                                                                                                    \
        rf_u_count_all<T>(P);                                                                            \
    }                                                                                                    \
    extern "C" __global__ void __launch_bounds__(T) rf_u_emit(const __grid_constant__ RfParams P)        \
    {                                                                                                    \
        rf_u_emit_all<T>(P);                                                                             \
    }
#endif  // RF_UNION

// ---------------------------------------------------------------------------------------
// Template 4: segmented reduce over run-end encoded rows (an Op over a 2-d vector whose output
// reduces each run, loopgen.cpp:34-38, 206-269).
//   The fragment defines RfAcc and its functions as template 1 does, RF_SEG_M (items of a tile, a
//   multiple of RF_SEG_T), rf_seg_runs(P) (the run-end column), struct RfSegRows (RF_SEG_M rows of
//   the columns a row reads), rf_seg_stage(P, r, i, S) and rf_seg_row(P, r, i, S, A).
//   P.aux_n0: rows, P.aux_n1: tiles; (long long*)P.aux4: the run each tile starts in (tiles + 1);
//   (RfAcc*)P.aux5: a state per run, then a state per tile (its rows after its last run end).
// Rows and run ends are merged into one sequence - run end j comes after the rows before it, at
// position ends[j] + j - and cut into tiles of RF_SEG_M items and threads of RF_SEG_M / RF_SEG_T,
// so every thread does the same work however long the runs are (Merrill and Garland, merge-based
// sparse matrix-vector product, SC16).  A run inside a thread is stored by it; a run that spans
// threads is joined by a segmented scan over the block, one that spans tiles by rf_seg_fix; all in
// row order, by the tiles alone, so the bits do not depend on the scheduling.  Bound by reading
// the rows: they are staged through shared memory, whole sectors a warp, and so are the run ends.
// (20M rows of one double in 2M Zipf(1.1) runs: 2.37 ms a call with a thread to each 256 rows of a
// run and one thread folding a run's pieces in turn, of which 1.94 ms were those folds; 0.21 ms so.)
// ---------------------------------------------------------------------------------------
#ifdef RF_SEG_REDUCE
RF_DEV long long rf_seg_end(const RfParams& P, long long run)
{
    const long long e = (long long)__ldg(rf_seg_runs(P).run_ends + run);
    return e < P.aux_n0 ? e : P.aux_n0;
}

// a state, through L2 (16 bytes in one load)
RF_DEV void rf_seg_ld(RfAcc& a, const RfAcc* p)
{
    if constexpr (sizeof(RfAcc) == 16) {
        union U {
            ulonglong2 v;
            RfAcc a;
            RF_DEV_MEMBER U() {}
        } u;
        u.v = __ldcg((const ulonglong2*)p);
        a = u.a;
    } else {
        rf_ld_words(&a, p, (int)sizeof(RfAcc));
    }
}

// the tile's first run: the run ends before item d
extern "C" __global__ void __launch_bounds__(256) rf_seg_part(const __grid_constant__ RfParams P)
{
    const long long t = (blockIdx.x * 256ll + threadIdx.x) >> 5;
    if (t > P.aux_n1) return;
    const long long n = rf_seg_runs(P).len, d = t * RF_SEG_M;
    const long long x = rf_warp_search(0, n, [&](long long j) { return rf_seg_end(P, j) + j < d; });
    if ((threadIdx.x & 31) == 0) ((long long*)P.aux4)[t] = x;
}

// segmented scan over the block: `closed`/`a` of this thread -> the state that the rows of the
// threads before it (and `in`, before the first) carry into it (those since the last run end); the
// block's own carry out in *out, by its last thread.  A state combines with what precedes it on the left.
template <int T>
RF_DEV RfAcc rf_seg_carry(const RfAcc& in, bool closed, const RfAcc& a, RfAcc* warp_a, unsigned char* warp_f, RfAcc* out)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    RfAcc v = a;
    bool f = closed;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        RfAcc u = rf_shfl_up(v, off);
        const bool uf = __shfl_up_sync(0xffffffffu, (int)f, off) != 0;
        if (lane >= off) {
            if (!f) {
                rf_acc_combine(u, v);
                v = u;
            }
            f = f || uf;
        }
    }
    if (lane == 31) {
        warp_a[warp] = v;
        warp_f[warp] = f;
    }
    __syncthreads();
    // what the warps before this one carry in, then this warp's lanes before this one
    RfAcc c = in;
    for (int w = 0; w < warp; w++) {
        if (warp_f[w]) c = warp_a[w];
        else rf_acc_combine(c, warp_a[w]);
    }
    if (threadIdx.x == T - 1) {
        RfAcc o = c;
        if (f) o = v;
        else rf_acc_combine(o, v);
        *out = o;
    }
    RfAcc u = rf_shfl_up(v, 1);
    const bool uf = __shfl_up_sync(0xffffffffu, (int)f, 1) != 0;
    if (lane > 0) {
        if (uf) c = u;
        else rf_acc_combine(c, u);
    }
    return c;
}

extern "C" __global__ void __launch_bounds__(RF_SEG_T) rf_seg_reduce(const __grid_constant__ RfParams P)
{
    constexpr int T = RF_SEG_T, K = RF_SEG_M / RF_SEG_T;
    __shared__ RfSegRows S;
    static_assert(RF_SEG_M < 65535, "run ends of a tile in 16 bits");
    __shared__ unsigned short ends[RF_SEG_M + 1];  // run ends of the tile, relative to its first row
    __shared__ RfAcc warp_a[T / 32];
    __shared__ unsigned char warp_f[T / 32];
    const long long* part = (const long long*)P.aux4;
    RfAcc* res = (RfAcc*)P.aux5;
    const long long n = rf_seg_runs(P).len;
    const long long total = (n > 0 ? rf_seg_end(P, n - 1) : 0) + n;  // items
    const long long tile = blockIdx.x;
    if (tile >= P.aux_n1) return;  // bounds tile and tile + 1 are rf_seg_part's
    long long d0 = tile * RF_SEG_M, d1 = d0 + RF_SEG_M;
    if (d0 > total) d0 = total;
    if (d1 > total) d1 = total;
    const long long xa = __ldg(part + tile), xb = __ldg(part + tile + 1);  // within the runs (rf_warp_search)
    // (bounded for columns whose run ends are out of order, too: never more than a tile's)
    int nx = (int)(xb - xa < 0 ? 0 : xb - xa > RF_SEG_M ? RF_SEG_M : xb - xa);
    const long long ra = d0 - xa;
    int nr = (int)(d1 - d0) - nx;
    if (nr < 0 || ra < 0 || ra + nr > P.aux_n0) nr = 0;
    for (int i = threadIdx.x; i < nr; i += T) rf_seg_stage(P, ra + i, i, S);
    for (int i = threadIdx.x; i < nx; i += T) {
        const long long e = rf_seg_end(P, xa + i) - ra;  // (in the tile, unless run ends are out of order)
        ends[i] = (unsigned short)(e < 0 ? 0 : e > RF_SEG_M ? RF_SEG_M : e);
    }
    __syncthreads();
    // the thread's first item: the run ends before it
    const int items = nr + nx;
    int at = (int)threadIdx.x * K;
    if (at > items) at = items;
    int lo = at - nr > 0 ? at - nr : 0, hi = at < nx ? at : nx;
    while (lo < hi) {
        const int m = (lo + hi) >> 1;
        if (ends[m] + m < at) lo = m + 1;
        else hi = m;
    }
    int x = lo, r = at - lo;
    const int first = x;
    RfAcc A, head;
    rf_acc_init(P, A);
    head = A;
    bool closed = false;
    int e = x < nx ? ends[x] : 0x7fffffff;
    for (int k = 0; k < K && r + x < items; k++) {
        if (r < e && r < nr) {
            rf_seg_row(P, ra + r, r, S, A);
            r++;
        } else if (x < nx) {
            if (!closed) head = A;
            else rf_st_words(res + xa + x, &A, (int)sizeof(RfAcc));
            closed = true;
            rf_acc_init(P, A);
            x++;
            e = x < nx ? ends[x] : 0x7fffffff;
        }
    }
    RfAcc none, out;
    rf_acc_init(P, none);
    RfAcc c = rf_seg_carry<T>(none, closed, A, warp_a, warp_f, &out);
    if (closed) {
        rf_acc_combine(c, head);
        rf_st_words(res + xa + first, &c, (int)sizeof(RfAcc));
    }
    if (threadIdx.x == T - 1) rf_st_words(res + n + tile, &out, (int)sizeof(RfAcc));
}

// Joins the runs that span tiles: the carries of the tiles since a run began, onto its state.  One
// block takes T * K tiles at a time, K to a thread, with all their loads issued before any is used
// (7800 tiles: 41 us with each thread walking its share twice, one load after another, 26 us so).
extern "C" __global__ void __launch_bounds__(512) rf_seg_fix(const __grid_constant__ RfParams P)
{
    // (1024 threads of 2 tiles take 40 us: every warp adds up what the ones before it carry in)
    constexpr int T = 512, K = sizeof(RfAcc) <= 16 ? 8 : sizeof(RfAcc) <= 32 ? 4 : 1;
    __shared__ RfAcc warp_a[T / 32], carry;
    __shared__ unsigned char warp_f[T / 32];
    const long long* part = (const long long*)P.aux4;
    RfAcc* res = (RfAcc*)P.aux5;
    const long long n = rf_seg_runs(P).len, nt = P.aux_n1;
    RfAcc in;
    rf_acc_init(P, in);
    for (long long base = 0; base < nt; base += T * K) {
        const long long t0 = base + (long long)threadIdx.x * K;
        long long x[K + 1];
        RfAcc b[K], h[K];
#pragma unroll
        for (int k = 0; k <= K; k++) x[k] = t0 + k <= nt ? __ldg(part + t0 + k) : 0;
#pragma unroll
        for (int k = 0; k < K; k++)
            if (t0 + k < nt) rf_seg_ld(b[k], res + n + t0 + k);
        // the states of the tiles' first runs, of those that end in their tile
#pragma unroll
        for (int k = 0; k < K; k++)
            if (t0 + k < nt && x[k + 1] > x[k]) rf_seg_ld(h[k], res + x[k]);
        RfAcc A;
        rf_acc_init(P, A);
        bool closed = false;
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (t0 + k >= nt) continue;
            if (x[k + 1] > x[k]) {
                closed = true;
                A = b[k];
            } else {
                rf_acc_combine(A, b[k]);
            }
        }
        RfAcc c = rf_seg_carry<T>(in, closed, A, warp_a, warp_f, &carry);
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (t0 + k >= nt) continue;
            if (x[k + 1] > x[k]) {
                rf_acc_combine(c, h[k]);
                rf_st_words(res + x[k], &c, (int)sizeof(RfAcc));
                c = b[k];
            } else {
                rf_acc_combine(c, b[k]);
            }
        }
        __syncthreads();
        in = carry;
        __syncthreads();  // warp_a and carry are rewritten by the next step
    }
}
#endif  // RF_SEG_REDUCE
