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

// Batched form: one persistent launch runs the work units of many queries of this shape.
// work[w] = {query, unit}; params[query] is the query's parameter block.  A query's units are
// the ones its stand-alone launch would run, folded in the same order: same bits either way.
#define RF_SCAN_REDUCE_KERNEL(NAME, T)                                                      \
    extern "C" __global__ void __launch_bounds__(T) NAME(const __grid_constant__ RfParams P) \
    {                                                                                       \
        RfAcc acc;                                                                          \
        rf_acc_init(P, acc);                                                                \
        rf_scan_reduce_rows<T>(P, P.unit0 + (int)blockIdx.x, P.nunits, acc);                \
        rf_scan_reduce_merge<T>(P, P.unit0 + (int)blockIdx.x, P.nunits, acc);               \
    }                                                                                       \
    extern "C" __global__ void __launch_bounds__(T)                                         \
        rf_batch(const RfParams* __restrict__ params, const int2* __restrict__ work, const int* nwork) \
    {                                                                                       \
        const int n = *nwork;                                                               \
        for (int w = blockIdx.x; w < n; w += gridDim.x) {                                   \
            const int2 it = work[w];                                                        \
            const RfParams& Q = params[it.x];                                               \
            if (it.y < 0 || it.y >= Q.nunits) { /* a malformed work item: report, skip */  \
                if (threadIdx.x == 0) atomicExch(Q.err, RF_DEVERR_RANGE);                    \
                continue;                                                                   \
            }                                                                               \
            RfAcc acc;                                                                      \
            rf_acc_init(Q, acc);                                                            \
            rf_scan_reduce_rows<T>(Q, it.y, Q.nunits, acc);                                 \
            rf_scan_reduce_merge<T>(Q, it.y, Q.nunits, acc);                                \
        }                                                                                   \
    }
#endif  // RF_SCAN_REDUCE

// ---------------------------------------------------------------------------------------
// Template 2: grouped scan-reduce with shared-memory privatised accumulators.
//   The fragment defines RF_G groups x RF_M aggregates, struct RfVals, rf_group(P, r, V)
//   (group id or -1, and the row's aggregate inputs), rf_slot_init(m) (64-bit identity),
//   rf_slot_combine(m, a, b), rf_slot_add(S, g, t, V, df), rf_slots_done(S, t, df) (df: the
//   thread keeps its FP64 sums as double-floats, see rf_device.cuh) and
//   rf_finish_groups(P, tot, out).  With RF_GROUP_SPLIT it also defines the row's loads apart,
//   struct RfRowLd, rf_group_ld(P, r, L) and rf_group_v(P, r, L, V) (rf_group is the two in turn).
// Each thread owns a private column of G*M 64-bit slots in shared memory (slot (q, t) at
// S[q * T + t]): no atomics and no bank conflicts on the per-row update.  At the end every
// slot column is folded over the block in a fixed order, then over units by the last unit.
// ---------------------------------------------------------------------------------------
#ifdef RF_GROUP_REDUCE
template <int T>
RF_DEV void rf_group_reduce(const RfParams& P, int unit, int nunits)
{
    extern __shared__ unsigned long long S[];
    __shared__ int last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Q = RF_G * RF_M;
    for (int q = 0; q < Q; q++) S[q * T + tid] = rf_slot_init(P, q % RF_M);
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
    rf_slots_done(S, tid, df);
    __syncthreads();
    unsigned long long* part = (unsigned long long*)P.partials;
    for (int q = warp; q < Q; q += T / 32) {
        const int m = q % RF_M;
        unsigned long long a = S[q * T + lane];
        for (int k = 1; k < T / 32; k++) a = rf_slot_combine(m, a, S[q * T + lane + 32 * k]);
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
            int u = lane;
            for (; u + 32 * (RF_FOLD - 1) < nunits; u += 32 * RF_FOLD) {
                unsigned long long v[RF_FOLD];
#pragma unroll
                for (int k = 0; k < RF_FOLD; k++) v[k] = __ldcg(part + (long long)(u + 32 * k) * Q + q);
#pragma unroll
                for (int k = 0; k < RF_FOLD; k++) a = rf_slot_combine(m, a, v[k]);
            }
            for (; u < nunits; u += 32) a = rf_slot_combine(m, a, __ldcg(part + (long long)u * Q + q));
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) a = rf_slot_combine(m, a, __shfl_down_sync(0xffffffffu, a, off));
            if (lane == 0) S[q] = a;
        }
        __syncthreads();
        if (tid == 0) {
            rf_finish_groups(P, S, P.out);
            *P.counter = 0u;
        }
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
        rf_batch(const RfParams* __restrict__ params, const int2* __restrict__ work, const int* nwork) \
    {                                                                                       \
        const int n = *nwork;                                                               \
        for (int w = blockIdx.x; w < n; w += gridDim.x) {                                   \
            const int2 it = work[w];                                                        \
            if (it.y < 0 || it.y >= params[it.x].nunits) { /* malformed work item */       \
                if (threadIdx.x == 0) atomicExch(params[it.x].err, RF_DEVERR_RANGE);         \
                continue;                                                                   \
            }                                                                               \
            rf_group_reduce<T>(params[it.x], it.y, params[it.x].nunits);                    \
        }                                                                                   \
    }
#endif  // RF_GROUP_REDUCE


// ---------------------------------------------------------------------------------------
// Template 3: Op materialisation (LoopGen::visit(Op), loopgen.cpp:113-204, and
// finalize_vector, vinstr.h:113-135).
//   The fragment defines rf_cond(P, r) (the iteration condition of element r) and
//   rf_emit(P, r, o) (computes the element's iterators and outputs, writes them at output row o).
//   Output columns: P.oc[c]; validity words: P.ov[c]; a bit per element that passes, 32 elements
//   from P.row_lo on to a word: (unsigned*)P.aux1; per-tile counts / offsets: (long long*)P.aux2;
//   results (long long*)P.aux3: [0] = rows written, [1] = null count.
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

// exclusive scan of n tile counts in place by one block; total -> *total
template <int T>
RF_DEV void rf_mat_scan(long long* cnt, long long n, long long* total)
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
    if (threadIdx.x == 0) *total = carry;
}

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
#pragma unroll
        for (int j = 0; j < RF_MAT_TILE; j += T) {
            const long long r = P.row_lo + t0 + j + threadIdx.x;
            const unsigned m = __ballot_sync(0xffffffffu, r >= lo && r < hi && rf_cond(P, r));
            if (lane == 0) {
                bits[(t0 + j + threadIdx.x) >> 5] = m;
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
    rf_mat_scan<T>(cnt, nt, (long long*)P.aux3);
    if (threadIdx.x == 0) *P.counter = 0u;
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
    if (lane == 0 && nulls) atomicAdd((unsigned long long*)P.aux3 + 1, (unsigned long long)nulls);
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
#endif  // RF_MATERIALIZE

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
// run and one thread folding a run's pieces in turn, of which 1.94 ms were those folds; 0.33 ms so.)
// ---------------------------------------------------------------------------------------
#ifdef RF_SEG_REDUCE
RF_DEV long long rf_seg_end(const RfParams& P, long long run)
{
    const long long e = (long long)__ldg(rf_seg_runs(P).run_ends + run);
    return e < P.aux_n0 ? e : P.aux_n0;
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
// threads before it carry into it (those since the last run end); the block's own carry out in
// *out.  A state combines with what precedes it on the left.
template <int T>
RF_DEV RfAcc rf_seg_carry(const RfParams& P, bool closed, const RfAcc& a, RfAcc* warp_a, unsigned char* warp_f, RfAcc* out)
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
    RfAcc c;
    rf_acc_init(P, c);
    for (int w = 0; w < warp; w++) {
        if (warp_f[w]) c = warp_a[w];
        else rf_acc_combine(c, warp_a[w]);
    }
    if (threadIdx.x == T - 1 && out) {
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
    __shared__ int ends[RF_SEG_M + 1];  // run ends of the tile, relative to its first row
    __shared__ RfAcc warp_a[T / 32];
    __shared__ unsigned char warp_f[T / 32];
    const long long* part = (const long long*)P.aux4;
    RfAcc* res = (RfAcc*)P.aux5;
    const long long n = rf_seg_runs(P).len;
    const long long total = (n > 0 ? rf_seg_end(P, n - 1) : 0) + n;  // items
    const long long tile = blockIdx.x;
    long long d0 = tile * RF_SEG_M, d1 = d0 + RF_SEG_M;
    if (d0 > total) d0 = total;
    if (d1 > total) d1 = total;
    const long long xa = __ldg(part + tile), xb = __ldg(part + tile + 1);
    // (bounded for columns whose run ends are out of order, too: never more than a tile's)
    int nx = (int)(xb - xa < 0 ? 0 : xb - xa > RF_SEG_M ? RF_SEG_M : xb - xa);
    const long long ra = d0 - xa;
    int nr = (int)(d1 - d0) - nx;
    if (nr < 0 || ra < 0 || ra + nr > P.aux_n0) nr = 0;
    for (int i = threadIdx.x; i < nr; i += T) rf_seg_stage(P, ra + i, i, S);
    for (int i = threadIdx.x; i < nx; i += T) ends[i] = (int)(rf_seg_end(P, xa + i) - ra);
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
    RfAcc out;
    RfAcc c = rf_seg_carry<T>(P, closed, A, warp_a, warp_f, &out);
    if (closed) {
        rf_acc_combine(c, head);
        rf_st_words(res + xa + first, &c, (int)sizeof(RfAcc));
    }
    if (threadIdx.x == T - 1) rf_st_words(res + n + tile, &out, (int)sizeof(RfAcc));
}

// joins the runs that span tiles: the carries of the tiles since a run began, onto its state
extern "C" __global__ void __launch_bounds__(512) rf_seg_fix(const __grid_constant__ RfParams P)
{
    constexpr int T = 512;
    __shared__ RfAcc warp_a[T / 32];
    __shared__ unsigned char warp_f[T / 32];
    const long long* part = (const long long*)P.aux4;
    RfAcc* res = (RfAcc*)P.aux5;
    const long long n = rf_seg_runs(P).len, nt = P.aux_n1;
    // a thread takes K consecutive tiles: first their carry out, then, with what is carried into
    // them, their first runs
    const long long K = (nt + T - 1) / T;
    const long long t0 = threadIdx.x * K < nt ? threadIdx.x * K : nt, t1 = t0 + K < nt ? t0 + K : nt;
    RfAcc A, b;
    rf_acc_init(P, A);
    bool closed = false;
    for (long long t = t0; t < t1; t++) {
        rf_ld_words(&b, res + n + t, (int)sizeof(RfAcc));
        if (part[t + 1] > part[t]) {
            closed = true;
            A = b;
        } else {
            rf_acc_combine(A, b);
        }
    }
    RfAcc c = rf_seg_carry<T>(P, closed, A, warp_a, warp_f, nullptr);
    for (long long t = t0; t < t1; t++) {
        const long long x = part[t];
        rf_ld_words(&b, res + n + t, (int)sizeof(RfAcc));
        if (part[t + 1] > x) {
            RfAcc h;
            rf_ld_words(&h, res + x, (int)sizeof(RfAcc));
            rf_acc_combine(c, h);
            rf_st_words(res + x, &c, (int)sizeof(RfAcc));
            c = b;
        } else {
            rf_acc_combine(c, b);
        }
    }
}
#endif  // RF_SEG_REDUCE
