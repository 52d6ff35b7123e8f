// Conservative AABB pair cull, in the reference's pair enumeration order.
//
// The reference has no broadphase: DetectCollisions runs GJK on every pair of a scene in the
// fixed order CC (i<j), CF, SF, CS, SS (code/nans.cpp:1355-1535) and appends hits in that order.
// Here a scene's pairs are numbered in that order and grouped in 32-pair mask words; a scene's
// words are contiguous and start on a word boundary (scene s owns words [sc_word0[s],
// sc_word0[s+1]); word_scene maps a word back to its scene). Two passes keep the order while
// skipping pairs whose inflated AABBs are disjoint:
//   k_cull_tiles  the words' bits: cube-cube pairs by 32 x 32 tiles, the others in chunks of 32
//   k_cull_place  the candidates in pair order: per block of words a scan, the block's
//                 place by looking back over the earlier blocks' counts (the decoupled look-back of
//                 Merrill and Garland's single-pass scan, 2016), one thread per candidate
// The all-pairs mode and the tuning's alternative make the bits in k_cull_place itself.
//
// 16,384 stacks (63 M pairs, 0.95 M candidates): the separate count, scan and write passes took 9 +
// 11 + 52 us, the write a thread per word with its pairs in turn.
#include "nans_kernels.cuh" // pair-space decode: nans_pairs.cuh

namespace nans
{

// Exclusive block scan of v; returns the prefix, writes the block total to *total.
__device__ __forceinline__ int block_exclusive_scan(int v, int *sh, int *total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = v;
    for (int o = 1; o < 32; o <<= 1)
    {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        sh[wid] = x;
    __syncthreads();
    if (wid == 0)
    {
        const int nw = blockDim.x >> 5;
        int t = (lane < nw) ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o)
                t += y;
        }
        if (lane < nw)
            sh[lane] = t;
    }
    __syncthreads();
    const int warp_prefix = (wid > 0) ? sh[wid - 1] : 0;
    *total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

// The mask word wo0 + lane of a warp's 32 words, one lane per pair at a time: the pairs' second boxes
// are read coalesced and a word is a ballot. Lane q first loads the scene data of word w0 + q and
// decodes its first pair (32 decodes side by side); the warp then walks its words with that data
// broadcast by shuffles.
__device__ __forceinline__ unsigned mask_words(const DevWorld &w, int wo, int lane, int all_pairs)
{
    const int w0 = wo - lane;
    int s = 0, nc = 0, ns = 0, c0 = 0, t0 = 0, i0 = 0, j0 = 0, cnt = 0;
    long long p0 = 0;
    if (wo < w.n_words)
    {
        s = __ldg(w.word_scene + wo);
        nc = __ldg(w.sc_nc + s);
        ns = __ldg(w.sc_ns + s);
        c0 = __ldg(w.sc_cube0 + s);
        p0 = (long long)(wo - __ldg(w.sc_word0 + s)) * 32;
        cnt = (int)min(32ll, scene_pair_count(nc, ns) - p0);
        decode_pair(p0, nc, ns, t0, i0, j0);
    }
    unsigned keep = 0u; // lane q keeps word w0 + q
    const int nq = min(32, w.n_words - w0);
    for (int q = 0; q < nq; ++q)
    {
        const int qcnt = __shfl_sync(0xffffffffu, cnt, q);
        const int qs = __shfl_sync(0xffffffffu, s, q);
        const int qnc = __shfl_sync(0xffffffffu, nc, q), qns = __shfl_sync(0xffffffffu, ns, q);
        const int qc0 = __shfl_sync(0xffffffffu, c0, q);
        const int qt = __shfl_sync(0xffffffffu, t0, q), qi = __shfl_sync(0xffffffffu, i0, q);
        const int qj = __shfl_sync(0xffffffffu, j0, q);
        const long long qp0 = __shfl_sync(0xffffffffu, p0, q);
        bool hit = false;
        if (lane < qcnt)
        {
            if (all_pairs)
                hit = true;
            else
            {
                int type, i, j, a, b;
                pair_after(qp0, qnc, qns, qt, qi, qj, lane, type, i, j);
                pair_ids(w, qs, qc0, qnc, type, i, j, a, b);
                const float4 la = __ldg(w.box_lo + a), ha = __ldg(w.box_hi + a);
                const float4 lb = __ldg(w.box_lo + b), hb = __ldg(w.box_hi + b);
                hit = la.x <= hb.x && lb.x <= ha.x && la.y <= hb.y && lb.y <= ha.y && la.z <= hb.z && lb.z <= ha.z;
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == q)
            keep = m;
    }
    return keep;
}

// ORs the row bits m (bit c = pair index base + c of the scene starting at bit wbit0) into the
// mask, from the first set bit on (so that no word before the scene's first is touched).
__device__ __forceinline__ void or_bits(unsigned *mask, long long wbit0, long long base, unsigned m)
{
    if (!m)
        return;
    const int c = __ffs(m) - 1;
    const long long b = wbit0 + base + c;
    m >>= c;
    const long long word = b >> 5;
    const int sh = (int)(b & 31);
    atomicOr(mask + word, m << sh);
    if (sh && (m >> (32 - sh)))
        atomicOr(mask + word + 1, m >> (32 - sh));
}

// A 32 x 32 tile of a scene's cube-cube pairs (rows i, columns j > i) by one warp: each lane holds one
// column's box and tests it against the rows' boxes from shared memory, a row's 32 tests are one
// ballot, and the row's bits are ORed into the mask at the row's pair indices (row i of the triangle
// is contiguous in j).
__device__ __forceinline__ void cull_tile(const DevWorld &w, int4 tile, float4 (*row)[2], int lane)
{
    const int s = tile.x, r0 = 32 * tile.y, k0 = 32 * tile.z;
    const int nc = __ldg(w.sc_nc + s), c0 = __ldg(w.sc_cube0 + s);
    const long long wbit0 = (long long)__ldg(w.sc_word0 + s) * 32;
    const int j = k0 + lane, ir = r0 + lane;
    float4 cl = make_float4(0.f, 0.f, 0.f, 0.f), ch = cl;
    if (j < nc)
    {
        cl = __ldg(w.box_lo + c0 + j);
        ch = __ldg(w.box_hi + c0 + j);
    }
    if (ir < nc)
    {
        row[lane][0] = __ldg(w.box_lo + c0 + ir);
        row[lane][1] = __ldg(w.box_hi + c0 + ir);
    }
    __syncwarp();
    const int rows = min(32, nc - r0);
    unsigned mine = 0u; // lane r: the bits of row r0 + r
#pragma unroll 4
    for (int r = 0; r < rows; ++r)
    {
        const float4 rl = row[r][0], rh = row[r][1];
        const bool hit = rl.x <= ch.x && cl.x <= rh.x && rl.y <= ch.y && cl.y <= rh.y && rl.z <= ch.z && cl.z <= rh.z;
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == r)
            mine = m;
    }
    __syncwarp(); // the rows' memory is the next tile's
    // columns beyond the scene's cubes, and in a diagonal tile those up to the row, are no pairs
    if (nc - k0 < 32)
        mine &= (1u << (nc - k0)) - 1u;
    if (tile.y == tile.z)
        mine &= ~((2u << lane) - 1u);
    if (lane < rows && mine)
    {
        const long long i = ir;
        // pair index of (i, k0): row i starts at i*nc - i*(i+1)/2 with column i + 1
        or_bits(w.pair_mask, wbit0, i * nc - i * (i + 1) / 2 + (k0 - i - 1), mine);
    }
}

// A task of the pairs that are not cube-cube: up to kRestChunksPerTask chunks of 32 consecutive pair
// indices of one scene (rest_tasks: scene, first chunk, chunks), so that a scene of many spheres
// (millions of cube-sphere pairs) spreads over the grid while a small scene is one task.
__device__ __forceinline__ void cull_rest(const DevWorld &w, int4 task, int lane)
{
    const int s = task.x;
    const int nc = __ldg(w.sc_nc + s), ns = __ldg(w.sc_ns + s), c0 = __ldg(w.sc_cube0 + s);
    const long long wbit0 = (long long)__ldg(w.sc_word0 + s) * 32;
    const long long np = scene_pair_count(nc, ns);
    const long long ncc = (long long)nc * (nc - 1) / 2;
    for (int q = 0; q < task.z; ++q)
    {
        const long long k0 = ncc + 32LL * (task.y + q);
        const long long k = k0 + lane;
        bool hit = false;
        if (k < np)
        {
            int type, i, j, a, b;
            decode_pair(k, nc, ns, type, i, j);
            pair_ids(w, s, c0, nc, type, i, j, a, b);
            const float4 la = __ldg(w.box_lo + a), ha = __ldg(w.box_hi + a);
            const float4 lb = __ldg(w.box_lo + b), hb = __ldg(w.box_hi + b);
            hit = la.x <= hb.x && lb.x <= ha.x && la.y <= hb.y && lb.y <= ha.y && la.z <= hb.z && lb.z <= ha.z;
        }
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0)
            or_bits(w.pair_mask, wbit0, k0, m);
    }
}

// The mask's bits (cleared before): one warp per tile, then per task of other pairs. The box test
// and the pair numbering are mask_words', so the mask is the same bit for bit. Bound by issue, six
// compares a row and lane at 30.6 of 32 lanes (94 us a step of 16,384 stacks, cold).
__global__ void __launch_bounds__(kCullTileThreads) k_cull_tiles(DevWorld w)
{
    __shared__ float4 rows[kCullTileThreads / 32][32][2];
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const long long n = (long long)w.n_tiles + w.n_rest_tasks;
    for (long long t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n; t += nwarps)
    {
        if (t < w.n_tiles)
            cull_tile(w, __ldg(w.tiles + t), rows[threadIdx.x >> 5], lane);
        else
            cull_rest(w, __ldg(w.rest_tasks + (t - w.n_tiles)), lane);
    }
}

// Block counts in cull_state: what is known of a block's candidates, its count or the count of all
// blocks up to it.
constexpr unsigned long long kStateCount = 1ull << 62, kStateTotal = 2ull << 62, kStateValue = (1ull << 62) - 1ull;
constexpr int kLookbackPolls = 1 << 20; // then the wait gives up (every earlier block is running: it does not)

// The candidates of the blocks before `block` (the calling warp; total = this block's). The blocks
// number themselves as they start, so every earlier one is running or done and its count will come.
__device__ __forceinline__ long long look_back(const DevWorld &w, int block, int total, int lane)
{
    volatile unsigned long long *st = w.cull_state;
    if (lane == 0)
        st[block] = (block == 0 ? kStateTotal : kStateCount) | (unsigned long long)total;
    long long before = 0;
    for (int last = block - 1; last >= 0; last -= 32)
    {
        const int k = last - lane;
        unsigned long long v = kStateTotal;
        for (int poll = 0; poll <= kLookbackPolls; ++poll)
        {
            if (k >= 0)
                v = st[k];
            if (__all_sync(0xffffffffu, (v >> 62) != 0))
                break;
            if (poll == kLookbackPolls && lane == 0)
                dev_check(w, false, 17, block, last);
            __nanosleep(20);
        }
        // the nearest block whose total is known, and the counts after it
        const unsigned known = __ballot_sync(0xffffffffu, (v >> 62) == 2);
        const int stop = known ? __ffs(known) - 1 : 31;
        long long x = lane <= stop ? (long long)(v & kStateValue) : 0;
        for (int o = 16; o > 0; o >>= 1)
            x += __shfl_xor_sync(0xffffffffu, x, o);
        before += x;
        if (known)
            break;
    }
    if (lane == 0 && block > 0)
        st[block] = kStateTotal | (unsigned long long)(before + total);
    return before;
}

// The culled pairs at their places (scene-major order). A block takes WPT words per thread; its set
// bits are listed in order in shared memory, then each thread decodes and writes one candidate at a
// time; a block of more than kCullList candidates does so in rounds. The last block writes the total
// and checks the capacity. MASK: the block makes its words itself. Bound by the scans' barriers and the
// look-back (37 us a step of 16,384 stacks, cold).
template <int WPT, bool MASK> __global__ void __launch_bounds__(kCullThreads) k_cull_place(DevWorld w, int all_pairs)
{
    __shared__ unsigned short list[kCullList]; // word of the block << 5 | bit
    __shared__ unsigned words[MASK ? WPT * kCullThreads : 1];
    __shared__ int sh[32];
    __shared__ int s_block;
    __shared__ long long s_before;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0)
        s_block = atomicAdd(w.work_counter + 1, 1);
    __syncthreads();
    const int block = s_block, w0 = block * WPT * kCullThreads;
    if (MASK)
    {
        for (int q = tid; q < WPT * kCullThreads; q += kCullThreads)
            words[q] = mask_words(w, w0 + q, lane, all_pairs);
        __syncthreads();
    }
    unsigned own[WPT]; // consecutive words
    int count = 0;
#pragma unroll
    for (int q = 0; q < WPT; ++q)
    {
        const int wo = w0 + WPT * tid + q;
        own[q] = MASK ? words[WPT * tid + q] : (wo < w.n_words ? w.pair_mask[wo] : 0u);
        count += __popc(own[q]);
    }
    int total;
    const int first = block_exclusive_scan(count, sh, &total);
    if (tid < 32)
    {
        const long long before = look_back(w, block, total, lane);
        if (lane == 0)
        {
            s_before = before;
            if (block == (int)gridDim.x - 1)
            {
                long long n = before + total;
                *w.cull_total = (int)min(n, (long long)INT32_MAX);
                *w.cull_max = max(*w.cull_max, *w.cull_total);
                if (n > w.cand_cap)
                {
                    atomicOr(w.status, (unsigned)ST_CANDIDATES);
                    n = w.cand_cap;
                }
                *w.n_cand = (int)n;
            }
        }
    }
    for (int round = 0; round < total; round += kCullList)
    {
        int at = first - round;
#pragma unroll
        for (int q = 0; q < WPT; ++q)
        {
            unsigned m = own[q];
            while (m)
            {
                const int bit = __ffs(m) - 1;
                m &= m - 1u;
                if (at >= 0 && at < kCullList)
                    list[at] = (unsigned short)(((WPT * tid + q) << 5) | bit);
                ++at;
            }
        }
        __syncthreads();
        const long long before = s_before + round;
        const int n = min(kCullList, total - round);
        for (int k = tid; k < n && before + k < w.cand_cap; k += kCullThreads)
        {
            const int e = list[k], we = w0 + (e >> 5), bit = e & 31;
            const int s = __ldg(w.word_scene + we);
            const int nc = __ldg(w.sc_nc + s), ns = __ldg(w.sc_ns + s), c0 = __ldg(w.sc_cube0 + s);
            int type, i, j, a, b;
            decode_pair((long long)(we - __ldg(w.sc_word0 + s)) * 32 + bit, nc, ns, type, i, j);
            pair_ids(w, s, c0, nc, type, i, j, a, b);
            const int pos = (int)before + k;
            w.cand_a[pos] = a;
            w.cand_b[pos] = b;
            w.cand_meta[pos] = (s << 3) | type;
            w.cand_pidx[pos] = we * 32 + bit;
        }
        __syncthreads();
    }
}

// Words per thread of the placement: one, so that a small world's candidates spread over more blocks,
// until the blocks no longer run side by side; then four, as more blocks would wait on each other's
// counts (38 against 61 us at 16,384 stacks' 2.0 M words; 28 against 16 at 18,000).
int cull_words_per_thread(int n_words, int sm_count) { return n_words > 8 * kCullThreads * sm_count ? 4 : 1; }

void launch_cull_place(const DevWorld &w, int mask, int all_pairs, cudaStream_t st)
{
    const bool four = cull_words_per_thread(w.n_words, w.sm_count) == 4;
    if (mask && four)
        k_cull_place<4, true><<<w.cull_blocks, kCullThreads, 0, st>>>(w, all_pairs);
    else if (mask)
        k_cull_place<1, true><<<w.cull_blocks, kCullThreads, 0, st>>>(w, all_pairs);
    else if (four)
        k_cull_place<4, false><<<w.cull_blocks, kCullThreads, 0, st>>>(w, all_pairs);
    else
        k_cull_place<1, false><<<w.cull_blocks, kCullThreads, 0, st>>>(w, all_pairs);
}

} // namespace nans
