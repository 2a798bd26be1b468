// Prefill attention for head size 64 on the 5th-generation tensor cores.
//
// Same result as prefill_mma_kernel (csrc/attention_mma.cu): causal attention of a step's query rows
// over their requests' pages (cached positions and the step's own), optionally with a window, by
// the online-softmax recurrence over tiles of keys (the reference computes the same sums with one
// thread block per query row and head, src/cuda/paged_attention.cu:230-337).  What differs is where the products
// run: a block owns 128 query rows of one head; per tile of 64 keys
//
//     S = Q K^T      tcgen05.mma, M = 128 (query rows = TMEM lanes), N = 64 keys, K = 64, into TMEM
//     P = exp2(..)   eight warps, half of a query row's 64 scores per thread, from TMEM with tcgen05.ld; P goes
//                    back into TMEM (tcgen05.st, two bfloat16 a column) as the next product's A operand
//     O_t = P V      tcgen05.mma with A in TMEM, N = 64, K = 64 keys, V read straight from its page
//                    layout [key][64] as an MN-major operand, accumulated into O in TMEM; the threads
//                    rescale O there only when a row's reference maximum has to move
//
// TMEM holds two score buffers and two P buffers (tile i uses buffer i & 1), so the products run a
// tile ahead of the softmax: the scores of tile i + 2 are issued when the softmax has read those of
// tile i, and the softmax of tile i + 1 finds its scores ready when it has written P of tile i.
//
// After a row's first tile the threads do not look for a tile's maximum first: they compute P against
// the reference as it is and find the maximum on the way; only if it lies more than 2^8 above the
// reference in some row of the warp does the reference move and the tile get walked again.  The two warps
// that share rows exchange their maxima through shared memory once a tile (a barrier of 64 threads), so both
// decide alike; a warp that has given up a wait still takes part in that barrier.
//
// TMEM allows two blocks an SM and a tile is a chain (scores, softmax, P, product), of which the softmax is the
// longest link: with four warps, a row a thread, 2330 of a tile's 3700 cycles.  With eight (us, 32 heads of 64 over 8): 2048 rows 54 -> 46,
// behind 6144 positions 258 -> 251, 8192 rows 543 -> 510; 16 heads, 32 rows behind 16 384 positions 76 -> 49.
//
// Shaped scores (`ZaiScoreOptions` in common.cuh) are an instantiation of their own: the cap by a tanh without a branch, the bias by distance
// from shared memory (a head's column of the table; neighbouring rows read neighbouring distances), the sink in the
// normalisation, kept first positions as tiles of their own ahead of the window's.  What bounds them is the shaping (a tile's
// 64 x 128 scores cost twice what its exponentials do).  Against the walk by mma.sync they take the place of (us, cap, bias and
// sink): 16 heads of 64 over 8, 2048 rows 164 -> 119, behind 6144 positions 630 -> 477, 8192 rows 1391 -> 870, 32 rows behind 16 384
// positions 684 -> 100; 32 heads, 2048 rows 299 -> 134; a window of 1024 with 4 kept positions, 2048 rows 97 -> 58.
// Their error against 64 bits is 0.93 to 1.00 of that walk's (relative 1.71e-3 to 2.10e-3, what bfloat16 P and results make it).
//
// Q, K and V reach shared memory by TMA (cp.async.bulk.tensor, no multicast), K and V page by page
// through the block table into five stages of 16 KB.  Roles: warp 0 one lane issues the loads (and the warp cleans the values of
// tiles that not every row sees whole), warp 1 one lane the products, warps 2-9 are the softmax.
//
// Blocks are handed out heads first, tiles of query rows from the last rows backwards: under the causal
// mask the last rows of a long span walk many more key tiles than the first, a block's tiles are a chain
// (scores, softmax, P, product), and the longest blocks of every head should start first.
// Every wait on an mbarrier is bounded; a block whose wait runs out raises the status word, its roles
// leave their loops, TMEM is freed and the block returns.
#include "attention_tc_helpers.cuh"

#define AT_D 64
#define AT_BM 128
#define AT_BN 64
#define AT_THREADS 320
#define AT_STAGES 5
#define AT_SHAPED_STAGES 4                            // (shaped scores: the bias by distance has the fifth's place, and more)
#define AT_Q_BYTES (AT_BM * AT_D * 2)                 // 16 KB
#define AT_KV_BYTES (2 * AT_BN * AT_D * 2)            // keys then values: 16 KB
#define AT_TMEM_COLS 256                              // two score buffers in columns 0..127, O in 128..191, two P buffers in 192..255
#define AT_COL_O (2 * AT_BN)
#define AT_COL_P (2 * AT_BN + AT_D)
#define AT_LAG 2                                      // tiles that the cleaning is behind the loads (below the number of stages)
typedef AtNotes<1, 128> AtTileNotes;

struct AtArgs {
    bf16* out;                  // [rows of the step, Hq, 64]
    const int* block_table;     // [S, table_width]
    const int* cu_q;            // [S + 1] first row of each request's span
    const int* ctx_lens;        // [S] positions cached before the step
    int* status;                // the step's status word: a wait that ran out, a page id outside the pool
    int num_pages;
    int table_width, S, page_size, page_shift, Hq, Hkv, window;
    float scale_log2;
    // With few tiles of query rows and long contexts, `splits` blocks (grid z) share a tile's key range; each
    // leaves its O [64][128], its rows' references and sums here, and the one that takes the last ticket of
    // the tile combines them (no block waits for another).
    int splits;
    float* part_o;              // [tiles of query rows x heads x splits][64][128]
    float* part_ml;             // [tiles of query rows x heads x splits][2][128]: reference (in the exponent's units), sum
    int* tickets;               // [tiles of query rows x heads], zero between launches
    ZaiScoreOptions opt;        // (shaped scores)
};

// tanh without a branch, so that a warp of mixed scores takes one way: the Taylor series up to x^9 below 0.3 (the next term is under
// 6e-8 of it there), the identity 1 - 2 / (1 + e^2x) beyond (a relative error of 4e-7 at most).
__device__ __forceinline__ float at_tanh(float x) {
    const float q = x * x;
    const float small = fmaf(x * q, fmaf(q, fmaf(q, fmaf(q, 62.f / 2835.f, -17.f / 315.f), 2.f / 15.f), -1.f / 3.f), x);
    const float large = 1.f - __fdividef(2.f, 1.f + at_exp2(x * 2.8853900817779268f));
    return fabsf(x) < 0.3f ? small : large;
}

// SHARED: several blocks (grid z) share a tile of query rows' keys; SHAPED: the scores pass `opt`
template <bool SHARED, bool SHAPED>
__global__ void __launch_bounds__(AT_THREADS, 2) prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                const __grid_constant__ CUtensorMap map_kv, const AtArgs a) {
    // All shared memory is dynamic and the tiles come first; with the system's 1 KB a block two blocks fit an SM's 233,472 bytes.
    constexpr int STAGES = SHAPED ? AT_SHAPED_STAGES : AT_STAGES;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = smem_raw;
    unsigned char* sQ = base;
    unsigned char* sKV = base + AT_Q_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + STAGES * AT_KV_BYTES);
    uint64_t& q_full = bars[0];
    uint64_t* kv_full = bars + 1;                               // [STAGES]
    uint64_t* kv_empty = bars + 1 + STAGES;                  // [STAGES]
    uint64_t* s_ready = bars + 1 + 2 * STAGES;               // [2] scores of tile i in buffer i & 1
    uint64_t* p_ready = bars + 3 + 2 * STAGES;               // [2] P of tile i in buffer i & 1
    uint64_t* o_ready = bars + 5 + 2 * STAGES;               // [2] the product of tile i has read P buffer i & 1 and added to O
    uint64_t* v_ready = bars + 7 + 2 * STAGES;               // [STAGES] the values of a stage are there and clean
    uint32_t& tmem_base_holder = *reinterpret_cast<uint32_t*>(bars + 7 + 3 * STAGES);
    int* words = reinterpret_cast<int*>(bars + 8 + 3 * STAGES);
    int& failed_flag = words[0];
    int& s_seq = words[1];
    int& s_i0 = words[2];
    float* exch = reinterpret_cast<float*>(words + 4);          // [2][2][128]: a tile's maxima by half, by turns; then the sums
    AtTileNotes& notes = *reinterpret_cast<AtTileNotes*>(exch + 4 * AT_BM);
    float* bias = reinterpret_cast<float*>(&notes + 1);         // [bias_rows] the head's bias by distance
    volatile int* failed = &failed_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        failed_flag = (at_smem(base) & 1023u) ? 1 : 0;          // the swizzled tiles need 1024-byte alignment
        notes.clear();
        at_mbar_init(&q_full, 1);
        for (int s = 0; s < STAGES; ++s) {
            at_mbar_init(&v_ready[s], 1);
            at_mbar_init(&kv_full[s], 1);
            at_mbar_init(&kv_empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            at_mbar_init(&s_ready[b], 1);
            at_mbar_init(&p_ready[b], 8);                       // one arrival per softmax warp
            at_mbar_init(&o_ready[b], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(at_smem(&tmem_base_holder)), "r"(AT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_holder;
    pdl_trigger();
    pdl_wait();
    if (tid == 0) {
        // Blocks are handed out x fastest, so the heads are x and the tiles of query rows y, numbered from
        // the last rows of the last request backwards: under the causal mask later rows have more keys
        // to walk, and the longest blocks of every head should start first
        int t = (int)gridDim.y - 1 - (int)blockIdx.y, s = 0;
        for (; s < a.S; ++s) {
            const int nt = (a.cu_q[s + 1] - a.cu_q[s] + AT_BM - 1) / AT_BM;
            if (t < nt) break;
            t -= nt;
        }
        s_seq = s;
        s_i0 = t * AT_BM;
    }
    const int h = blockIdx.x;
    __syncthreads();
    const int s = s_seq, i0 = s_i0;
    if (SHAPED && a.opt.bias) {
        // (as far as the block's rows reach; rows past the span's end read what is there; their scores are hidden)
        const int reach = s < a.S ? min(a.opt.bias_rows, a.ctx_lens[s] + min(a.cu_q[s + 1] - a.cu_q[s], i0 + AT_BM)) : 0;
        for (int i = tid; i < reach; i += AT_THREADS) bias[i] = a.opt.bias[(size_t)i * a.Hq + h] * 1.4426950408889634f;
        __syncthreads();
    }
    // the softmax threads' state, kept past the roles for a shared tile's combination
    float m = -INFINITY, l = 0.f;                               // m: the row's reference, in units of the scores
    bool have_o = false;                                        // the row's O in TMEM is complete
    int row0 = 0, rows = 0;
    if (s < a.S && !failed_flag) {
        const int hk = h / (a.Hq / a.Hkv);
        row0 = a.cu_q[s];
        const int q_len = a.cu_q[s + 1] - row0, ctx = a.ctx_lens[s];
        rows = min(AT_BM, q_len - i0);                              // valid query rows of this block
        const int kend = ctx + i0 + rows;                           // one past the last visible key of the block
        const int kbeg = zai_first_visible(ctx + i0, a.window);
        const int tile0 = kbeg / AT_BN, tile1 = (kend + AT_BN - 1) / AT_BN;
        // (kept first positions under a window: their tiles come first)
        const int n_kept = SHAPED && a.window > 0 ? min((min(a.opt.keep_first, zai_first_visible(kend - 1, a.window)) + AT_BN - 1) / AT_BN, tile0) : 0;
        int n_tiles = n_kept + tile1 - tile0, from = 0;
        if (SHARED) {                                               // this block's share of the key tiles
            const int per = (n_tiles + a.splits - 1) / a.splits;
            from = min((int)blockIdx.z * per, n_tiles);
            n_tiles = min(per, n_tiles - from);
        }
        auto key_of = [&](int i) { return (SHAPED && from + i < n_kept ? from + i : tile0 + from + i - n_kept) * AT_BN; };   // the first key of tile i
        // the tiles that some row does not see whole: those that end behind the first row (from tile p0 on, three at most; the last one
        // counts as such: when its values are ready, so are all), and those before the last row's first key that are not kept (p1 to p2)
        auto parts = [&](int& p0, int& p1, int& p2, int keep) {
            auto index_of = [&](int t) { return min(max((t < n_kept ? t : max(t, tile0) - tile0 + n_kept) - from, 0), n_tiles); };
            p0 = min(index_of((ctx + i0 + 1) / AT_BN), n_tiles - 1);
            p1 = index_of(keep / AT_BN);
            p2 = min(index_of((zai_first_visible(kend - 1, a.window) + AT_BN - 1) / AT_BN), p0);
        };

        if (warp == 0) {
            if (n_tiles > 0) {
                // ---- loads: the block's queries, then a stage of keys and values per tile, page by page
                const int* table = a.block_table + (size_t)s * a.table_width;
                const int ps = a.page_size, box_rows = ps < AT_BN ? ps : AT_BN, per_tile = AT_BN / box_rows;
                if (lane == 0) {
                    at_mbar_expect_tx(&q_full, AT_Q_BYTES);
                    at_tma_load_2d(sQ, &map_q, h * AT_D, row0 + i0, &q_full);
                }
                const int keep = SHAPED && a.window > 0 ? a.opt.keep_first : 0;
                int p0, p1, p2, issued = 0;
                parts(p0, p1, p2, keep);
                auto load = [&](int end) {                      // by one lane: the tiles up to `end`
                    for (; issued < end; ++issued) {
                        const int st = issued % STAGES;
                        if (!at_mbar_wait(&kv_empty[st], ((issued / STAGES) & 1) ^ 1, failed)) break;
                        at_mbar_expect_tx(&kv_full[st], AT_KV_BYTES);
                        unsigned char* dst = sKV + (size_t)st * AT_KV_BYTES;
                        for (int p = 0; p < per_tile; ++p) {
                            const int key0 = key_of(issued) + p * box_rows;
                            const int idx = key0 >> a.page_shift, off = key0 & (ps - 1);
                            int page = idx < a.table_width ? table[idx] : 0;          // beyond the table: the null page
                            if ((unsigned)page >= (unsigned)a.num_pages) {            // outside the pool: page 0, and the step is void
                                zai_raise(a.status, ZAI_ST_PAGE);
                                page = 0;
                            }
                            const int krow = ((page * 2 + 0) * a.Hkv + hk) * ps + off;
                            const int vrow = ((page * 2 + 1) * a.Hkv + hk) * ps + off;
                            at_tma_load_2d(dst + (size_t)p * box_rows * 128, &map_kv, 0, krow, &kv_full[st]);
                            at_tma_load_2d(dst + AT_BN * 128 + (size_t)p * box_rows * 128, &map_kv, 0, vrow, &kv_full[st]);
                        }
                        if (issued < p0 && (issued < p1 || issued >= p2)) at_mbar_arrive(&v_ready[st]);
                    }
                };
                auto clean = [&](int i) {                       // by the warp: the values of tile i
                    const int st = i % STAGES, tile_key = key_of(i);
                    if (!at_mbar_wait_warp(&kv_full[st], (i / STAGES) & 1, failed)) return false;
                    unsigned char* values = sKV + (size_t)st * AT_KV_BYTES + AT_KV_BYTES / 2;
                    const unsigned long long shown = at_below(kend - tile_key) & (~at_below(kbeg - tile_key) | at_below(keep - tile_key));
                    if (__any_sync(0xffffffffu, at_clean<4>(values, lane >> 3, shown)))
                        for (int k0 = 0; k0 < AT_BN; k0 += 4) {
                            const unsigned long long odd = at_take_odd(values, k0 + (lane >> 3), true);
                            if ((lane & 7) == 0 && odd) {
                                const int e = notes.add(tile_key + k0 + (lane >> 3));
                                if (e >= 0) notes.cols[e][0] = odd;
                            }
                        }
                    at_proxy_fence();                           // (generic writes, which the product reads)
                    __syncwarp();
                    if (lane == 0) at_mbar_arrive(&v_ready[st]);
                    return true;
                };
                // A window's first tiles with the loads AT_LAG tiles ahead of them, then all other loads by the one lane alone (with the warp
                // in step beside it a tile's load came a third later), then the last tiles, whose loads need none of their products
                bool ok = true;
                for (int i = p1; i < p2 && ok; ++i) {
                    if (lane == 0) load(min(i + AT_LAG + 1, n_tiles));
                    __syncwarp();
                    ok = clean(i);
                }
                if (lane == 0) load(n_tiles);
                __syncwarp();
                for (int i = p0; i < n_tiles && ok; ++i) ok = clean(i);
                if (lane == 0 && *failed) {                     // loads already issued still land here: wait for them
                    for (int i = max(issued - STAGES, 0); i < issued; ++i) {
                        const uint32_t addr = at_smem(&kv_full[i % STAGES]);
                        const uint32_t ph = (i / STAGES) & 1;
                        for (int spin = 0; spin < AT_SPIN_LIMIT; ++spin) {
                            uint32_t done;
                            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                                         : "=r"(done) : "r"(addr), "r"(ph) : "memory");
                            if (done) break;
                        }
                    }
                    const uint32_t addr = at_smem(&q_full);
                    for (int spin = 0; spin < AT_SPIN_LIMIT; ++spin) {
                        uint32_t done;
                        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                                     : "=r"(done) : "r"(addr), "r"(0u) : "memory");
                        if (done) break;
                    }
                }
            }
        } else if (warp == 1) {
            if (lane == 0 && n_tiles > 0) {
                // ---- products.  Instruction descriptors: D 32-bit, A and B bfloat16, M = 128, N = 64; the
                // scores have both operands K-major; O_t has A (P) in TMEM and B (the values) MN-major.
                constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AT_BN >> 3) << 17) | ((uint32_t)(AT_BM >> 4) << 24);
                constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(AT_D >> 3) << 17) |
                                             ((uint32_t)(AT_BM >> 4) << 24);
                const uint32_t tS = tmem_base, tO = tmem_base + AT_COL_O, tP = tmem_base + AT_COL_P;
                const uint32_t aQ = at_smem(sQ);
                bool ok = at_mbar_wait(&q_full, 0, failed);
                auto scores = [&](int i) {                      // S = Q K^T of tile i into score buffer i & 1
                    const int st = i % STAGES;
                    if (!at_mbar_wait(&kv_full[st], (i / STAGES) & 1, failed)) return false;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t aK = at_smem(sKV + (size_t)st * AT_KV_BYTES);
#pragma unroll
                    for (int k = 0; k < AT_D / 16; ++k)
                        at_umma(tS + (i & 1) * AT_BN, at_desc(aQ + k * 32), at_desc(aK + k * 32), idesc_s, k > 0 ? 1u : 0u);
                    at_commit(&s_ready[i & 1]);
                    return true;
                };
                // the scores run a tile ahead of the softmax: those of tile i + 2 are issued when the softmax
                // has read those of tile i (same buffer), so tile i + 1's are ready when the softmax of
                // tile i ends
                if (ok) ok = scores(0);
                if (ok && n_tiles > 1) ok = scores(1);
                auto product = [&](int i, bool wait) {          // O += P V of tile i, and the scores of tile i + 2; `wait`: its values are cleaned
                    const int st = i % STAGES;
                    ok = at_mbar_wait(&p_ready[i & 1], (i >> 1) & 1, failed) && (!wait || at_mbar_wait(&v_ready[st], (i / STAGES) & 1, failed));
                    if (!ok) return;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t aV = at_smem(sKV + (size_t)st * AT_KV_BYTES + AT_BN * 128);
#pragma unroll
                    for (int kk = 0; kk < AT_BN / 16; ++kk)     // 16 keys a step: eight columns of P, two groups of 8 keys of V
                        at_umma_ts(tO, tP + (i & 1) * (AT_BN / 2) + kk * 8, at_desc(aV + kk * 2048), idesc_o, (i > 0 || kk > 0) ? 1u : 0u);
                    at_commit(&o_ready[i & 1]);
                    at_commit(&kv_empty[st]);
                    if (i + 2 < n_tiles) ok = scores(i + 2);
                };
                int p0, p1, p2, i = 0;
                parts(p0, p1, p2, SHAPED && a.window > 0 ? a.opt.keep_first : 0);
                for (; i < p2 && ok; ++i) product(i, i >= p1);
                for (; i < p0 && ok; ++i) product(i, false);
                for (; i < n_tiles && ok; ++i) product(i, true);
            }
        } else if (n_tiles > 0) {
            // ---- softmax: thread = half of a query row (32 of a tile's 64 columns).  O stays in TMEM (the products add to
            // it); the row's reference maximum is only moved, and O and the sum rescaled, when a tile's maximum exceeds
            // it by more than 2^8 (P then stays below 256, exact enough in bfloat16 and 32-bit sums; the
            // result O / l does not depend on the reference).
            const int qd = warp & 3, half = (warp - 2) >> 2;    // this warp's quarter of the TMEM lanes, its half of the columns
            const int row = qd * 32 + lane;
            const bool valid = row < rows;
            const int qpos = ctx + i0 + row;                    // the row's position: keys 0..qpos are visible
            const int klo = zai_first_visible(qpos, a.window);
            const int kept = SHAPED && a.window > 0 ? min(a.opt.keep_first, klo) : 0;
            const uint32_t tS = tmem_base + ((uint32_t)(qd * 32) << 16) + half * 32, tO = tS + AT_COL_O, tP = tmem_base + ((uint32_t)(qd * 32) << 16) + AT_COL_P + half * 16;
            const float c = SHAPED ? 1.f : a.scale_log2;        // (shaped scores are made in the exponent's units)
            const float unit = SHAPED && a.opt.softcap > 0.f ? a.opt.scale / a.opt.softcap : 0.f, cap = a.opt.softcap * 1.4426950408889634f;
            bool alive = true;
            for (int i = 0; i < n_tiles; ++i) {
                const int key0 = key_of(i) + half * 32;
                if (alive && !at_mbar_wait_warp(&s_ready[i & 1], (i >> 1) & 1, failed)) alive = false;      // (the warp together)
                const uint32_t tSi = tS + (i & 1) * AT_BN, tPi = tP + (i & 1) * (AT_BN / 2);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                // keys of this half that the row sees: [lo, hi), and those below `first`
                const int lo = valid ? max(klo - key0, 0) : 32, hi = valid ? min(qpos + 1 - key0, 32) : 0;
                const int first = valid ? kept - key0 : 0;
                const bool full = lo <= 0 && hi >= 32;          // the row sees them all: no masking needed
                // the 32 scores, shaped and with the hidden ones at minus infinity
                auto load = [&](uint32_t (&x)[32]) {
                    at_tmem_ld32_nowait(tSi, x);
                    at_tmem_wait_ld(x);
                    if (SHAPED) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            float v = __uint_as_float(x[j]);
                            v = a.opt.softcap > 0.f ? cap * at_tanh(v * unit) : v * a.scale_log2;
                            if (a.opt.bias) v += bias[min(max(qpos - key0 - j, 0), a.opt.bias_rows - 1)];
                            x[j] = __float_as_uint(v);
                        }
                    }
                    if (!full) {
                        // (a hidden score may be anything, also NaN: it is replaced before the exponential)
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            if (!((j >= lo && j < hi) || (SHAPED && j < first))) x[j] = __float_as_uint(-INFINITY);
                    }
                };
                // one walk over them: their maximum (`mx`), and with `emit` the probabilities against `ref` into P and their sum (`lt`)
                auto walk = [&](const uint32_t (&x)[32], bool emit, float ref, float& mx, float& lt) {
                    float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, lt4[4] = {0.f, 0.f, 0.f, 0.f};   // four chains each, not one of 32 links
                    if (!emit) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], __uint_as_float(x[j]));
                    } else {
                        uint32_t pk[16];
#pragma unroll
                        for (int j = 0; j < 32; j += 2) {
                            const float s0 = __uint_as_float(x[j]), s1 = __uint_as_float(x[j + 1]);
                            mx4[(j >> 1) & 3] = fmaxf(mx4[(j >> 1) & 3], fmaxf(s0, s1));
                            const float p0 = at_exp2(s0 * c - ref), p1 = at_exp2(s1 * c - ref);
                            lt4[(j >> 1) & 3] += p0 + p1;
                            __nv_bfloat162 v = __floats2bfloat162_rn(p0, p1);
                            pk[j >> 1] = *reinterpret_cast<uint32_t*>(&v);
                        }
                        // (This P buffer was read by the product of the tile two before.  That product was issued
                        // before this tile's scores, and the commit behind the scores covers every product issued
                        // before it: the scores being ready says the buffer is free.)
                        at_tmem_st16(tPi, pk);                  // 32 keys = 16 columns of P
                    }
                    mx = fmaxf(mx, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])));
                    lt += (lt4[0] + lt4[1]) + (lt4[2] + lt4[3]);
                };
                // With a reference in every row of the warp, the tile is walked once against it; else the
                // maximum is found first, as a walk of its own.  Shaped scores are dear: they stay in registers, their maximum is
                // always found first, and the reference is the row's running maximum itself.
                uint32_t x[32];
                const bool speculate = !SHAPED && i > 0 && __all_sync(0xffffffffu, m != -INFINITY || !valid);
                float mx = -INFINITY, lt = 0.f;
                if (alive) {
                    load(x);
                    walk(x, speculate, m == -INFINITY ? 0.f : m * c, mx, lt);
                }
                // the row's maximum over both halves, which the two warps then decide by alike
                float* turn = exch + (i & 1) * (2 * AT_BM);
                turn[half * AT_BM + row] = mx;
                asm volatile("bar.sync %0, 64;" ::"r"(1 + qd) : "memory");
                mx = fmaxf(mx, turn[(half ^ 1) * AT_BM + row]);
                if (!alive) continue;                           // (this warp has given up; the other one must not wait for it)
                // move the reference?  (warp-wide decision: the TMEM accesses below are the whole warp's)
                float alpha = 1.f;
                if (m == -INFINITY) {
                    m = mx;                                     // nothing summed so far (O and l are 0, or this is the first tile)
                } else if (mx * c > m * c + (SHAPED ? 0.f : 8.f)) {
                    alpha = at_exp2(m * c - mx * c);
                    m = mx;
                }
                const bool moved = __any_sync(0xffffffffu, alpha != 1.f);
                float again = -INFINITY;
                if (SHAPED) walk(x, true, m == -INFINITY ? 0.f : m * c, again, lt);       // (before the rescaling: x is in registers no longer then)
                if (i > 0 && moved) {
                    if (!at_mbar_wait_warp(&o_ready[(i - 1) & 1], ((i - 1) >> 1) & 1, failed)) { alive = false; continue; }   // the product before (and with it all before) has added to O
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    uint32_t r[32];
                    at_tmem_ld32(tO, r);
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
                    at_tmem_st32(tO, r);
                    l *= alpha;
                }
                if (!SHAPED && (!speculate || moved)) {
                    lt = 0.f;
                    load(x);
                    walk(x, true, m == -INFINITY ? 0.f : m * c, again, lt);   // no key seen so far: every p is 0
                }
                l += lt;
                // P (and a rescaled O) are in TMEM before the product-issuing thread hears of it
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) at_mbar_arrive(&p_ready[i & 1]);
            }
            // the row's sum over both halves
            float* turn = exch + (n_tiles & 1) * (2 * AT_BM);
            turn[half * AT_BM + row] = l;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + qd) : "memory");
            l += turn[(half ^ 1) * AT_BM + row];
            if (alive && at_mbar_wait_warp(&o_ready[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, failed)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                have_o = at_mbar_wait_warp(&v_ready[(n_tiles - 1) % STAGES], ((n_tiles - 1) / STAGES) & 1, failed);    // (long since; the notes are seen)
                float inv = l > 0.f ? 1.f / l : 0.f;
                if (SHAPED && a.opt.sink) {                     // one more term of the denominator
                    const float M = m * c, sk = a.opt.sink[h] * 1.4426950408889634f, top = fmaxf(M, sk);
                    const float e = at_exp2(M - top);
                    inv = e / (l * e + at_exp2(sk - top));
                }
                bf16* dst = a.out + ((size_t)(row0 + i0 + row) * a.Hq + h) * AT_D + half * 32;
                if (!SHARED) {
                    uint32_t r[32];
                    at_tmem_ld32(tO, r);
                    if (valid) {
#pragma unroll
                        for (int d = 0; d < 32; d += 8) {
                            uint32_t v[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                __nv_bfloat162 p = __floats2bfloat162_rn(__uint_as_float(r[d + 2 * e]) * inv, __uint_as_float(r[d + 2 * e + 1]) * inv);
                                v[e] = *reinterpret_cast<uint32_t*>(&p);
                            }
                            *reinterpret_cast<uint4*>(dst + d) = make_uint4(v[0], v[1], v[2], v[3]);
                        }
                        if (notes.count) notes.put_nans(dst, 1, half, 1, qpos, klo, kept);
                    }
                }
            }
        }
    }
    if (SHARED && s < a.S && warp >= 2) {
        // ---- a shared tile of query rows: this block's part into memory, a ticket, and the last one combines
        const int qd = warp & 3, half = (warp - 2) >> 2, row = qd * 32 + lane;
        const uint32_t tO = tmem_base + ((uint32_t)(qd * 32) << 16) + AT_COL_O + half * 32;
        const int slot = ((int)gridDim.y - 1 - (int)blockIdx.y) * a.Hq + h;
        const size_t mine = (size_t)slot * a.splits + blockIdx.z;
        float* po = a.part_o + mine * (AT_D * AT_BM) + half * 32 * AT_BM;
        float* pml = a.part_ml + mine * (2 * AT_BM);
        const bool ok = have_o && !failed_flag;                 // (a block without key tiles, or one that gave up, has no part)
        if (half == 0) {
            pml[row] = (ok && m != -INFINITY) ? m * (SHAPED ? 1.f : a.scale_log2) : -INFINITY;
            pml[AT_BM + row] = ok ? l : 0.f;
        }
        if (ok) {
            uint32_t r[32];
            at_tmem_ld32(tO, r);
#pragma unroll
            for (int j = 0; j < 32; ++j) po[j * AT_BM + row] = __uint_as_float(r[j]);
            if (notes.count) {
                const int qpos = a.ctx_lens[s] + i0 + row, klo = zai_first_visible(qpos, a.window);
                notes.put_nans(po + row, AT_BM, half, 1, qpos, klo, SHAPED && a.window > 0 ? min(a.opt.keep_first, klo) : 0);
            }
        }
        asm volatile("bar.sync 5, 256;" ::: "memory");          // the eight softmax warps
        if (tid == 64) {
            __threadfence();                                    // (one fence behind the barrier: it is cumulative)
            s_seq = atomicAdd(a.tickets + slot, 1);
        }
        asm volatile("bar.sync 5, 256;" ::: "memory");
        if (s_seq == a.splits - 1) {
            __threadfence();
            float top = -INFINITY, sum = 0.f, acc[32];
#pragma unroll
            for (int d = 0; d < 32; ++d) acc[d] = 0.f;
            for (int z = 0; z < a.splits; ++z) {
                const size_t other = (size_t)slot * a.splits + z;
                const volatile float* qml = a.part_ml + other * (2 * AT_BM);
                const float mz = qml[row], lz = qml[AT_BM + row];
                if (mz == -INFINITY) continue;                  // nothing from this part (its O may be unwritten)
                const float ntop = fmaxf(top, mz);
                const float f_old = top == -INFINITY ? 0.f : at_exp2(top - ntop), f_new = at_exp2(mz - ntop);
                const volatile float* qo = a.part_o + other * (AT_D * AT_BM) + half * 32 * AT_BM;
                sum = sum * f_old + lz * f_new;
#pragma unroll
                for (int d = 0; d < 32; ++d) acc[d] = acc[d] * f_old + qo[d * AT_BM + row] * f_new;
                top = ntop;
            }
            float inv = sum > 0.f ? 1.f / sum : 0.f;
            if (SHAPED && a.opt.sink) {
                const float sk = a.opt.sink[h] * 1.4426950408889634f, most = fmaxf(top, sk), e = at_exp2(top - most);
                inv = e / (sum * e + at_exp2(sk - most));
            }
            if (row < rows) {
                bf16* dst = a.out + ((size_t)(row0 + i0 + row) * a.Hq + h) * AT_D + half * 32;
#pragma unroll
                for (int d = 0; d < 32; d += 8) {
                    uint32_t v[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        __nv_bfloat162 p = __floats2bfloat162_rn(acc[d + 2 * e] * inv, acc[d + 2 * e + 1] * inv);
                        v[e] = *reinterpret_cast<uint32_t*>(&p);
                    }
                    *reinterpret_cast<uint4*>(dst + d) = make_uint4(v[0], v[1], v[2], v[3]);
                }
            }
            if (tid == 64) a.tickets[slot] = 0;                 // ready for the next launch
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(AT_TMEM_COLS) : "memory");
    }
    if (tid == 0 && failed_flag) zai_raise(a.status, ZAI_ST_WAIT);
}

// ------------------------------------------------------------------------------------------ host side
// 1 if this kernel takes the sizes: head size 64, a page size that is a power of two from 8 to 128 (a tile
// of 64 keys is loaded page by page, or as half of a page of 128)
ZAI_API int zai_prefill_attention_tc_supports(int D, int Hq, int Hkv, int page_size) {
    if (D != AT_D || Hkv < 1 || Hq % Hkv != 0 || Hq > 32767) return 0;
    if (page_size < 8 || page_size > 128 || (page_size & (page_size - 1))) return 0;
    return at_encode_tiled() != nullptr;
}

#define AT_MAX_BIAS 7168
ZAI_API int zai_prefill_attention_tc_max_bias() { return AT_MAX_BIAS; }

// How many blocks should share a tile of query rows' keys: 1 when the tiles alone fill the SMs (two blocks
// each) or the contexts are short; else enough to fill them, with at least eight key tiles for each at the
// longest context a block-table row holds, and 16 at most.  Shaped scores make a tile twice as long: three suffice there.
static int at_splits(int n_tiles, int Hq, int table_width, int page_size, int least) {
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) sms = n;
        else sms = 148;
    }
    const long long blocks = (long long)n_tiles * Hq, places = 2LL * sms;
    if (blocks <= 0 || 2 * blocks > places) return 1;
    long long want = (places + blocks - 1) / blocks;
    const long long key_tiles = ((long long)table_width * page_size + AT_BN - 1) / AT_BN;
    const long long most = key_tiles / least;
    if (want > most) want = most;
    if (want > 16) want = 16;
    return want < 2 ? 1 : (int)want;
}
ZAI_API int zai_prefill_attention_tc_splits(int n_tiles, int Hq, int table_width, int page_size) {
    return at_splits(n_tiles, Hq, table_width, page_size, 8);
}
ZAI_API int zai_prefill_attention_tc_shaped_splits(int n_tiles, int Hq, int table_width, int page_size) {
    return at_splits(n_tiles, Hq, table_width, page_size, 3);
}

// out [N, Hq, 64] = attention of q [N, Hq, 64] (N rows in all, `n_tiles` blocks of 128 rows over the
// requests' spans) over the pages [num_pages, 2, Hkv, page_size, 64]; arguments as
// zai_prefill_attention_mma, plus the row and page counts and the status word that a block raises
// if one of its waits ran out or a page id lay outside the pool.  With splits > 1 (zai_prefill_attention_tc_splits
// proposes a number) the caller gives the scratch for the parts: part_o [n_tiles * Hq * splits * 64 * 128]
// and part_ml [n_tiles * Hq * splits * 2 * 128] floats, and tickets [n_tiles * Hq] ints that are zero.  The score options (see
// ZaiScoreOptions; all off: zeros and null pointers) go with a bias of at most zai_prefill_attention_tc_max_bias() rows.
ZAI_API int zai_prefill_attention_tc(void* out, const void* q, const void* pages, int num_pages, int* status,
                                     const int* block_table, int table_width, const int* cu_q, const int* ctx_lens, int N,
                                     int S, int n_tiles, int page_size, int Hq, int Hkv, int D, float scale, int window,
                                     int splits, float* part_o, float* part_ml, int* tickets, float softcap, const float* bias,
                                     int bias_rows, const float* sink, int keep_first, cudaStream_t stream) {
    if (N <= 0 || S <= 0 || n_tiles <= 0) return ZAI_OK;
    if (!zai_prefill_attention_tc_supports(D, Hq, Hkv, page_size) || n_tiles > 65535) return ZAI_BAD_SIZE;
    if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(pages) | reinterpret_cast<uintptr_t>(out)) & 15) return ZAI_BAD_SIZE;
    CUtensorMap mq, mkv;
    int e = at_make_map(&mq, q, (cuuint64_t)Hq * AT_D, (cuuint64_t)N, AT_BM);
    if (e) return e;
    e = at_make_map(&mkv, pages, AT_D, (cuuint64_t)num_pages * 2 * Hkv * page_size, (cuuint32_t)(page_size < AT_BN ? page_size : AT_BN));
    if (e) return e;
    AtArgs a;
    a.out = (bf16*)out; a.block_table = block_table; a.cu_q = cu_q; a.ctx_lens = ctx_lens; a.status = status; a.num_pages = num_pages;
    a.table_width = table_width; a.S = S; a.page_size = page_size; a.Hq = Hq; a.Hkv = Hkv; a.window = window;
    a.scale_log2 = scale * 1.4426950408889634f;
    if (splits < 1 || splits > 64 || (splits > 1 && (!part_o || !part_ml || !tickets))) return ZAI_BAD_SIZE;
    a.splits = splits; a.part_o = part_o; a.part_ml = part_ml; a.tickets = tickets;
    a.page_shift = 0;
    while ((1 << a.page_shift) < page_size) ++a.page_shift;
    const bool shaped = softcap > 0.f || bias || sink || keep_first > 0;
    a.opt = {softcap, bias, bias_rows, sink, keep_first, scale};
    constexpr size_t words = 256 + 4 * AT_BM * sizeof(float) + sizeof(AtTileNotes);
    constexpr size_t smem = AT_Q_BYTES + (size_t)AT_STAGES * AT_KV_BYTES + words;
    constexpr size_t smem_shaped = AT_Q_BYTES + (size_t)AT_SHAPED_STAGES * AT_KV_BYTES + words;
    static_assert(2 * (smem + 1024) <= 233472 && 2 * (smem_shaped + AT_MAX_BIAS * sizeof(float) + 1024) <= 233472, "two blocks an SM");
    static unsigned long long configured = 0;
    if (zai_first_on_device(&configured)) {
        // two blocks per SM: ask for the largest shared-memory carve-out
        auto set = [](const void* f, size_t bytes) {
            cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
            if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
            return e;
        };
        cudaError_t err = set((const void*)prefill_tc_kernel<false, false>, smem);
        if (err == cudaSuccess) err = set((const void*)prefill_tc_kernel<true, false>, smem);
        if (err == cudaSuccess) err = set((const void*)prefill_tc_kernel<true, true>, smem_shaped + AT_MAX_BIAS * sizeof(float));
        if (err == cudaSuccess) err = set((const void*)prefill_tc_kernel<false, true>, smem_shaped + AT_MAX_BIAS * sizeof(float));
        if (err != cudaSuccess) return (int)err;
    }
    if (shaped) {
        if (softcap < 0.f || keep_first < 0 || (keep_first && window <= 0) || (bias && (bias_rows < 1 || bias_rows > AT_MAX_BIAS))) return ZAI_BAD_SIZE;
        if (splits > 1)
            return launch_pdl(prefill_tc_kernel<true, true>, dim3(Hq, n_tiles, splits), dim3(AT_THREADS), smem_shaped + (bias ? bias_rows * sizeof(float) : 0),
                              stream, mq, mkv, a);
        return launch_pdl(prefill_tc_kernel<false, true>, dim3(Hq, n_tiles), dim3(AT_THREADS), smem_shaped + (bias ? bias_rows * sizeof(float) : 0), stream,
                          mq, mkv, a);
    }
    if (splits > 1) return launch_pdl(prefill_tc_kernel<true, false>, dim3(Hq, n_tiles, splits), dim3(AT_THREADS), smem, stream, mq, mkv, a);
    return launch_pdl(prefill_tc_kernel<false, false>, dim3(Hq, n_tiles), dim3(AT_THREADS), smem, stream, mq, mkv, a);
}
