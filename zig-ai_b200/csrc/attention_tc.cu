// Prefill attention for head size 64 on the 5th-generation tensor cores.
//
// Same result as prefill_mma_kernel (csrc/attention_mma.cu): causal attention of a step's query rows
// over their requests' pages (cached positions and the step's own), optionally with a window, by
// the online-softmax recurrence over tiles of keys (the reference computes the same sums with one
// thread block per query row and head, src/cuda/paged_attention.cu:230-337).  What differs is where the products
// run: a block owns 128 query rows of one head; per tile of 64 keys
//
//     S = Q K^T      tcgen05.mma, M = 128 (query rows = TMEM lanes), N = 64 keys, K = 64, into TMEM
//     P = exp2(..)   four warps, a query row a thread, from TMEM with tcgen05.ld; P goes back into TMEM (tcgen05.st, two
//                    bfloat16 a column) as the next product's A operand
//     O += P V       tcgen05.mma with A in TMEM, N = 64, K = 64 keys, V read straight from its page
//                    layout [key][64] as an MN-major operand; the threads rescale O there only when a row's reference moves
//
// Eight softmax warps take the tiles by turns, four the even ones and four the odd ones, each turn with a score buffer and a
// P buffer: tile i + 1 is in the softmax of the other turn while tile i's P is multiplied and tile i + 2's scores are made.
// A product is issued as soon as what it needs is there, in whatever order that comes.
//
// What bounds it: of a turn's 2900 cycles a tile, 1100 are exponentials and packing (512 of them the special-function unit's for
// one warp), 700 the scores' load and maximum, the rest waits and what goes with them; two blocks an SM (TMEM allows no more)
// run beside each other.  us, 32 heads of 64 over 8, 2048 rows behind 6144 positions: 271 with half a row a thread and the two
// halves' maxima exchanged every tile, 243 with a row a thread and products issued by one lane behind `lane == 0`, 212 now.
//
// Shaped scores (`ZaiScoreOptions` in common.cuh) are an instantiation of their own: the cap by a tanh without a branch, the bias by distance
// from shared memory (a head's column of the table; neighbouring rows read neighbouring distances), the sink in the
// normalisation, kept first positions as tiles of their own ahead of the window's.  What bounds them is the shaping (a tile's
// scores cost four times what its exponentials do); it takes two numbers an instruction (fma.rn.f32x2).  16 heads of 64 over 4,
// 2048 rows, cap, bias and sink: 103 -> 90 us.  Before that, against the walk by mma.sync (us, cap, bias and sink): 16 heads of 64 over
// 8, 2048 rows 164 -> 119, behind 6144 positions 630 -> 477, 8192 rows 1391 -> 870, 32 rows behind 16 384 positions 684 -> 100;
// 32 heads, 2048 rows 299 -> 134; a window of 1024 with 4 kept positions, 2048 rows 97 -> 58.
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
#include <type_traits>

#include "attention_tc_helpers.cuh"

#define AT_D 64
#define AT_BM 128
#define AT_BN 64
#define AT_THREADS 320
#define AT_STAGES 5
#define AT_SHAPED_STAGES 4                            // (shaped scores: the bias by distance has the fifth's place, and more)
#define AT_Q_BYTES (AT_BM * AT_D * 2)                 // 16 KB
#define AT_KV_BYTES (2 * AT_BN * AT_D * 2)            // keys then values: 16 KB
#define AT_TMEM_COLS 256                              // two score buffers in columns 0..127, O in 128..191, two P buffers in 192..255; shaped
                                                      // scores: P in the first half of its scores' columns, a second O in 192..255
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

// two 32-bit numbers in one instruction
__device__ __forceinline__ float2 at_fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)), "l"(reinterpret_cast<unsigned long long&>(c)));
    return d;
}
__device__ __forceinline__ float2 at_mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return d;
}
__device__ __forceinline__ float2 at_add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return d;
}
__device__ __forceinline__ uint32_t at_pack(float2 v) {
    __nv_bfloat162 p = __floats2bfloat162_rn(v.x, v.y);
    return *reinterpret_cast<uint32_t*>(&p);
}
__device__ __forceinline__ float2 at_two(float v) { return make_float2(v, v); }
__device__ __forceinline__ float at_max3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
// tanh of two numbers without a branch, so that a warp of mixed scores takes one way: the Taylor series up to x^9 below 0.3 (the next
// term is under 6e-8 of it there), the identity 1 - 2 / (1 + e^2x) beyond (a relative error of 4e-7 at most).
__device__ __forceinline__ float2 at_tanh2(float2 x) {
    const float2 q = at_mul2(x, x);
    float2 small = at_fma2(q, at_two(62.f / 2835.f), at_two(-17.f / 315.f));
    small = at_fma2(q, small, at_two(2.f / 15.f));
    small = at_fma2(q, small, at_two(-1.f / 3.f));
    small = at_fma2(at_mul2(x, q), small, x);
    const float2 z = at_mul2(x, at_two(2.8853900817779268f));
    const float2 d = at_add2(make_float2(at_exp2(z.x), at_exp2(z.y)), at_two(1.f));
    const float2 large = at_fma2(make_float2(__fdividef(1.f, d.x), __fdividef(1.f, d.y)), at_two(-2.f), at_two(1.f));
    return make_float2(fabsf(x.x) < 0.3f ? small.x : large.x, fabsf(x.y) < 0.3f ? small.y : large.y);
}

// A row's reference on its way from the warp that has tile i to the one with its rows in tile i + 1: a barrier of 64 threads, of which
// the one side arrives and goes on
__device__ __forceinline__ void at_pass_on(int qd, int i) { asm volatile("bar.arrive %0, 64;" ::"r"(2 + qd * 2 + (i & 1)) : "memory"); }
__device__ __forceinline__ void at_pass_wait(int qd, int i) { asm volatile("bar.sync %0, 64;" ::"r"(2 + qd * 2 + (i & 1)) : "memory"); }

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
    uint64_t* s_empty = bars + 5 + 2 * STAGES;               // [2] the scores of buffer i & 1 have been read
    uint64_t* v_ready = bars + 7 + 2 * STAGES;               // [STAGES] the values of a stage are there and clean
    uint32_t& tmem_base_holder = *reinterpret_cast<uint32_t*>(bars + 7 + 3 * STAGES);
    int* words = reinterpret_cast<int*>(bars + 8 + 3 * STAGES);
    int& failed_flag = words[0];
    int& s_seq = words[1];
    int& s_i0 = words[2];
    float* exch = reinterpret_cast<float*>(words + 4);          // [2][2][128]: the references by turn (even, odd tiles), then the sums
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
            at_mbar_init(&p_ready[b], 4);                       // one arrival per softmax warp of the tile
            at_mbar_init(&s_empty[b], 4);
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
    float m = -INFINITY, l = 0.f;                               // m: the row's reference, in the exponent's units
    bool have_o = false;                                        // the row's O is complete
    float out[32];                                              // ... a half of it
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
                        if (!at_mbar_wait<AT_NAP_NS>(&kv_empty[st], ((issued / STAGES) & 1) ^ 1, failed)) break;
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
            if (n_tiles > 0 && zai_elect()) {
                // ---- products.  (By the lane that elect.sync picks: the compiler then knows that one lane is left and issues a product in
                // half the time that it takes behind `lane == 0`, where a tile's eight products and three commits took 2000 cycles,
                // more than its softmax.)
                // Instruction descriptors: D 32-bit, A and B bfloat16, M = 128, N = 64; the scores have both operands K-major; O has
                // A (P) in TMEM and B (the values) MN-major.
                constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AT_BN >> 3) << 17) | ((uint32_t)(AT_BM >> 4) << 24);
                constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(AT_D >> 3) << 17) |
                                             ((uint32_t)(AT_BM >> 4) << 24);
                const uint32_t tS = tmem_base, tO = tmem_base + AT_COL_O, tP = tmem_base + AT_COL_P;
                const uint32_t aQ = at_smem(sQ);
                int p0, p1, p2;
                parts(p0, p1, p2, SHAPED && a.window > 0 ? a.opt.keep_first : 0);
                bool ok = at_mbar_wait(&q_full, 0, failed);
                // A stage's release is also what says that its product, and all before it, are in O.
                auto scores = [&](int i) {
                    const uint32_t aK = at_smem(sKV + (size_t)(i % STAGES) * AT_KV_BYTES);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int k = 0; k < AT_D / 16; ++k)
                        at_umma(tS + (i & 1) * AT_BN, at_desc(aQ + k * 32), at_desc(aK + k * 32), idesc_s, k > 0 ? 1u : 0u);
                    at_commit(&s_ready[i & 1]);
                };
                auto product = [&](int i) {
                    const uint32_t aV = at_smem(sKV + (size_t)(i % STAGES) * AT_KV_BYTES + AT_BN * 128);
                    const uint32_t d = SHAPED ? tO + (i & 1) * AT_D : tO, p = SHAPED ? tS + (i & 1) * AT_BN : tP + (i & 1) * (AT_BN / 2);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int kk = 0; kk < AT_BN / 16; ++kk)     // 16 keys a step: eight columns of P, two groups of 8 keys of V
                        at_umma_ts(d, p + kk * 8, at_desc(aV + kk * 2048), idesc_o, (i > (SHAPED ? 1 : 0) || kk > 0) ? 1u : 0u);
                };
                auto cleaned = [&](int i) { return i >= p0 || (i >= p1 && i < p2); };
                if (SHAPED && n_tiles == 1) {
                    // a tile alone: the turns have half of its keys each, for an O each
                    if (ok) ok = at_mbar_wait(&kv_full[0], 0, failed);
                    if (ok) scores(0);
                    if (ok) ok = at_mbar_wait(&v_ready[0], 0, failed) && at_mbar_wait(&p_ready[0], 0, failed) && at_mbar_wait(&p_ready[1], 0, failed);
                    if (ok) {
                        const uint32_t aV = at_smem(sKV + AT_BN * 128);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                        for (int kk = 0; kk < AT_BN / 16; ++kk)
                            at_umma_ts(tO + (kk >> 1) * AT_D, tS + (kk >> 1) * 32 + (kk & 1) * 8, at_desc(aV + kk * 2048), idesc_o, kk & 1);
                        at_commit(&kv_empty[0]);
                    }
                } else if (SHAPED) {
                    // P lies over its scores, so the scores of tile i + 2 are issued behind the product of tile i (products of one
                    // thread run in order); the other turn's tile i + 1 is in the softmax meanwhile
#pragma unroll 1
                    for (int i = -2; i < n_tiles && ok; ++i) {
                        if (i >= 0) {
                            ok = (!cleaned(i) || at_mbar_wait(&v_ready[i % STAGES], (i / STAGES) & 1, failed)) && at_mbar_wait(&p_ready[i & 1], (i >> 1) & 1, failed);
                            if (ok) product(i);
                        }
                        if (ok && i + 2 < n_tiles) {
                            ok = at_mbar_wait(&kv_full[(i + 2) % STAGES], ((i + 2) / STAGES) & 1, failed);
                            if (ok) scores(i + 2);
                        }
                        if (ok && i >= 0) at_commit(&kv_empty[i % STAGES]);
                    }
                } else {
                    // Scores as soon as their buffer has been read, products as soon as their P is there, whichever comes first (in a
                    // fixed order each waited for the other turn's warps: a turn took 3000 cycles)
                    int s_at = 0, p_at = 0;
                    for (int spin = 0; p_at < n_tiles && ok; ++spin) {
                        if (s_at < n_tiles && at_mbar_test(&kv_full[s_at % STAGES], (s_at / STAGES) & 1)
                            && (s_at < 2 || at_mbar_test(&s_empty[s_at & 1], ((s_at - 2) >> 1) & 1))) {
                            scores(s_at++);
                            spin = 0;
                        }
                        if (at_mbar_test(&p_ready[p_at & 1], (p_at >> 1) & 1)
                            && (!cleaned(p_at) || at_mbar_test(&v_ready[p_at % STAGES], (p_at / STAGES) & 1))) {
                            product(p_at);
                            at_commit(&kv_empty[p_at++ % STAGES]);
                            spin = 0;
                        }
                        if (spin >= AT_SPIN_LIMIT) *failed = 1;
                        if (spin > 0 && *failed) ok = false;
                    }
                }
            }
        } else if (n_tiles > 0) {
            // ---- softmax: thread = a query row; four warps have the even tiles, four the odd ones.  O stays in TMEM (the products add
            // to it); a row's reference is only moved, and O and the sums rescaled, when a tile's maximum exceeds it by more than
            // 2^8 (P then stays below 256, exact enough in bfloat16 and 32-bit sums; the result O / l does not depend on the
            // reference).  The reference goes from tile to tile through shared memory, so from one turn's warp to the other's,
            // early in a tile.  Shaped scores have the running maximum as their reference, which moves in most tiles: there each
            // turn has a reference, a sum and an O of its own.
            const int qd = warp & 3, turn = (warp - 2) >> 2;    // this warp's quarter of the TMEM lanes, the tiles it has
            const int row = qd * 32 + lane;
            const bool valid = row < rows;
            const int qpos = ctx + i0 + row;                    // the row's position: keys 0..qpos are visible
            const int klo = zai_first_visible(qpos, a.window);
            const int kept = SHAPED && a.window > 0 ? min(a.opt.keep_first, klo) : 0;
            const uint32_t lanes = tmem_base + ((uint32_t)(qd * 32) << 16), tS = lanes + turn * AT_BN, tO = lanes + AT_COL_O + (SHAPED ? turn * AT_D : 0),
                           tPlain = lanes + AT_COL_P + turn * (AT_BN / 2);
            const float c = SHAPED ? 1.f : a.scale_log2;        // (shaped scores are made in the exponent's units)
            const float unit = SHAPED && a.opt.softcap > 0.f ? a.opt.scale / a.opt.softcap : 0.f, cap = a.opt.softcap * 1.4426950408889634f;
            bool alive = true;
            // tile i's keys from key0 on (64 of them, or 32), whose scores come into column tSc
            auto tile = [&](int i, int key0, uint32_t tSc, uint64_t* scores_ready, auto keys_of) {
                constexpr int KEYS = decltype(keys_of)::value;
                const uint32_t tP = SHAPED ? tSc : tPlain;
                if (alive) alive = at_mbar_wait_warp(scores_ready, (i >> 1) & 1, failed);   // (the warp together)
                if (!alive) {                                   // (the other turn's warps still wait for this one's word)
                    if (SHAPED) return;
                    if (i > 0) at_pass_wait(qd, i - 1);
                    if (i + 1 < n_tiles) at_pass_on(qd, i);
                    return;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t x[KEYS / 32][32];
#pragma unroll
                for (int j = 0; j < KEYS / 32; ++j) at_tmem_ld32_nowait(tSc + j * 32, x[j]);
#pragma unroll
                for (int j = 0; j < KEYS / 32; ++j) at_tmem_wait_ld(x[j]);
                if (!SHAPED) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    if (lane == 0) at_mbar_arrive(&s_empty[turn]);
                }
                if (SHAPED) {
                    const int far = qpos - key0, last = a.opt.bias_rows - 1;
                    // a distance below zero is a hidden key's (what it reads lies in this block's shared memory); beyond the
                    // table its last entry counts.  Most tiles lie on one side of that for the whole warp.
                    const bool near = __all_sync(0xffffffffu, far <= last);
                    const float* from = bias + far;
                    auto shape = [&](auto entry) {
#pragma unroll
                        for (int j = 0; j < KEYS; j += 2) {
                            float2 v = make_float2(__uint_as_float(x[j >> 5][j & 31]), __uint_as_float(x[j >> 5][(j & 31) + 1]));
                            const float2 add = make_float2(entry(j), entry(j + 1));
                            v = a.opt.softcap > 0.f ? at_fma2(at_tanh2(at_mul2(v, at_two(unit))), at_two(cap), add) : at_fma2(v, at_two(a.scale_log2), add);
                            x[j >> 5][j & 31] = __float_as_uint(v.x);
                            x[j >> 5][(j & 31) + 1] = __float_as_uint(v.y);
                        }
                    };
                    if (!a.opt.bias) shape([](int) { return 0.f; });
                    else if (near) shape([&](int j) { return from[-j]; });
                    else shape([&](int j) { return bias[min(max(far - j, 0), last)]; });
                }
                // keys that the row sees: [lo, hi), and those below `first`
                const int lo = valid ? max(klo - key0, 0) : KEYS, hi = valid ? min(qpos + 1 - key0, KEYS) : 0;
                const int first = valid ? kept - key0 : 0;
                if (__any_sync(0xffffffffu, lo > 0 || hi < KEYS)) {                     // (the warp's branch: no tile without it pays for its instructions)
                    // (a hidden score may be anything, also NaN: it is replaced before the exponential)
                    const unsigned long long seen = (at_below(hi) & ~at_below(lo)) | (SHAPED ? at_below(first) : 0ull);
                    const uint32_t some[2] = {(uint32_t)seen, (uint32_t)(seen >> 32)};
#pragma unroll
                    for (int j = 0; j < KEYS; ++j)
                        if (!(some[j >> 5] >> (j & 31) & 1)) x[j >> 5][j & 31] = __float_as_uint(-INFINITY);
                }
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};            // four chains, not one of 32 links
#pragma unroll
                for (int j = 0; j < KEYS; j += 2)
                    mx4[(j >> 1) & 3] = at_max3(mx4[(j >> 1) & 3], __uint_as_float(x[j >> 5][j & 31]), __uint_as_float(x[j >> 5][(j & 31) + 1]));
                const float mx = fmaxf(at_max3(mx4[0], mx4[1], mx4[2]), mx4[3]) * c;
                // move the reference?  (warp-wide decision: the TMEM accesses below are the whole warp's)
                float alpha = 1.f, ref = m;
                if (!SHAPED && i > 0) {
                    at_pass_wait(qd, i - 1);
                    ref = exch[((i - 1) & 1) * AT_BM + row];
                }
                if (ref == -INFINITY) {
                    ref = mx;                                   // nothing summed so far (O and l are 0, or this is the first tile)
                } else if (mx > ref + (SHAPED ? 0.f : 8.f)) {
                    alpha = at_exp2(ref - mx);
                    ref = mx;
                }
                if (!SHAPED && i + 1 < n_tiles) {
                    exch[(i & 1) * AT_BM + row] = ref;
                    at_pass_on(qd, i);
                }
                if (m != ref && m != -INFINITY) l *= at_exp2(m - ref);
                m = ref;
                if (__any_sync(0xffffffffu, alpha != 1.f)) {
                    // (shaped: this tile's scores came behind the turn's products so far, so those are in O)
                    if (!SHAPED) alive = at_mbar_wait_warp(&kv_empty[(i - 1) % STAGES], ((i - 1) / STAGES) & 1, failed);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                    for (int d = 0; d < AT_D; d += 16) {
                        uint32_t r[16];
                        at_tmem_ld16(tO + d, r);
#pragma unroll
                        for (int j = 0; j < 16; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
                        at_tmem_st16(tO + d, r);
                    }
                }
                // P, two keys a column; its sum on the way
                const float2 c2 = at_two(c), minus = at_two(m == -INFINITY ? 0.f : -m);  // (no key seen so far: every p is 0)
                float2 lt[4] = {};
                // (plain scores: the product of tile i - 2 reads this P buffer)
                if (!SHAPED && i > 1 && alive) alive = at_mbar_wait_warp(&kv_empty[(i - 2) % STAGES], ((i - 2) / STAGES) & 1, failed);
#pragma unroll
                for (int j0 = 0; j0 < KEYS; j0 += 16) {         // (16 keys a store: with 64 the registers for them cost moves and spills)
                    uint32_t pk[8];
#pragma unroll
                    for (int j = j0; j < j0 + 16; j += 2) {
                        const float2 z = at_fma2(make_float2(__uint_as_float(x[j >> 5][j & 31]), __uint_as_float(x[j >> 5][(j & 31) + 1])), c2, minus);
                        const float2 p = make_float2(at_exp2(z.x), at_exp2(z.y));
                        lt[(j >> 1) & 3] = at_add2(lt[(j >> 1) & 3], p);
                        pk[(j - j0) >> 1] = at_pack(p);
                    }
                    at_tmem_st8(tP + j0 / 2, pk);
                }
                const float2 sum = at_add2(at_add2(lt[0], lt[1]), at_add2(lt[2], lt[3]));
                l += sum.x + sum.y;
                // P (and a rescaled O) are in TMEM before the product-issuing thread hears of it
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) at_mbar_arrive(&p_ready[turn]);
            };
            if (SHAPED && n_tiles == 1) {
                // a tile alone: each turn has 32 of its keys, or half of the warps would have nothing to do.  (64 rows, cap, bias and sink, 16
                // heads: 9.0 us with all keys in one turn, 7.2 so; 64 spans of 40 rows 45 and 39.)
                if constexpr (SHAPED) tile(0, key_of(0) + turn * 32, lanes + turn * 32, &s_ready[0], std::integral_constant<int, 32>{});
            } else {
                for (int i = turn; i < n_tiles; i += 2) tile(i, key_of(i), tS, &s_ready[turn], std::integral_constant<int, AT_BN>{});
            }
            // the row's two parts: what weighs them, and the sum over both
            if (!SHAPED) asm volatile("bar.sync 1, 256;" ::: "memory");     // (the last reference has been read)
            exch[turn * AT_BM + row] = m;
            exch[(2 + turn) * AT_BM + row] = l;
            asm volatile("bar.sync 1, 256;" ::: "memory");      // the eight softmax warps
            const float m0 = exch[row], m1 = exch[AT_BM + row], l0 = exch[2 * AT_BM + row], l1 = exch[3 * AT_BM + row];
            m = fmaxf(m0, m1);
            const float f0 = m0 == -INFINITY ? 0.f : at_exp2(m0 - m), f1 = m1 == -INFINITY ? 0.f : at_exp2(m1 - m);
            l = l0 * f0 + l1 * f1;
            if (alive && at_mbar_wait_warp(&kv_empty[(n_tiles - 1) % STAGES], ((n_tiles - 1) / STAGES) & 1, failed)) {      // the last product is in O
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                have_o = at_mbar_wait_warp(&v_ready[(n_tiles - 1) % STAGES], ((n_tiles - 1) / STAGES) & 1, failed);    // (long since; the notes are seen)
                float inv = l > 0.f ? 1.f / l : 0.f;
                if (SHAPED && a.opt.sink) {                     // one more term of the denominator
                    const float sk = a.opt.sink[h] * 1.4426950408889634f, top = fmaxf(m, sk);
                    const float e = at_exp2(m - top);
                    inv = e / (l * e + at_exp2(sk - top));
                }
                // this thread's half of the columns of O, the two parts together
                uint32_t o0[32], o1[32];
                at_tmem_ld32(lanes + AT_COL_O + turn * 32, o0);
                if (SHAPED) at_tmem_ld32(lanes + AT_COL_O + AT_D + turn * 32, o1);
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    out[j] = __uint_as_float(o0[j]) * (SHAPED ? f0 : 1.f);
                    if (SHAPED) out[j] = fmaf(__uint_as_float(o1[j]), f1, out[j]);
                }
                bf16* dst = a.out + ((size_t)(row0 + i0 + row) * a.Hq + h) * AT_D + turn * 32;
                if (!SHARED && valid) {
#pragma unroll
                    for (int d = 0; d < 32; d += 8) {
                        uint32_t v[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            __nv_bfloat162 p = __floats2bfloat162_rn(out[d + 2 * e] * inv, out[d + 2 * e + 1] * inv);
                            v[e] = *reinterpret_cast<uint32_t*>(&p);
                        }
                        *reinterpret_cast<uint4*>(dst + d) = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                    if (notes.count) notes.put_nans(dst, 1, turn, 1, qpos, klo, kept);
                }
            }
        }
    }
    if (SHARED && s < a.S && warp >= 2) {
        // ---- a shared tile of query rows: this block's part into memory, a ticket, and the last one combines
        const int qd = warp & 3, half = (warp - 2) >> 2, row = qd * 32 + lane;
        const int slot = ((int)gridDim.y - 1 - (int)blockIdx.y) * a.Hq + h;
        const size_t mine = (size_t)slot * a.splits + blockIdx.z;
        float* po = a.part_o + mine * (AT_D * AT_BM) + half * 32 * AT_BM;
        float* pml = a.part_ml + mine * (2 * AT_BM);
        const bool ok = have_o && !failed_flag;                 // (a block without key tiles, or one that gave up, has no part)
        if (half == 0) {
            pml[row] = ok ? m : -INFINITY;
            pml[AT_BM + row] = ok ? l : 0.f;
        }
        if (ok) {
#pragma unroll
            for (int j = 0; j < 32; ++j) po[j * AT_BM + row] = out[j];
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
