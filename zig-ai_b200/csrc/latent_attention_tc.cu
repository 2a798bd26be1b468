// Attention of many heads over one shared cached vector per position (see latent_attention.cu for the sums), spans of rows, on the
// 5th-generation tensor cores.
//
// The cached rows [c | r] are the same for every head, so the (row, head) pairs of a span are one list of queries over the same
// keys: a block owns 128 neighbouring pairs (8 rows of 16 heads).  Per tile of 64 cached rows
//
//     S = Q K^T      tcgen05.mma, M = 128 pairs, N = 64 keys, K = R + Dr, operands from shared memory, into TMEM
//     P = exp2(..)   four warps, a pair a thread: its 64 scores from TMEM, P back into TMEM as the next product's first operand
//     O += P C       tcgen05.mma, the tile's own first R columns as values: the same bytes that were the keys, read as an MN-major
//                    operand 64 columns at a time; O (R columns) stays in TMEM and is rescaled there when some pair's maximum moves
//
// Queries and cached rows come by TMA (no multicast) in boxes of 64 columns, the cached rows page by page into LT_STAGES stages; the
// last box reaches beyond the row and is filled with zeros.  TMEM holds two score and two P buffers, so the scores of tile i + 2
// are issued behind the product of tile i.  Roles: warp 0 one lane issues the loads (and the warp cleans the values of tiles that
// not every pair sees whole), warp 1 one lane the products, warps 2-5 are the softmax.  Blocks are handed out from the last pairs
// backwards (they have the most keys).  Every wait on an mbarrier is bounded; a block whose wait runs out raises the status word, its roles leave their loops, TMEM is freed and the block returns.
//
// What bounds it: the chain of a tile (scores, softmax, P, product), 2.1 us of 64 keys, with one block an SM (200 KB of shared memory);
// the products' tensor time is about 0.8 us of it.  16 heads, R = 256, Dr = 32, mma.sync (four warps sharing tiles of 32) and here: 2048
// rows 275 and 77 us, 128 behind 4000 160 and 136 (the reference as the running maximum takes 5 % of it, the cleaning 2 %).
#include "attention_tc_helpers.cuh"

#define LT_BM 128
#define LT_BN 64
#define LT_THREADS 192
#define LT_STAGES 3
#define LT_MAX_R 256
#define LT_MAX_BLOCKS 5                               // boxes of 64 columns: R / 64 and one for the rotated part
#define LT_Q_BLOCK (LT_BM * 128)                      // 16 KB
#define LT_K_BLOCK (LT_BN * 128)                      // 8 KB
#define LT_TMEM_COLS 512                              // two score buffers in columns 0..127, O in 128..383, two P buffers in 384..447
#define LT_COL_O (2 * LT_BN)
#define LT_COL_P (LT_COL_O + LT_MAX_R)
typedef AtNotes<LT_MAX_R / 64, 64> LtNotes;

struct LtArgs {
    bf16* out;                  // [N, H, R]
    const int* block_table;     // [S, table_width]
    const int* cu_q;            // [S + 1] first row of each request's span
    const int* ctx_lens;        // [S] positions cached before the step
    int* status;
    const float* sink;          // [H] or null
    int num_pages, table_width, S, page_size, page_shift, H, R, Dr, min_rows;
    float scale_log2;
};

// waits for a load already issued, so that none lands in shared memory of a block that has gone
__device__ __forceinline__ void lt_drain(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = at_smem(bar);
    for (int spin = 0; spin < AT_SPIN_LIMIT; ++spin) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done) : "r"(addr), "r"(parity) : "memory");
        if (done) break;
    }
}

__global__ void __launch_bounds__(LT_THREADS) latent_attention_tc_kernel(const __grid_constant__ CUtensorMap map_lat,
                                                                         const __grid_constant__ CUtensorMap map_rot,
                                                                         const __grid_constant__ CUtensorMap map_kv, const LtArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int n_lat = a.R / 64, n_blocks = n_lat + (a.Dr > 0 ? 1 : 0);
    const uint32_t q_bytes = (uint32_t)n_blocks * LT_Q_BLOCK, kv_bytes = (uint32_t)n_blocks * LT_K_BLOCK;
    unsigned char* sQ = smem_raw;
    unsigned char* sKV = smem_raw + q_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + (size_t)LT_STAGES * kv_bytes);
    uint64_t& q_full = bars[0];
    uint64_t* kv_full = bars + 1;                               // [LT_STAGES]
    uint64_t* kv_empty = bars + 1 + LT_STAGES;                  // [LT_STAGES]
    uint64_t* s_ready = bars + 1 + 2 * LT_STAGES;               // [2] scores of tile i in buffer i & 1
    uint64_t* p_ready = bars + 3 + 2 * LT_STAGES;               // [2] P of tile i in buffer i & 1
    uint64_t* o_ready = bars + 5 + 2 * LT_STAGES;               // [2] the product of tile i has read P buffer i & 1 and added to O
    uint64_t* v_ready = bars + 7 + 2 * LT_STAGES;               // [LT_STAGES] the values of a stage are there and clean
    uint32_t& tmem_base_holder = *reinterpret_cast<uint32_t*>(bars + 7 + 3 * LT_STAGES);
    int* words = reinterpret_cast<int*>(bars + 8 + 3 * LT_STAGES);
    int& failed_flag = words[0];
    int& s_seq = words[1];
    int& s_i0 = words[2];
    LtNotes& notes = *reinterpret_cast<LtNotes*>(words + 4);
    volatile int* failed = &failed_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    if (tid == 0) {
        failed_flag = (at_smem(smem_raw) & 1023u) ? 1 : 0;      // the swizzled tiles need 1024-byte alignment
        notes.clear();
        at_mbar_init(&q_full, 1);
        for (int s = 0; s < LT_STAGES; ++s) {
            at_mbar_init(&v_ready[s], 1);
            at_mbar_init(&kv_full[s], 1);
            at_mbar_init(&kv_empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            at_mbar_init(&s_ready[b], 1);
            at_mbar_init(&p_ready[b], 4);                       // one arrival per softmax warp
            at_mbar_init(&o_ready[b], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(at_smem(&tmem_base_holder)), "r"(LT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_holder;
    pdl_trigger();
    pdl_wait();
    if (tid == 0) {
        int t = (int)gridDim.x - 1 - (int)blockIdx.x, s = 0;    // tiles of pairs from the last request's last ones backwards
        for (; s < a.S; ++s) {
            const int n = a.cu_q[s + 1] - a.cu_q[s], nt = n < a.min_rows ? 0 : (n * a.H + LT_BM - 1) / LT_BM;
            if (t < nt) break;
            t -= nt;
        }
        s_seq = s;
        s_i0 = t * LT_BM;
    }
    __syncthreads();
    const int s = s_seq, i0 = s_i0;
    if (s < a.S && !failed_flag) {
        const int row0 = a.cu_q[s], ctx = a.ctx_lens[s];
        const int pairs = min(LT_BM, (a.cu_q[s + 1] - row0) * a.H - i0);      // valid pairs of this block
        const int kend = ctx + (i0 + pairs - 1) / a.H + 1;                    // one past the last visible key of the block
        const int n_tiles = (kend + LT_BN - 1) / LT_BN;
        // the tiles that end behind the first pair's row, three at most (the last one counts as such: when its values are ready, so are all)
        auto first_part = [&]() { return min((ctx + i0 / a.H + 1) / LT_BN, n_tiles - 1); };

        if (warp == 0) {
            // ---- loads: the block's queries, then a stage of cached rows per tile, page by page
            const int* table = a.block_table + (size_t)s * a.table_width;
            const int ps = a.page_size, box_rows = ps < LT_BN ? ps : LT_BN, per_tile = LT_BN / box_rows;
            if (lane == 0) {
                at_mbar_expect_tx(&q_full, q_bytes);
                for (int b = 0; b < n_blocks; ++b)
                    at_tma_load_2d(sQ + (size_t)b * LT_Q_BLOCK, b < n_lat ? &map_lat : &map_rot, b < n_lat ? b * 64 : 0, row0 * a.H + i0, &q_full);
            }
            const int p0 = first_part();
            int issued = 0;
            if (lane == 0)
                for (; issued < n_tiles; ++issued) {
                    const int st = issued % LT_STAGES;
                    if (!at_mbar_wait(&kv_empty[st], ((issued / LT_STAGES) & 1) ^ 1, failed)) break;
                    at_mbar_expect_tx(&kv_full[st], kv_bytes);
                    unsigned char* dst = sKV + (size_t)st * kv_bytes;
                    for (int p = 0; p < per_tile; ++p) {
                        const int key0 = issued * LT_BN + p * box_rows;
                        const int idx = key0 >> a.page_shift, off = key0 & (ps - 1);
                        int page = idx < a.table_width ? table[idx] : 0;              // beyond the table: the null page
                        if ((unsigned)page >= (unsigned)a.num_pages) {                // outside the pool: page 0, and the step is void
                            zai_raise(a.status, ZAI_ST_PAGE);
                            page = 0;
                        }
                        for (int b = 0; b < n_blocks; ++b)
                            at_tma_load_2d(dst + (size_t)b * LT_K_BLOCK + (size_t)p * box_rows * 128, &map_kv, b * 64, page * ps + off, &kv_full[st]);
                    }
                    if (issued < p0) at_mbar_arrive(&v_ready[st]);
                }
            __syncwarp();
            // the last tiles' values, behind all loads (which need none of their products): with the warp in step beside the one lane a
            // tile's load came a sixth later
            for (int i = p0; i < n_tiles; ++i) {
                // as keys the rows have to stay what they are until the scores are there
                const int st = i % LT_STAGES;
                if (!at_mbar_wait_warp(&kv_full[st], (i / LT_STAGES) & 1, failed) || !at_mbar_wait_warp(&s_ready[i & 1], (i >> 1) & 1, failed)) break;
                unsigned char* rows = sKV + (size_t)st * kv_bytes + (size_t)(lane >> 3) * LT_K_BLOCK;
                const bool mine = (lane >> 3) < n_lat;          // (a row a turn, eight lanes a block of 64 columns)
                const bool odd = mine && at_clean<1>(rows, 0, at_below(kend - i * LT_BN));
                if (__any_sync(0xffffffffu, odd))
                    for (int k = 0; k < LT_BN; ++k) {
                        const unsigned long long cols = at_take_odd(rows, k, mine);
                        if (!__any_sync(0xffffffffu, cols != 0)) continue;
                        int e = lane == 0 ? notes.add(i * LT_BN + k) : 0;
                        e = __shfl_sync(0xffffffffu, e, 0);
                        if (e >= 0 && (lane & 7) == 0) notes.cols[e][lane >> 3] = cols;
                    }
                at_proxy_fence();                               // (generic writes, which the product reads)
                __syncwarp();
                if (lane == 0) at_mbar_arrive(&v_ready[st]);
            }
            if (lane == 0 && *failed) {                         // loads already issued still land here: wait for them
                for (int i = max(issued - LT_STAGES, 0); i < issued; ++i) lt_drain(&kv_full[i % LT_STAGES], (i / LT_STAGES) & 1);
                lt_drain(&q_full, 0);
            }
        } else if (warp == 1) {
            if (zai_elect()) {                                   // (issued behind `lane == 0` a product takes twice as long)
                // ---- products.  Instruction descriptors: D 32-bit, A and B bfloat16, M = 128, N = 64; the scores have both
                // operands K-major; O has A (P) in TMEM and B (the cached rows' first R columns) MN-major.
                constexpr uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_BN >> 3) << 17) | ((uint32_t)(LT_BM >> 4) << 24);
                constexpr uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(64 >> 3) << 17) |
                                             ((uint32_t)(LT_BM >> 4) << 24);
                const uint32_t tS = tmem_base, tO = tmem_base + LT_COL_O, tP = tmem_base + LT_COL_P;
                const uint32_t aQ = at_smem(sQ);
                const int k_steps = (a.R + a.Dr) / 16;
                bool ok = at_mbar_wait(&q_full, 0, failed);
                auto scores = [&](int i) {                      // S = Q K^T of tile i into score buffer i & 1
                    const int st = i % LT_STAGES;
                    if (!at_mbar_wait(&kv_full[st], (i / LT_STAGES) & 1, failed)) return false;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t aK = at_smem(sKV + (size_t)st * kv_bytes);
                    for (int k = 0; k < k_steps; ++k)
                        at_umma(tS + (i & 1) * LT_BN, at_desc(aQ + (k >> 2) * LT_Q_BLOCK + (k & 3) * 32),
                                at_desc(aK + (k >> 2) * LT_K_BLOCK + (k & 3) * 32), idesc_s, k > 0 ? 1u : 0u);
                    at_commit(&s_ready[i & 1]);
                    return true;
                };
                if (ok) ok = scores(0);
                if (ok && n_tiles > 1) ok = scores(1);
                auto product = [&](int i, bool wait) {          // O += P C of tile i, and the scores of tile i + 2; `wait`: its values are cleaned
                    const int st = i % LT_STAGES;
                    ok = at_mbar_wait(&p_ready[i & 1], (i >> 1) & 1, failed) && (!wait || at_mbar_wait(&v_ready[st], (i / LT_STAGES) & 1, failed));
                    if (!ok) return;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t aV = at_smem(sKV + (size_t)st * kv_bytes);
                    for (int b = 0; b < n_lat; ++b) {
#pragma unroll
                        for (int kk = 0; kk < LT_BN / 16; ++kk) // 16 keys a step: eight columns of P, two groups of 8 cached rows
                            at_umma_ts(tO + b * 64, tP + (i & 1) * (LT_BN / 2) + kk * 8, at_desc(aV + b * LT_K_BLOCK + kk * 2048), idesc_o,
                                       (i > 0 || kk > 0) ? 1u : 0u);
                    }
                    at_commit(&o_ready[i & 1]);
                    if (i + 2 < n_tiles) ok = scores(i + 2);
                    at_commit(&kv_empty[st]);
                };
                const int p0 = first_part();
#pragma unroll 1
                for (int i = 0; i < n_tiles && ok; ++i) product(i, i >= p0);
            }
        } else {
            // ---- softmax: thread = pair.  The pair's reference is its running maximum, so that the largest weight is exactly 1
            // whatever it is rounded to.
            const int qd = warp & 3;                            // this warp's quarter of the TMEM lanes
            const int row = qd * 32 + lane;
            const bool valid = row < pairs;
            const int qpos = ctx + (i0 + row) / a.H;            // the pair's position: keys 0..qpos are visible
            const uint32_t tS = tmem_base + ((uint32_t)(qd * 32) << 16), tO = tS + LT_COL_O, tP = tS + LT_COL_P;
            const float c = a.scale_log2;
            float m = -INFINITY, l = 0.f;                       // m: the pair's maximum, in units of the scores
            bool alive = true;
            for (int i = 0; i < n_tiles && alive; ++i) {
                if (!at_mbar_wait_warp(&s_ready[i & 1], (i >> 1) & 1, failed)) { alive = false; break; }    // (the warp leaves together)
                const uint32_t tSi = tS + (i & 1) * LT_BN, tPi = tP + (i & 1) * (LT_BN / 2);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int hi = valid ? min(qpos + 1 - i * LT_BN, LT_BN) : 0;      // keys of this tile that the pair sees: below hi
                const bool full = hi >= LT_BN;
                // the pair's 64 scores: their maximum, their weights against the reference into P, the weights' sum
                uint32_t r[2][32];
                at_tmem_ld32_nowait(tSi, r[0]);
                at_tmem_ld32_nowait(tSi + 32, r[1]);
                at_tmem_wait_ld(r[0]);
                at_tmem_wait_ld(r[1]);
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int k = 0; k < 2; ++k)
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        // (a hidden score may be anything, also NaN: it is replaced before the exponential)
                        if (!full && 32 * k + j >= hi) r[k][j] = __float_as_uint(-INFINITY);
                        mx4[j & 3] = fmaxf(mx4[j & 3], __uint_as_float(r[k][j]));
                    }
                const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
                // move the reference?  (warp-wide decision: the TMEM accesses below are the whole warp's)
                float alpha = 1.f;
                if (m == -INFINITY) {
                    m = mx;                                     // nothing summed so far
                } else if (mx > m) {
                    alpha = at_exp2(m * c - mx * c);
                    m = mx;
                }
                if (i > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                    if (!at_mbar_wait_warp(&o_ready[(i - 1) & 1], ((i - 1) >> 1) & 1, failed)) { alive = false; break; }   // the product before has added to O
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int c0 = 0; c0 < a.R; c0 += 32) {
                        uint32_t o[32];
                        at_tmem_ld32(tO + c0, o);
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
                        at_tmem_st32(tO + c0, o);
                    }
                    l *= alpha;
                }
                const float ref = m == -INFINITY ? 0.f : m * c;
                float lt4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    uint32_t pk[16];
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const float p0 = at_exp2(__uint_as_float(r[k][j]) * c - ref), p1 = at_exp2(__uint_as_float(r[k][j + 1]) * c - ref);
                        lt4[(j >> 1) & 3] += p0 + p1;
                        __nv_bfloat162 v = __floats2bfloat162_rn(p0, p1);
                        pk[j >> 1] = *reinterpret_cast<uint32_t*>(&v);
                    }
                    // (This P buffer was read by the product of the tile two before.  That product was issued before this tile's
                    // scores, and the commit behind the scores covers every product issued before it.)
                    at_tmem_st16(tPi + 16 * k, pk);             // 32 keys = 16 columns of P
                }
                l += (lt4[0] + lt4[1]) + (lt4[2] + lt4[3]);
                // P (and a rescaled O) are in TMEM before the product-issuing thread hears of it
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) at_mbar_arrive(&p_ready[i & 1]);
            }
            if (alive && at_mbar_wait_warp(&o_ready[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, failed)
                && at_mbar_wait_warp(&v_ready[(n_tiles - 1) % LT_STAGES], ((n_tiles - 1) / LT_STAGES) & 1, failed)) {     // (the latter: the notes are seen)
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                float inv = l > 0.f ? 1.f / l : 0.f;
                if (a.sink) {                                   // one more term of the denominator
                    const float M = m * c, sk = a.sink[(i0 + row) % a.H] * 1.4426950408889634f, n = fmaxf(M, sk);
                    const float e = at_exp2(M - n);
                    inv = e / (l * e + at_exp2(sk - n));
                }
                bf16* dst = a.out + ((size_t)row0 * a.H + i0 + row) * a.R;
                for (int c0 = 0; c0 < a.R; c0 += 32) {
                    uint32_t o[32];
                    at_tmem_ld32(tO + c0, o);
                    if (valid) {
#pragma unroll
                        for (int d = 0; d < 32; d += 8) {
                            uint32_t v[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                __nv_bfloat162 p = __floats2bfloat162_rn(__uint_as_float(o[d + 2 * e]) * inv, __uint_as_float(o[d + 2 * e + 1]) * inv);
                                v[e] = *reinterpret_cast<uint32_t*>(&p);
                            }
                            *reinterpret_cast<uint4*>(dst + c0 + d) = make_uint4(v[0], v[1], v[2], v[3]);
                        }
                    }
                }
                if (valid && notes.count) notes.put_nans(dst, 1, 0, a.R / 32, qpos, 0, 0);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(LT_TMEM_COLS) : "memory");
    }
    if (tid == 0 && failed_flag) zai_raise(a.status, ZAI_ST_WAIT);
}

// 1 if this kernel takes the sizes: latents of a multiple of 64 up to 256, a rotated part of a multiple of 16 up to 64, pages of a
// power of two from 8 to 128 positions (a tile of 64 cached rows is loaded page by page, or as half of a page of 128)
ZAI_API int zai_latent_attention_tc_supports(int H, int R, int Dr, int page_size) {
    if (H < 1 || H > 32767 || R < 64 || R > LT_MAX_R || R % 64 || Dr < 0 || Dr > 64 || Dr % 16) return 0;
    if (page_size < 8 || page_size > 128 || (page_size & (page_size - 1))) return 0;
    return at_encode_tiled() != nullptr;
}
ZAI_API int zai_latent_attention_tc_pairs() { return LT_BM; }

// out [N, H, R] from q_lat [N, H, R], q_rot [N, H, Dr] and pages [num_pages, page_size, R + Dr], bfloat16; spans of at least min_rows rows
// are run; n_tiles: the sum over them of their rows x H / 128, rounded up (or more); sink [H] 32-bit or null.
ZAI_API int zai_latent_attention_tc(void* out, const void* q_lat, const void* q_rot, const void* pages, int num_pages, int* status,
                                    const int* block_table, int table_width, const int* cu_q, const int* ctx_lens, int N, int S,
                                    int n_tiles, int page_size, int H, int R, int Dr, float scale, const float* sink, int min_rows,
                                    cudaStream_t stream) {
    if (N <= 0 || S <= 0 || n_tiles <= 0) return ZAI_OK;
    if (!zai_latent_attention_tc_supports(H, R, Dr, page_size) || (long long)N * H > 0x7fffffffLL) return ZAI_BAD_SIZE;
    if ((reinterpret_cast<uintptr_t>(q_lat) | (Dr ? reinterpret_cast<uintptr_t>(q_rot) : 0) | reinterpret_cast<uintptr_t>(pages) | reinterpret_cast<uintptr_t>(out)) & 15)
        return ZAI_BAD_SIZE;
    CUtensorMap ml, mr, mkv;
    int e = at_make_map(&ml, q_lat, (cuuint64_t)R, (cuuint64_t)N * H, LT_BM);
    if (e) return e;
    if (Dr) e = at_make_map(&mr, q_rot, (cuuint64_t)Dr, (cuuint64_t)N * H, LT_BM);
    else mr = ml;
    if (e) return e;
    e = at_make_map(&mkv, pages, (cuuint64_t)(R + Dr), (cuuint64_t)num_pages * page_size, (cuuint32_t)(page_size < LT_BN ? page_size : LT_BN));
    if (e) return e;
    LtArgs a;
    a.out = (bf16*)out; a.block_table = block_table; a.cu_q = cu_q; a.ctx_lens = ctx_lens; a.status = status; a.sink = sink;
    a.num_pages = num_pages; a.table_width = table_width; a.S = S; a.page_size = page_size; a.H = H; a.R = R; a.Dr = Dr; a.min_rows = min_rows;
    a.scale_log2 = scale * 1.4426950408889634f;
    a.page_shift = 0;
    while ((1 << a.page_shift) < page_size) ++a.page_shift;
    const int n_blocks = R / 64 + (Dr > 0 ? 1 : 0);
    constexpr size_t words = 256 + sizeof(LtNotes);
    static_assert(LT_MAX_BLOCKS * (LT_Q_BLOCK + LT_STAGES * LT_K_BLOCK) + words <= 227 * 1024, "one block an SM");
    const size_t smem = (size_t)n_blocks * (LT_Q_BLOCK + LT_STAGES * LT_K_BLOCK) + words;
    static unsigned long long configured = 0;
    if (zai_first_on_device(&configured)) {
        const cudaError_t err = cudaFuncSetAttribute(latent_attention_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)(LT_MAX_BLOCKS * (LT_Q_BLOCK + LT_STAGES * LT_K_BLOCK) + words));
        if (err != cudaSuccess) return (int)err;
    }
    return launch_pdl(latent_attention_tc_kernel, dim3(n_tiles), dim3(LT_THREADS), smem, stream, ml, mr, mkv, a);
}
