// What the tcgen05 attention kernels share: bounded waits on mbarriers, TMA loads, operand descriptors, tcgen05 products with the
// first operand in shared memory or in TMEM, TMEM loads and stores, and the tensor maps.
#pragma once
#include <cuda.h>
#include "common.cuh"

#define AT_SPIN_LIMIT 4000000
#define AT_NAP_NS 100

__device__ __forceinline__ uint32_t at_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void at_mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(at_smem(bar)), "r"(count));
}
__device__ __forceinline__ void at_mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(at_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void at_mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(at_smem(bar)) : "memory");
}
// NAP: how long a try that finds the phase open sleeps before the next (a waiting lane without that issues instructions all the time)
template <int NAP = 0>
__device__ __forceinline__ bool at_mbar_wait(uint64_t* bar, uint32_t parity, volatile int* failed) {
    const uint32_t a = at_smem(bar);
#pragma unroll 1
    for (int it = 0; it < AT_SPIN_LIMIT; ++it) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(a), "r"(parity) : "memory");
        if (ok) return true;
        if (*failed) return false;
        if (NAP > 0) __nanosleep(NAP);
    }
    *failed = 1;
    return false;
}
// Is the phase over?  (Does not wait.)
__device__ __forceinline__ bool at_mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(at_smem(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// A warp's wait, all lanes in step
__device__ __forceinline__ bool at_mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* failed) {
    return __all_sync(0xffffffffu, at_mbar_wait(bar, parity, failed));
}
__device__ __forceinline__ void at_tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(at_smem(dst)), "l"(map), "r"(at_smem(bar)), "r"(c0), "r"(c1) : "memory");
}
// Operand tile of 128-byte rows with the 128-byte swizzle, groups of 8 rows 1024 bytes apart.  For a
// K-major operand a row is a matrix row (64 k); for an MN-major one a row is one k (64 n).
__device__ __forceinline__ uint64_t at_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void at_umma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void at_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(at_smem(bar)) : "memory");
}
__device__ __forceinline__ void at_tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 2^x by the special-function unit (x <= 0 here; -inf gives 0)
__device__ __forceinline__ float at_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ void at_tmem_ld32_nowait(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
}
__device__ __forceinline__ void at_tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
                 "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                   "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
                   "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
                 : "memory");
}

__device__ __forceinline__ void at_tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void at_tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
                   "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void at_tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// A product whose A operand lies in TMEM (row = lane, two bfloat16 of k per 32-bit column)
__device__ __forceinline__ void at_umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
// The wait for a thread's TMEM loads, tied to the registers of one of them: what is computed from those
// registers cannot be scheduled ahead of the wait, while another load may stay in flight across it.
__device__ __forceinline__ void at_tmem_wait_ld(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                   "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :: "memory");
}

// ---- values that some rows of a block do not see.  A tile's hidden keys have weights of exactly zero, but zero times NaN or
// infinity is NaN in the product: a recycled page's last owner, or a later row of the span, would reach every row of the block.  So
// before the product of a tile that not every row sees whole, the warp that loads tiles puts zeros over the values that no row
// sees and takes what is not finite out of the others; AtNotes holds those keys and their columns, and a row that sees such a key
// ends as NaN there.  The softmax warps, whose chain bounds these kernels, have no part in it (there it cost 4 to 13 %).
__device__ __forceinline__ void at_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// eight bfloat16 values: is one of them infinite or NaN (an exponent of ones)?
__device__ __forceinline__ bool at_not_finite(const uint4& v) {
    auto two = [](uint32_t x) { return ((x & 0x7f807f80u) + 0x00800080u) & 0x80008000u; };
    return (two(v.x) | two(v.y) | two(v.z) | two(v.w)) != 0;
}
// A lane's part of a tile's values, 16 bytes of every STEP-th key from `key` on (a key's 64 columns are one swizzled row of 128 bytes,
// eight lanes): zeros where the tile's key is not among `shown`.  Returns whether another value is not finite.
template <int STEP>
__device__ __forceinline__ bool at_clean(unsigned char* tile, int key, unsigned long long shown) {
    uint4* p = reinterpret_cast<uint4*>(tile) + (threadIdx.x & 7);
    bool odd = false;
#pragma unroll 8
    for (int t = 0; t < 64 / STEP; ++t) {                       // (a loop of loads alone: they are in flight together)
        const int k = key + t * STEP;
        const bool o = at_not_finite(p[k * 8]);
        odd |= o && (shown >> k & 1);
    }
    if (~shown)
        for (int t = 0; t < 64 / STEP; ++t)
            if (!(shown >> (key + t * STEP) & 1)) p[(key + t * STEP) * 8] = make_uint4(0u, 0u, 0u, 0u);
    return odd;
}
// Takes what is not finite out of a lane's 16 bytes of a key; every lane of the warp calls it (`on`: this lane has such a part).  Returns
// those columns of the key's 64, the same in its eight lanes.
__device__ __forceinline__ unsigned long long at_take_odd(unsigned char* tile, int key, bool on) {
    const int chunk = threadIdx.x & 7;
    uint4* p = reinterpret_cast<uint4*>(tile + key * 128) + chunk;
    unsigned long long odd = 0;
    if (on && at_not_finite(*p)) {
        unsigned short* v = reinterpret_cast<unsigned short*>(p);
        for (int e = 0; e < 8; ++e)
            if ((v[e] & 0x7f80) == 0x7f80) {
                v[e] = 0;
                odd |= 1ull << ((chunk ^ (key & 7)) * 8 + e);
            }
    }
    for (int o = 1; o < 8; o <<= 1) odd |= __shfl_xor_sync(0xffffffffu, odd, o);
    return odd;
}
// the lowest n of 64 bits
__device__ __forceinline__ unsigned long long at_below(int n) { return n <= 0 ? 0ull : n >= 64 ? ~0ull : (1ull << n) - 1; }
template <int PARTS, int MOST>                                  // columns in 64s; keys that find room
struct AtNotes {
    unsigned long long cols[MOST][PARTS];
    int key[MOST];                                              // positions in the request
    int count, low, high;                                       // keys noted; those that found no room lie from low to high
    __device__ __forceinline__ void clear() { count = 0; low = 0x7fffffff; high = -1; }
    // by one lane, for a key's part of the columns; returns the place for other parts, or -1
    __device__ __forceinline__ int add(int k) {
        const int i = atomicAdd(&count, 1);
        if (i < MOST) {
            key[i] = k;
            for (int p = 0; p < PARTS; ++p) cols[i][p] = 0;
            return i;
        }
        atomicMin(&low, k);
        atomicMax(&high, k);
        return -1;
    }
    // NaN into the values of a row's columns [32 w, 32 w + 32 n), `step` values apart, that have met a value that is not finite at a key of
    // [from, pos] or [0, kept) (all of them, if it may see a key without room).  A call behind the row's stores: rare, and not
    // to be carried by what comes before it
    template <typename T>
    __device__ __noinline__ void put_nans(T* row, size_t step, int w, int n, int pos, int from, int kept) const {
        for (int k = w; k < w + n; ++k) {
            uint32_t m = low <= pos && (high >= from || low < kept) ? 0xffffffffu : 0u;
            for (int i = 0; i < min(count, MOST); ++i)
                if (key[i] <= pos && (key[i] >= from || key[i] < kept)) m |= (uint32_t)(cols[i][k >> 1] >> ((k & 1) * 32));
            for (int j = 0; j < 32; ++j)
                if (m >> j & 1) row[((k - w) * 32 + j) * step] = from_float<T>(__int_as_float(0x7fc00000));
        }
    }
};
// ------------------------------------------------------------------------------------------ host side
typedef CUresult (*AtEncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                    const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static AtEncodeTiledFn at_encode_tiled() {
    static AtEncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (AtEncodeTiledFn)p;
    }
    return fn;
}
// Rows of `cols` bfloat16 values; a box is 64 columns (128 bytes, swizzled; zeros beyond the row) of box_rows rows.
static int at_make_map(CUtensorMap* map, const void* ptr, cuuint64_t cols, cuuint64_t rows, cuuint32_t box_rows) {
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return at_encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS ? 0 : -6;
}
