// Shared pieces of the tensor-core sparse attention (attn_tc.cu): operand panels, splits, tensor-memory moves.
//
// Queries pick K of the keys behind them, but K is a sizeable share of a sequence of a few thousand, and the gather
// kernels (sparse_attn.cu) move every picked row through the L1 once per query: 26 GB of it at 32 x 8 x 1024 queries x
// 128 keys against 0.7 GB of tensors.  Here a tile of 128 queries meets tiles of 128 keys on the tensor cores and a
// map says which of the products are picked.  At C5's density of 1/4 (causal) that is four times the arithmetic on
// hardware that has thirty times the rate.
//
// fp32 and fp16 inputs are split into three bf16 parts each (8 + 8 + 8 bits: the fp32 mantissa, exactly) and a product
// is the six partial products down to 2^-16 x 2^-8 of the largest, accumulated in fp32: the arithmetic has fp32's
// precision.  bf16 inputs are one part; probabilities and score gradients, which are fp32, always are three.
#pragma once
#include "tcgen05.cuh"

namespace cinn {
namespace atc {

constexpr int T = 128;                     // queries per tile, keys per tile
constexpr int PANEL = T * 128;             // bytes of 128 rows x 64 bf16 columns, 128-byte swizzle
constexpr int PARTS = 3;                   // bf16 parts of an fp32 value
constexpr int MAX_SLOTS = 512;             // K: a warp permutes a row of probabilities in registers
constexpr int MAX_COUNT = 255;             // times one query may pick one key

// What the queries picked, per (batch, query): one bit per key; the rank of every slot's key among the query's picked
// keys in ascending order (0xffff for an index that takes no part); and how often each picked key was picked, by rank.
struct Picks {
    const uint32_t* bits;                  // (B, L, Lp / 32)
    const uint16_t* rank;                  // (B, L, K)
    const uint8_t* count;                  // (B, L, K)
    const uint16_t* before;                // (B, L, Lp / 32): picked keys before each word
    const int* repeats;                    // (B, tiles): whether a query of the tile picked a key more than once
};

// 32 lanes x 32 columns, without waiting
__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, "
        "%19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
// the same, 16 columns
__device__ __forceinline__ void ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
          "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, uint32_t bar, uint32_t dst, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}

// a box of shared memory to global memory, written or added (fp32, rounded to nearest, in L2)
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_add_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}
// Two fp32 values in a register pair and one instruction for both.
__device__ __forceinline__ uint64_t pair2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpair2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// two fp32 values as three packed bf16 pairs whose sum they are
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    auto pack = [](float x, float y) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(x, y);
        return *reinterpret_cast<const uint32_t*>(&t);
    };
    const uint64_t minus = pair2(-1.0f, -1.0f);
    auto rest = [&](uint32_t part) {                      // what the part leaves: exact
        unpair2(fma2(pair2(__uint_as_float(part << 16), __uint_as_float(part & 0xffff0000u)), minus, pair2(a, b)), a, b);
    };
    hi = pack(a, b);
    rest(hi);
    mid = pack(a, b);
    rest(mid);
    lo = pack(a, b);
}

// 2^x and e^x; a result below 2^-126 is 0
__device__ __forceinline__ float exp2_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float exp_fast(float x) { return exp2_fast(x * 1.4426950408889634f); }

// if (bits & mask) *to++ = x; else p = 0.  As predicated instructions: a branch costs a warp some sixty cycles.
__device__ __forceinline__ void push_if(uint32_t bits, uint32_t mask, float*& to, float x, float& p) {
    asm volatile(
        "{\n\t.reg .pred t;\n\t.reg .b32 m;\n\t"
        "and.b32 m, %2, %3;\n\t"
        "setp.ne.u32 t, m, 0;\n\t"
        "@t st.global.f32 [%0], %4;\n\t"
        "@t add.u64 %0, %0, 4;\n\t"
        "selp.f32 %1, %1, 0f00000000, t;\n\t}"
        : "+l"(to), "+f"(p) : "r"(bits), "r"(mask), "f"(x) : "memory");
}

// *p = (x, y) if take is not zero, as one predicated instruction
__device__ __forceinline__ void store2_if(float2* p, float x, float y, uint32_t take) {
    asm volatile(
        "{\n\t.reg .pred t;\n\t"
        "setp.ne.u32 t, %3, 0;\n\t"
        "@t st.global.v2.f32 [%0], {%1, %2};\n\t}"
        ::"l"(p), "f"(x), "f"(y), "r"(take) : "memory");
}
__device__ __forceinline__ void st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}
// Writes 16 consecutive reduction positions (keys or queries: one step of an MMA) of this lane's row as an A operand in tensor
// memory: the leading parts in 8 columns at `lead`, the second and third in 8 columns each at `rest`.
__device__ __forceinline__ void store_parts16(uint32_t rest, uint32_t lead, const float* v) {
    uint32_t hi[8], mid[8], lo[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split2(v[2 * i], v[2 * i + 1], hi[i], mid[i], lo[i]);
    st8(lead, hi);
    st8(rest, mid);
    st8(rest + 8, lo);
}

// D (+)= part X of a tensor-memory operand of 16 STEPS positions (store_parts16) times an MN-major panel
template <int X, int STEPS = 8>
__device__ __forceinline__ void mma_part_at(uint32_t d, uint32_t rest, uint32_t lead, uint32_t b, uint32_t idesc, bool fresh) {
    static_assert(STEPS == 8 || STEPS == 2, "the steps are written out");
    const uint32_t a = X == 0 ? lead : rest + (X - 1) * 8;
#define CINN_MMA_TS_FIRST                                                                                                           \
    "{\n\t.reg .pred p, e;\n\t.reg .b64 b;\n\t.reg .b32 x, y;\n\t"                                                                  \
    "elect.sync _|e, 0xffffffff;\n\t"                                                                                               \
    "setp.ne.b32 p, %5, 0;\n\t"                                                                                                     \
    "mov.b64 b, {%2, %4};\n\t"                                                                                                      \
    "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n\t"
#define CINN_MMA_TS_STEP(B, A)                                                                                                      \
    "add.u32 x, %1, " A ";\n\tadd.u32 y, %2, " B ";\n\tmov.b64 b, {y, %4};\n\t"                                                     \
    "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [x], b, %3, 1;\n\t"
#define CINN_MMA_TS_ARGS ::"r"(d), "r"(a), "r"(b), "r"(idesc), "r"(DESC_HI), "r"(fresh ? 0u : 1u) : "memory"
    if constexpr (STEPS == 8 && X == 0)
        asm volatile(CINN_MMA_TS_FIRST CINN_MMA_TS_STEP("128", "8") CINN_MMA_TS_STEP("256", "16") CINN_MMA_TS_STEP("384", "24")
                         CINN_MMA_TS_STEP("512", "32") CINN_MMA_TS_STEP("640", "40") CINN_MMA_TS_STEP("768", "48")
                             CINN_MMA_TS_STEP("896", "56") "}" CINN_MMA_TS_ARGS);
    else if constexpr (STEPS == 8)
        asm volatile(CINN_MMA_TS_FIRST CINN_MMA_TS_STEP("128", "16") CINN_MMA_TS_STEP("256", "32") CINN_MMA_TS_STEP("384", "48")
                         CINN_MMA_TS_STEP("512", "64") CINN_MMA_TS_STEP("640", "80") CINN_MMA_TS_STEP("768", "96")
                             CINN_MMA_TS_STEP("896", "112") "}" CINN_MMA_TS_ARGS);
    else if constexpr (X == 0)
        asm volatile(CINN_MMA_TS_FIRST CINN_MMA_TS_STEP("128", "8") "}" CINN_MMA_TS_ARGS);
    else
        asm volatile(CINN_MMA_TS_FIRST CINN_MMA_TS_STEP("128", "16") "}" CINN_MMA_TS_ARGS);
#undef CINN_MMA_TS_FIRST
#undef CINN_MMA_TS_STEP
#undef CINN_MMA_TS_ARGS
}

}  // namespace atc
}  // namespace cinn
