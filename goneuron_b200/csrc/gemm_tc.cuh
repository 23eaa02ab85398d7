// gemm_tc.cuh -- fp32-accurate contraction on the 5th-generation tensor cores (sm_100a).
//
//   C[M,N] = act( A[M,K] * B[N,K]^T + bias[N] + R[M,N] )
//
// Split-operand scheme (three half-precision products per fp32 product).  Every operand row (one output row's or
// output column's K-vector) is first multiplied by a power of two s that brings its largest magnitude into
// [2^14, 2^15), and each scaled element is written as
//     x s = x0 + x1 + r,   x0 = fp16(x s),  x1 = fp16(x s - x0),  |r| <= 2^-22 |x s| + 2^-25
// (fp16 carries 11 significant bits, so two planes hold 22 of the 24 bits of an fp32 mantissa; elements far below the
// row's maximum land in fp16's subnormal range, where the absolute error 2^-25 is 2^-39 of the row's maximum).  Then
//     a*b  =  ( a0*b0  +  a0*b1 + a1*b0 ) / (s_a s_b)      (dropped: a1*b1, r_a*b, a*r_b -- each about 2^-22 |a b|).
// All three terms are tcgen05.mma.kind::f16 instructions with fp32 accumulation in tensor memory; a product of two
// fp16 numbers is exact in fp32, and the division by the two powers of two in the epilogue is exact.  Against the
// other ways of reaching fp32 accuracy on these tensor cores -- three TF32 instructions (6 units of tensor time per
// product, 8-byte operand planes), or one TF32 and two BF16 instructions (4 units, 8 bytes; what this file did
// before) -- this costs 3 units and the operand planes are 4 bytes per element, the size of the fp32 source.  That
// halves what the kernel pulls through L2 and shared memory, which matters because the kernel is bound by
// shared-memory bandwidth, not by the tensor pipe: with 128 x 128 tiles every MMA re-reads both operands from shared
// memory (8 KB per 64 tensor cycles = the full 128 B/clk) while TMA writes the next stage into the same memory.  The
// large-problem variant therefore uses 128 x 256 tiles (12 KB per 128 tensor cycles).
//
// The operand planes (K-major fp16, interleaved in blocks of 32 indices) and the per-row inverse scales are written
// by a memory-bound pass (split2_rows_kernel / split2_cols_kernel); the contraction kernel itself is a pure
// TMA -> shared memory -> tcgen05.mma pipeline:
//
//   warp 0   TMA producer: 3 tiled bulk copies per stage (128-byte rows, 128-byte swizzle; 3-D maps, third
//            coordinate = problem index of a batch)
//   warp 1   allocates TMEM, issues the MMAs (one elected lane), commits to mbarriers
//   warps 2-9  epilogue: tcgen05.ld of the accumulators, scales / bias / residual / ReLU / gate, whole 128-byte lines
//
// Persistent: one CTA per SM walks 128 x BN output tiles.  TMEM holds two accumulator slots, so the epilogue
// of tile i runs under the mainloop of tile i+1.  The tensor core truncates when it adds a group of products
// to the accumulator, an error proportional to the accumulator's magnitude per MMA instruction.  With BN = 64
// or 128 each slot therefore has two accumulators -- the a0*b0 products go to one, the small cross terms to
// the other, and the epilogue adds them -- and with BN = 256 (one accumulator per slot, 512 columns in all) the
// host cuts long contractions into shorter accumulator runs instead.
// Every mbarrier wait is bounded.  A wait that gives up sets the context's status word and a flag in shared
// memory; every role of the CTA then leaves its loops without issuing further copies or MMAs, the producer
// waits (bounded) for its copies in flight, the MMA role for its instructions in flight, and TMEM is released.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cstdlib>
#include "common.cuh"
#include "fmath.cuh"
#include "gemm_simt.cuh"

namespace gn {

constexpr int TC_BM = 128;
constexpr unsigned TC_SPIN_LIMIT = 1u << 24;    // default number of polls of one wait (Ctx::spin_limit overrides it)
constexpr unsigned TC_DRAIN_LIMIT = 1u << 20;   // polls spent waiting for own work in flight after a wait gave up
constexpr int TC_QUEUE_POOL = 2048;   // tile-queue counters per context before the pool is cleared again
constexpr int TC_FLAG_SCALE = 8192; // plane output: `mask` holds factors (a GELU layer's derivatives, all below 1.25), not a gate
constexpr int TC_FLAG_VEC = 4096;   // epilogue may use 16-byte accesses (set by the host when every pointer and stride allows it)
// One stage = 32 contraction indices of both operands.  The two fp16 planes of an operand are interleaved in blocks of 32:
// element (r, k) of a plane row has its high part at pl_off(k) and its low part PL_LO halves further, so a block of a row is 128
// contiguous bytes, one TMA copy brings both planes of a stage, and the tile has 128-byte rows (128-byte swizzle).  With separate
// planes and 64-byte rows (64-byte swizzle) every MMA took 141 cycles, whatever its width (128 x 128 x 16 needs 64 of arithmetic).
// With this, the issue loops in uniform registers and the epilogue below, [8192, 256] x [256, 256] went from 16.5 to 10.4 us,
// [8192, 1024] x [1024, 256] from 26.8 to 18.6, [32768, 1024] x [1024, 1024] from 136 to 119 (zeros as data: no power limit).
constexpr int TC_BK = 32, PL_LO = 32;
__host__ __device__ __forceinline__ int pl_off(int k) { return ((k >> 5) << 6) | (k & 31); }
// What a variant of the kernel writes: fp32 in 16-byte pieces or in NCHW order, operand planes, or rows of fp32 that 16-byte pieces do not fit (an odd number of columns).  (The
// last one's code beside the first one's cost every product 2 %; without the NCHW order's beside it 256-wide tiles were 0.3 us slower, [4096, 1000] over 256 11.5 -> 11.8.)  PL: planes.
enum TcOut { TC_OUT_VEC, TC_OUT_PLANES, TC_OUT_ROWS };
template <int BN, bool PL> struct TcCfg {
  static constexpr int EW = PL ? 16 : 8, CG = EW / 4, CC = PL ? 16 : 32;          // epilogue warps, column groups, columns of a chunk
  static constexpr int THREADS = 64 + 32 * EW;                                    // TMA warp, MMA warp, epilogue warps
  static constexpr int A_BYTES = TC_BM * 128, B_BYTES = BN * 128;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (192 * 1024) / STAGE_BYTES > 8 ? 8 : (192 * 1024) / STAGE_BYTES;
  static constexpr int STG_FLOATS = EW * 32 * CC;                                 // per epilogue warp: 32 rows x CC columns in transit
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/ + STG_FLOATS * 4;
  static constexpr bool MERGED = BN > 128;                                        // one accumulator per slot
  static constexpr int SLOT_COLS = MERGED ? BN : 2 * BN;
  static constexpr int TMEM_COLS = 2 * SLOT_COLS;
  static_assert(2 * STAGES + 6 <= 30, "barrier area");
  static_assert(TMEM_COLS <= 512, "accumulator slots must fit the 512 TMEM columns");
};

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded wait: returns false when it gave up -- after `limit` polls, or as soon as `*abort_flag` (a word in
// shared memory that a role of this CTA sets when one of its own waits gave up) is non-zero.  A poll is
// mbarrier.try_wait, which may suspend the thread for a while by itself; limits below 4096 poll with the
// non-suspending mbarrier.test_wait instead, so that a small limit really is a short time (the failure-detection
// tests rely on that to make a wait run out).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned limit = TC_SPIN_LIMIT, const volatile int* abort_flag = nullptr) {
  if (limit < 4096u) {
    for (unsigned it = 0; it < limit; it++) {
      uint32_t done;
      asm volatile("{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
      if (done) return true;
    }
    return false;
  }
  for (unsigned it = 0; it < limit; it++) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if (abort_flag && (it & 63) == 63 && *abort_flag) return false;
  }
  return false;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
// One lane of a converged warp, always the same one.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
               ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// Two consecutive products with the same A operand: the first leaves it in the tensor core's collector, the second takes it
// from there instead of reading shared memory again (128 x 128 tiles over 1024 indices: 20.4 -> 18.6 us).
__device__ __forceinline__ void tc_mma_f16_same_a(uint32_t d1, uint32_t d2, uint64_t adesc, uint64_t b1, uint64_t b2, uint32_t idesc, uint32_t acc1, uint32_t acc2) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %6, 0;\nsetp.ne.b32 q, %7, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16.collector::a::fill [%0], %2, %3, %5, p;\n"
               "tcgen05.mma.cta_group::1.kind::f16.collector::a::lastuse [%1], %2, %4, %5, q;\n}"
               ::"r"(d1), "r"(d2), "l"(adesc), "l"(b1), "l"(b2), "r"(idesc), "r"(acc1), "r"(acc2) : "memory");
}
// Shared-memory matrix descriptor, K-major operand, 128-byte swizzle: rows are 128 bytes apart, groups of 8
// rows 1024 bytes apart (stride byte offset), descriptor version 1 (sm_100), layout type 2 = SWIZZLE_128B.
template <int BK>
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {
  constexpr uint64_t sbo = (8 * BK * 4) >> 4, layout = BK == 32 ? 2 : 4;
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (1ull << 16) | (sbo << 32) | (1ull << 46) | (layout << 61);
}
// Instruction descriptor of kind::f16 with A = B = fp16 (format code 0 at bits 7-9 and 10-12), D = f32 (bits 4-5 = 1), both
// operands K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28.
__host__ __device__ constexpr uint32_t make_idesc_f16(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
        "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
        "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}


__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
        "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}

// ------------------------------------------------------------------ splitting a value into operand planes
// Power of two s that brings a row whose largest magnitude is mx into [2^14, 2^15) (fp16 overflows at 65504), and its
// inverse.  s = 1 for a row of zeros (and for a row that holds an infinity or a NaN, which the products then carry on).
__device__ __forceinline__ float row_scale(float mx, float* inv) {
  if (!(mx > 0.f) || !(mx <= 3.0e38f)) { *inv = 1.f; return 1.f; }
  int se = 14 - (((__float_as_int(mx) >> 23) & 0xff) - 127);
  se = max(-100, min(100, se));
  *inv = __int_as_float((127 - se) << 23); return __int_as_float((127 + se) << 23);
}
// (x s) -> (fp16(x s), fp16(x s - fp16(x s))) for two neighbouring elements, packed
__device__ __forceinline__ void split2_pair(float a, float b, float s, uint32_t& p0, uint32_t& p1) {
  a *= s; b *= s;
  const __half2 h = __floats2half2_rn(a, b);
  const float2 hf = __half22float2(h);
  const __half2 l = __floats2half2_rn(a - hf.x, b - hf.y);
  p0 = *reinterpret_cast<const uint32_t*>(&h); p1 = *reinterpret_cast<const uint32_t*>(&l);
}

// Output side of one launch.  Batched problems: problem z -> (z / batch2, z % batch2) selects the
// output (and residual) sub-matrix; the operand planes of problem z are slice z of the 3-D tensor maps.
struct TcParams {
  float* C; long ldc, c_b1, c_b2; const float* bias; const float* R; long ldr, r_b1, r_b2;
  int act, M, N, K, batch2, flags; int* status;
  const float* mask; long mask_ld; int mask_group;    // optional gate, see GemmDesc::mask
  const float* isa = nullptr; const float* isb = nullptr;   // inverse row scales of the operand planes: [nbatch][M], [nbatch][N]
  unsigned spin_limit = TC_SPIN_LIMIT;                // polls per wait before the kernel gives up
  int nchw_P = 0;      // > 0: output row r = (sample r / P, position r % P) is stored as C[sample][col][position] (N channels of P positions)
  // Plane output (out_p != null): the result is not stored as fp32 but directly as the operand planes of the next
  // contraction (two interleaved fp16 planes [M][2 out_ldp] and an inverse scale per row), see TcPlaneOut.  C may then be null.
  __half* out_p = nullptr; float* out_inv = nullptr; long out_ldp = 0;
  const float* a_rownorm = nullptr; const int* b_maxabs = nullptr;     // the bound's factors: |row of A|_2 and max |entry of B (and bias)| as float bits
  float* c_last = nullptr; int last_T = 0;                             // fp32 copy of the rows r with r % last_T == last_T - 1: c_last[(r / last_T) * N + col]
  float* z_last = nullptr;                                             // ... and of their values before the activation
  int n_seg = 0; long c_seg = 0, bias_seg = 0;                         // > 0 (a multiple of 32): columns j n_seg .. lie c_seg (biases: bias_seg) floats after those of segment j - 1, see GemmDesc::n_seg
  int* zmax = nullptr; int zmax_T = 0, zmax_H = 0; long zmax_seg = 0;  // receives the largest magnitude per (segment, sequence of zmax_T rows, head of 64 columns), see attn_tc_max_words
  int k_slice = 0, splits = 1;                                         // k_slice > 0 (a multiple of 32): z is not a problem but a slice of the contraction, C + z c_b1 its partial result
  const int* z_first = nullptr;                                        // problems (i, j) with j < z_first[i] are left out
  float* rowsum32 = nullptr;                                           // plane output: sums of the result over every 32 consecutive rows, [ceil(M / 32)][N]
};

// Epilogue of one output tile.  8 or 16 warps share it: a warp may only read the TMEM lanes of its quadrant (warp % 4), so
// two or four warps serve each quadrant and take a part of the tile's columns each (`cg`), in chunks of TcCfg::CC.  tcgen05.ld gives a
// thread consecutive columns of one output row (TMEM lane = row); the chunk goes through `stg`, the warp's staging buffer of 32 rows
// (16-byte units swizzled by the row: no bank conflicts either way), and comes back with eight (planes: four) neighbouring lanes on
// a row and four columns of eight (four) rows per lane.  From there on an access to global memory touches four lines of 128 bytes (eight half
// lines).  A chunk's column factors and residual, and for planes the gate where 32 rows have two gate rows at most (mask_group >= 32), are
// fetched while the chunk before it is stored, the first chunk's before the accumulator is waited for; any other gate is read where it is applied.
// (A thread that kept the row TMEM gave it and moved whole 32-byte sectors of it touched 32 lines per instruction: 1700 cycles to
// store a chunk, 13 bytes per clock and SM; 9000 cycles for a 128 x 128 tile with a residual, as much as its MMAs over 384.  Now
// about 4500.  [3072, 512] over 512 with a residual 13.7 -> 11.4 us, [3072, 1536] over 512 16.9 -> 15.5; as planes [3072, 2048] over
// 512 23.6 -> 21.5, [3600, 1536] over 384 gated by factors 23.3 -> 20.1, with GELU 29.1 -> 28.4.  Where the main loop hides the epilogue the
// exchange takes shared-memory bandwidth from it: [16384, 1024] over 1024 77.6 -> 78.5, [32768, 3072] over 1024 431 -> 432.)
// fp32 results go best with eight warps and unrolled rows; planes take twice the arithmetic per element and 16 warps (with eight,
// GELU: 35 us).  The loops over chunks are not unrolled: a launch with one tile per CTA runs this code once, from a cold instruction cache.
// acc[j] of column j of a chunk for this lane's row, times the row's inverse scale
template <bool MERGED, int CC>
__device__ __forceinline__ void tc_acc_chunk(uint32_t taddr, uint32_t acc_main, uint32_t acc_cross, bool any, float isa, float (&v)[CC]) {
  if (any) {
    uint32_t r[CC], q[MERGED ? 1 : CC];
    if constexpr (CC == 32) { tmem_ld32(taddr + acc_main, r); if constexpr (!MERGED) tmem_ld32(taddr + acc_cross, q); }
    else { tmem_ld16(taddr + acc_main, r); if constexpr (!MERGED) tmem_ld16(taddr + acc_cross, q); }
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < CC; j++) {
      if constexpr (MERGED) v[j] = __uint_as_float(r[j]) * isa; else v[j] = (__uint_as_float(r[j]) + __uint_as_float(q[j])) * isa;
    }
  } else {
#pragma unroll
    for (int j = 0; j < CC; j++) v[j] = 0.f;
  }
}
// `acc_main` / `acc_cross` are the TMEM column offsets of the two accumulators of this tile (MERGED: there is only acc_main); `bw` is the
// tile's width (BN, or BN / 2 for a half tile).  `wait` blocks until the accumulator is complete; false: it gave up.
template <int BN, TcOut OUT, bool MERGED, class W>
__device__ __forceinline__ bool tc_epilogue_tile(const TcParams& ep, uint32_t tmem_base, uint32_t acc_main, uint32_t acc_cross,
                                                 int m0, int n0, int z, int quad, int cg, int lane, int nkb, int bw, float* stg, W&& wait) {
  constexpr bool PL = OUT == TC_OUT_PLANES; using Cfg = TcCfg<BN, PL>;
  const int z1 = z / ep.batch2, z2 = z - z1 * ep.batch2, nch = max(bw / (Cfg::CC * Cfg::CG), 1);      // chunks per warp
  if (cg * nch * Cfg::CC >= bw) return wait();                               // a narrow tile has fewer chunks than column groups
  const int rbase = m0 + quad * 32, row = rbase + lane, c_end = min(cg * nch + nch, (ep.N - n0 + Cfg::CC - 1) / Cfg::CC);
  const bool row_ok = row < ep.M;
  const uint32_t tquad = tmem_base + ((uint32_t)(quad * 32) << 16);
  const float isa = row_ok ? ep.isa[(ep.k_slice ? 0L : (long)z * ep.M) + row] : 1.f;             // 1 / (scale of this row's A vector), a power of two
  const float* isb = ep.isb + (ep.k_slice ? 0L : (long)z * ep.N);
  if constexpr (PL) {
    // Plane output: the result becomes the next contraction's A operand.  Twice the work per element (activation or factors, scale,
    // two conversions): 16 warps, chunks of 16 columns, after the exchange four lanes on a row.
    const int rl = lane >> 2, c4 = lane & 3, r0 = rbase + rl;                // this lane's rows r0 + 8 t and columns 4 c4 .. 4 c4 + 3 of a chunk
    const bool few = ep.mask_group >= 32;                                    // 32 rows belong to two sequences at most: their gates are fetched ahead
    const int g0 = ep.mask ? rbase / ep.mask_group : 0, g_next = ep.mask ? (g0 + 1) * ep.mask_group : 0;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f); float4 sv = zero, bv = zero, k0 = zero, k1 = zero;
    auto fetch = [&](int c) {
      const int col = n0 + c * 16 + 4 * c4; if (c >= c_end) return;          // (N is a multiple of 32)
      sv = __ldg(reinterpret_cast<const float4*>(isb + col)); if (ep.bias) bv = __ldg(reinterpret_cast<const float4*>(ep.bias + col));
      if (ep.mask && few) {
        const float* q = ep.mask + (long)g0 * ep.mask_ld + col;
        if (rbase < ep.M) k0 = __ldg(reinterpret_cast<const float4*>(q));
        if (g_next < min(rbase + 32, ep.M)) k1 = __ldg(reinterpret_cast<const float4*>(q + ep.mask_ld));
      }
    };
    fetch(cg * nch);
    float osc = 1.f;                                                         // the scale of row `row`
    if (row_ok) {
      const float an = ep.a_rownorm[row], bound = sqrtf(fmaf(an, an, 1.f)) * sqrtf((float)ep.K + 1.f) * __int_as_float(*ep.b_maxabs);
      float oinv; osc = row_scale(ep.flags & TC_FLAG_SCALE ? 1.25f * bound : bound, &oinv);
      if (n0 == 0 && cg == 0) ep.out_inv[row] = oinv;
    }
    const unsigned last = ep.c_last ? __ballot_sync(0xffffffffu, row_ok && row % ep.last_T == ep.last_T - 1) >> rl : 0u;      // bit 8 t: row r0 + 8 t is a sequence's last
    if (!wait()) return false;
#pragma unroll 1
    for (int c = cg * nch; c < c_end; c++) {
      const int col = n0 + c * 16 + 4 * c4;
      {
        float v[16]; tc_acc_chunk<MERGED, 16>(tquad + c * 16, acc_main, acc_cross, nkb > 0, isa, v);
        __syncwarp();                                                        // the previous chunk has been read back
#pragma unroll
        for (int j = 0; j < 4; j++) *reinterpret_cast<float4*>(stg + lane * 16 + ((j ^ (lane >> 1 & 3)) << 2)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        __syncwarp();
      }
      float4 a[4];
#pragma unroll
      for (int t = 0; t < 4; t++) { const int r = 8 * t + rl; a[t] = *reinterpret_cast<const float4*>(stg + r * 16 + ((c4 ^ (r >> 1 & 3)) << 2)); }
#pragma unroll
      for (int t = 0; t < 4; t++) a[t] = make_float4(a[t].x * sv.x + bv.x, a[t].y * sv.y + bv.y, a[t].z * sv.z + bv.z, a[t].w * sv.w + bv.w);
      if (ep.act == GN_ACT_RELU) {
#pragma unroll
        for (int t = 0; t < 4; t++) a[t] = make_float4(fmaxf(a[t].x, 0.f), fmaxf(a[t].y, 0.f), fmaxf(a[t].z, 0.f), fmaxf(a[t].w, 0.f));
      } else if (ep.act == GN_ACT_GELU) {
        if (last && ep.z_last) {
#pragma unroll
          for (int t = 0; t < 4; t++) if (last >> (8 * t) & 1) *reinterpret_cast<float4*>(ep.z_last + (long)((r0 + 8 * t) / ep.last_T) * ep.N + col) = a[t];
        }
#pragma unroll
        for (int t = 0; t < 4; t++) a[t] = make_float4(gelu_f(a[t].x), gelu_f(a[t].y), gelu_f(a[t].z), gelu_f(a[t].w));
      }
      if (ep.mask) {
        float4 m[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
          const int r = r0 + 8 * t;
          m[t] = few ? (r < g_next ? k0 : k1) : r < ep.M ? *reinterpret_cast<const float4*>(ep.mask + (long)(r / ep.mask_group) * ep.mask_ld + col) : zero;
        }
#pragma unroll
        for (int t = 0; t < 4; t++) {
          if (ep.flags & TC_FLAG_SCALE) { a[t].x *= m[t].x; a[t].y *= m[t].y; a[t].z *= m[t].z; a[t].w *= m[t].w; }
          else { if (!(m[t].x > 0.f)) a[t].x = 0.f; if (!(m[t].y > 0.f)) a[t].y = 0.f; if (!(m[t].z > 0.f)) a[t].z = 0.f; if (!(m[t].w > 0.f)) a[t].w = 0.f; }
        }
      }
      fetch(c + 1);                                                          // under this chunk's conversions and stores
      if (last) {
#pragma unroll
        for (int t = 0; t < 4; t++) if (last >> (8 * t) & 1) *reinterpret_cast<float4*>(ep.c_last + (long)((r0 + 8 * t) / ep.last_T) * ep.N + col) = a[t];
      }
      __half* o = ep.out_p + (long)r0 * 2 * ep.out_ldp + pl_off(col); float4 u = zero;
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const float sc = __shfl_sync(0xffffffffu, osc, 8 * t + rl);
        uint2 hi, lo; split2_pair(a[t].x, a[t].y, sc, hi.x, lo.x); split2_pair(a[t].z, a[t].w, sc, hi.y, lo.y);
        if (r0 + 8 * t < ep.M) {
          __half* q = o + (long)(16 * t) * ep.out_ldp; *reinterpret_cast<uint2*>(q) = hi; *reinterpret_cast<uint2*>(q + PL_LO) = lo;
          u.x += a[t].x; u.y += a[t].y; u.z += a[t].z; u.w += a[t].w;
        }
      }
      if (ep.rowsum32) {
        // the consumer of a plane output's token sums (the weight gradient of the layer below) gets them from here instead of
        // re-reading the planes: the sum of every column over the warp's rows, in a fixed order
#pragma unroll
        for (int h = 4; h < 32; h <<= 1) {
          u.x += __shfl_xor_sync(0xffffffffu, u.x, h); u.y += __shfl_xor_sync(0xffffffffu, u.y, h);
          u.z += __shfl_xor_sync(0xffffffffu, u.z, h); u.w += __shfl_xor_sync(0xffffffffu, u.w, h);
        }
        if (rl == 0 && rbase < ep.M) *reinterpret_cast<float4*>(ep.rowsum32 + (long)(rbase >> 5) * ep.N + col) = u;
      }
    }
    __syncwarp();
    return true;
  }
  float* C = ep.C + z1 * ep.c_b1 + z2 * ep.c_b2;
  const float* R = ep.R ? ep.R + z1 * ep.r_b1 + z2 * ep.r_b2 : nullptr;
  if (OUT == TC_OUT_VEC && (ep.flags & TC_FLAG_VEC)) {
    const int rl = lane >> 3, c8 = lane & 7, r0 = rbase + rl;                // after the exchange: this lane's rows r0 + 4 t and columns 4 c8 .. 4 c8 + 3 of a chunk
    float4 sv, bv, rv[8];                                                    // what the next chunk needs for them
    auto fetch = [&](int c) {
      const int col = n0 + c * 32 + 4 * c8; const bool ok = c < c_end && col < ep.N; const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      const int seg = ep.n_seg && ok ? col / ep.n_seg : 0;                   // (32 columns lie in one segment)
      sv = ok ? __ldg(reinterpret_cast<const float4*>(isb + col)) : zero;
      bv = ok && ep.bias ? __ldg(reinterpret_cast<const float4*>(ep.bias + col + (long)seg * (ep.bias_seg - ep.n_seg))) : zero;
      const float* q = R ? R + (long)seg * (ep.c_seg - ep.n_seg) + (long)r0 * ep.ldr + col : nullptr;      // (with segments R is C)
#pragma unroll
      for (int t = 0; t < 8; t++) rv[t] = R && ok && r0 + 4 * t < ep.M ? *reinterpret_cast<const float4*>(q + (long)(4 * t) * ep.ldr) : zero;
    };
    fetch(cg * nch);
    if (!wait()) return false;
#pragma unroll 1
    for (int c = cg * nch; c < c_end; c++) {
      const int col = n0 + c * 32 + 4 * c8; const bool col_ok = col < ep.N;
      {
        float v[32]; tc_acc_chunk<MERGED, 32>(tquad + c * 32, acc_main, acc_cross, nkb > 0, isa, v);
        __syncwarp();                                                        // the previous chunk has been read back
#pragma unroll
        for (int j = 0; j < 8; j++) *reinterpret_cast<float4*>(stg + lane * 32 + ((j ^ (lane & 7)) << 2)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        __syncwarp();
      }
      float4 a[8];
#pragma unroll
      for (int t = 0; t < 8; t++) { const int r = 4 * t + rl; a[t] = *reinterpret_cast<const float4*>(stg + r * 32 + ((c8 ^ (r & 7)) << 2)); }
#pragma unroll
      for (int t = 0; t < 8; t++) a[t] = make_float4(a[t].x * sv.x + bv.x + rv[t].x, a[t].y * sv.y + bv.y + rv[t].y, a[t].z * sv.z + bv.z + rv[t].z, a[t].w * sv.w + bv.w + rv[t].w);
      fetch(c + 1);                                                          // under this chunk's stores
      if (ep.act == GN_ACT_RELU) {
#pragma unroll
        for (int t = 0; t < 8; t++) a[t] = make_float4(fmaxf(a[t].x, 0.f), fmaxf(a[t].y, 0.f), fmaxf(a[t].z, 0.f), fmaxf(a[t].w, 0.f));
      }
      if (ep.mask && col_ok) {
        float4 m[8];
#pragma unroll
        for (int t = 0; t < 8; t++) m[t] = r0 + 4 * t < ep.M ? *reinterpret_cast<const float4*>(ep.mask + (long)((r0 + 4 * t) / ep.mask_group) * ep.mask_ld + col) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int t = 0; t < 8; t++) { if (!(m[t].x > 0.f)) a[t].x = 0.f; if (!(m[t].y > 0.f)) a[t].y = 0.f; if (!(m[t].z > 0.f)) a[t].z = 0.f; if (!(m[t].w > 0.f)) a[t].w = 0.f; }
      }
      const int seg = ep.n_seg ? col / ep.n_seg : 0; float* o = C + (long)seg * (ep.c_seg - ep.n_seg) + (long)r0 * ep.ldc + col;
      float zm = 0.f;
#pragma unroll
      for (int t = 0; t < 8; t++) if (col_ok && r0 + 4 * t < ep.M) {
        *reinterpret_cast<float4*>(o + (long)(4 * t) * ep.ldc) = a[t];
        zm = fmaxf(zm, fmaxf(fmaxf(fabsf(a[t].x), fabsf(a[t].y)), fmaxf(fabsf(a[t].z), fabsf(a[t].w))));
      }
      if (ep.zmax) {                                                         // (32 rows of one sequence, 32 columns of one head)
        zm = warp_max(zm); if (!(zm <= 3.0e38f)) zm = 3.4e38f;
        const int c32 = n0 + c * 32, sg = c32 / ep.n_seg;
        if (lane == 0 && rbase < ep.M) atomicMax(ep.zmax + sg * ep.zmax_seg + (long)(rbase / ep.zmax_T) * ep.zmax_H + (c32 - sg * ep.n_seg) / 64, __float_as_int(zm));
      }
    }
    __syncwarp();
    return true;
  }
  if constexpr (OUT == TC_OUT_ROWS) {
    // rows that 16-byte accesses do not fit (an odd number of columns): through the staging buffer all the same, then a row at a time, a column per lane.
    // (A row per lane, a column at a time, touched 32 lines per instruction: [2048, 1001] over 256 29 -> 16 us.)
    if (!wait()) return false;
#pragma unroll 1
    for (int c = cg * nch; c < c_end; c++) {
      const int col = n0 + c * 32 + lane; const bool col_ok = col < ep.N; const int seg = ep.n_seg ? (n0 + c * 32) / ep.n_seg : 0;      // (32 columns lie in one segment)
      const float sv = col_ok ? __ldg(isb + col) : 0.f, bv = col_ok && ep.bias ? __ldg(ep.bias + col + (long)seg * (ep.bias_seg - ep.n_seg)) : 0.f;
      {
        float v[32]; tc_acc_chunk<MERGED, 32>(tquad + c * 32, acc_main, acc_cross, nkb > 0, isa, v);
        __syncwarp();                                                        // the previous chunk has been read back
#pragma unroll
        for (int j = 0; j < 8; j++) *reinterpret_cast<float4*>(stg + lane * 32 + ((j ^ (lane & 7)) << 2)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        __syncwarp();
      }
      const long off = (long)seg * (ep.c_seg - ep.n_seg) + col; float* o = C + off; const float* q = R ? R + off : nullptr;      // (with segments R is C)
#pragma unroll 1
      for (int r4 = 0; r4 < 32; r4 += 4) {
        float a[4];
#pragma unroll
        for (int t = 0; t < 4; t++) {
          const int r = r4 + t; const bool ok = col_ok && rbase + r < ep.M;
          a[t] = stg[r * 32 + ((((lane >> 2) ^ (r & 7)) << 2) | (lane & 3))] * sv + bv + (q && ok ? q[(long)(rbase + r) * ep.ldr] : 0.f);
          if (ep.act == GN_ACT_RELU) a[t] = fmaxf(a[t], 0.f);
          if (ep.mask && ok && !(ep.mask[(long)((rbase + r) / ep.mask_group) * ep.mask_ld + col] > 0.f)) a[t] = 0.f;
        }
#pragma unroll
        for (int t = 0; t < 4; t++) if (col_ok && rbase + r4 + t < ep.M) o[(long)(rbase + r4 + t) * ep.ldc] = a[t];
      }
    }
    __syncwarp();
    return true;
  }
  if (!wait()) return false;
  // NCHW store: one output row per thread
  float* Crow = C + (long)(row / ep.nchw_P) * ep.N * ep.nchw_P + row % ep.nchw_P;
#pragma unroll 1
  for (int cc = 0; cc < nch; cc++) {
    const int col0 = n0 + (cg * nch + cc) * 32;
    if (col0 >= ep.N) break;
    float v[32]; tc_acc_chunk<MERGED, 32>(tquad + (cg * nch + cc) * 32, acc_main, acc_cross, nkb > 0, isa, v);
#pragma unroll
    for (int j = 0; j < 32; j++) {
      const int col = col0 + j;
      if (!row_ok || col >= ep.N) continue;
      float x = v[j] * isb[col];
      if (ep.bias) x += ep.bias[col];
      if (ep.act == GN_ACT_RELU) x = fmaxf(x, 0.f);
      Crow[(long)col * ep.nchw_P] = x;
    }
  }
  return true;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

template <int BN, TcOut OUT>
__global__ void __launch_bounds__(TcCfg<BN, OUT == TC_OUT_PLANES>::THREADS, 1)
gemm_tc_persist_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const __grid_constant__ TcParams ep, int tiles_m, int tiles_n, int total_tiles, int full_end, int n_half, int* tile_queue) {
  using Cfg = TcCfg<BN, OUT == TC_OUT_PLANES>;
  constexpr int STAGES = Cfg::STAGES, STAGE_BYTES = Cfg::STAGE_BYTES, BK = TC_BK;
  constexpr bool MERGED = Cfg::MERGED;
  constexpr uint32_t TMEM_COLS = Cfg::TMEM_COLS, SLOT_COLS = Cfg::SLOT_COLS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = (uint64_t*)(smem + STAGES * STAGE_BYTES);       // full[S], empty[S], tfull[2], tempty[2], drain
  uint32_t* tmem_slot = (uint32_t*)(bars + 2 * STAGES + 5);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);       // set by the first role whose wait gave up
  uint64_t* qbars = bars + 2 * STAGES + 6;                         // tile queue: qfull[4], qempty[4], then the four queued items
  volatile int* qitem = (volatile int*)(qbars + 8);
  const uint32_t qfull0 = smem_u32(qbars), qempty0 = smem_u32(qbars + 4);
  float* stg_all = (float*)(smem + STAGES * STAGE_BYTES + 256);    // epilogue warps' staging buffers
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + STAGES), tfull0 = smem_u32(bars + 2 * STAGES), tempty0 = smem_u32(bars + 2 * STAGES + 2);
  const uint32_t drain = smem_u32(bars + 2 * STAGES + 4);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (warp-uniform for the compiler, too)
  const uint32_t smem0 = smem_u32(smem);
  constexpr uint32_t OFF_B = Cfg::A_BYTES;                         // stage layout: A | B, rows of hi 32 | lo 32
  const unsigned limit = ep.spin_limit;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mapA) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&mapB) : "memory");
    for (int s = 0; s < STAGES; s++) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
    for (int b = 0; b < 2; b++) { mbar_init(tfull0 + 8 * b, 1); mbar_init(tempty0 + 8 * b, Cfg::EW); }
    mbar_init(drain, 1);
    for (int b = 0; b < 4; b++) { mbar_init(qfull0 + 8 * b, 1); mbar_init(qempty0 + 8 * b, 1 + Cfg::EW); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // Work list of this CTA (identical in every role): tiles blockIdx.x, + gridDim.x, ... below full_end; then, when the
  // tiles left over would occupy at most half of the CTAs (n_half = twice their number, else 0), one HALF of a left-over
  // tile each (BN / 2 columns), so that the last, short round costs about 0.6 instead of 1 tile time.
  // a wait gave up: record which role, and tell the other roles of this CTA to stop
  auto give_up = [&](int code) { atomicExch(ep.status, code); *abort_flag = 1; __threadfence_block(); };
  auto item = [&](long t, int& tile, int& half) -> bool {
    if (t < full_end) { tile = (int)t; half = -1; return true; }
    const long h = t - full_end;
    if (h >= n_half) return false;
    tile = full_end + (int)(h >> 1); half = (int)(h & 1); return true;
  };
  // With a tile queue (tile_queue != null: a zeroed counter in global memory) the producer thread draws the items with
  // atomicAdd and hands each to the MMA thread and the epilogue warps through a four-entry ring in shared memory, so a
  // CTA that gets its SM late (other kernels -- the collectives of a multi-GPU step -- holding SMs when the launch
  // starts) simply finds less left to do, instead of the whole launch waiting for its fixed share.
  const bool queued = tile_queue != nullptr;
  auto work = [&](int k, int& tile, int& half) -> bool {
    if (!queued) return item((long)blockIdx.x + (long)k * gridDim.x, tile, half);
    const uint32_t qs = (uint32_t)k & 3, qu = (uint32_t)k >> 2; int t = -1;
    if (lane == 0) {
      if (warp == 0) {                                    // producer: draw and publish
        if (qu > 0 && !mbar_wait(qempty0 + 8 * qs, (qu - 1) & 1, limit, abort_flag)) { if (!*abort_flag) give_up(4); t = -2; }
        else {
          t = atomicAdd(tile_queue, 1);
          if ((long)t >= (long)full_end + n_half) t = -1;
          qitem[qs] = t;
          mbar_arrive(qfull0 + 8 * qs);
        }
      } else if (mbar_wait(qfull0 + 8 * qs, qu & 1, limit, abort_flag)) { t = qitem[qs]; mbar_arrive(qempty0 + 8 * qs); }      // consumers: one thread per warp reads
      else if (!*abort_flag) give_up(5);
    }
    t = __shfl_sync(0xffffffffu, t, 0);
    return t >= 0 && item(t, tile, half);
  };
  // tile -> coordinates and contraction range
  auto decode = [&](int tile, int half, int& m0, int& n0, int& z, int& kb0, int& nkb) -> bool {
    const int nt = tile % tiles_n, q = tile / tiles_n, mt = q % tiles_m; z = q / tiles_m;
    m0 = mt * TC_BM; n0 = nt * BN + (half > 0 ? BN / 2 : 0);
    if ((ep.flags & GEMM_SKIP_UPPER) && n0 > m0 + TC_BM - 1) return false;
    if (ep.z_first && z % ep.batch2 < ep.z_first[z / ep.batch2]) return false;
    int kbeg = 0, kend = ep.K;
    if (ep.k_slice) { kbeg = z * ep.k_slice; kend = min(ep.K, kbeg + ep.k_slice); }
    if (ep.flags & GEMM_KBEG_AT_M0) kbeg = (m0 / BK) * BK;
    if (ep.flags & GEMM_KEND_AT_M0) kend = min(ep.K, m0 + TC_BM);
    kb0 = kbeg / BK; nkb = (kend - kbeg + BK - 1) / BK;
    return true;
  };

  // The producer and the MMA warp run their loops with all lanes and issue from one elected lane: the loop state then lives in
  // uniform registers.  With `if (lane == 0)` around the loops every MMA took its issuing thread 70 cycles (descriptors moved to
  // uniform registers one word at a time) and every stage 400 more, 820 cycles per stage whatever the tile's width.
  uint32_t issued = 0;          // producer: stages whose copies it has started
  const bool elected = elect_one();
  if (warp == 0) {
    bool ok = true; uint32_t s = 0, ph = 0;                   // next stage and the parity of its previous use
    int tile, half;
    for (int w = 0; ok && work(w, tile, half); w++) {
      int m0, n0, z, kb0, nkb; if (!decode(tile, half, m0, n0, z, kb0, nkb)) continue;
      if (ep.k_slice) z = 0;
      for (int i = 0; i < nkb; i++) {
        const int kc = 2 * (kb0 + i) * BK;
        if (issued >= (uint32_t)STAGES && !mbar_wait(empty0 + 8 * s, ph ^ 1, limit, abort_flag)) { ok = false; break; }
        if (elected) {
          const uint32_t base = smem0 + s * STAGE_BYTES, bar = full0 + 8 * s;
          mbar_expect_tx(bar, half < 0 ? STAGE_BYTES : STAGE_BYTES - Cfg::B_BYTES / 2);
          tma_load_3d(base, &mapA, kc, m0, z, bar);
          tma_load_3d(base + OFF_B, &mapB, kc, n0, z, bar);        // the B copies are BN / 2 rows each
          if (half < 0) tma_load_3d(base + OFF_B + Cfg::B_BYTES / 2, &mapB, kc, n0 + BN / 2, z, bar);
        }
        issued++;
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
    if (!ok && !*abort_flag) give_up(1);
    __syncwarp();
  } else if (warp == 1) {
    bool ok = true; uint32_t s = 0, ph = 0, lt = 0;
    constexpr uint32_t idesc_full = make_idesc_f16(TC_BM, BN), idesc_half = make_idesc_f16(TC_BM, BN / 2);
    const uint64_t desc0 = make_desc<32>(smem0);
    int tile, half;
    for (int w = 0; ok && work(w, tile, half); w++) {
      int m0, n0, z, kb0, nkb; if (!decode(tile, half, m0, n0, z, kb0, nkb)) continue;
      const uint32_t idesc = half < 0 ? idesc_full : idesc_half;
      const uint32_t slot = lt & 1, u = lt >> 1; lt++;
      if (!mbar_wait(tempty0 + 8 * slot, (u & 1) ^ 1, limit, abort_flag)) { ok = false; break; }     // slot drained by the epilogue (passes at once the first time)
      tc_fence_after();
      const uint32_t acc_main = tmem_base + slot * SLOT_COLS, acc_cross = MERGED ? acc_main : acc_main + BN;
      for (int i = 0; i < nkb; i++) {
        if (!mbar_wait(full0 + 8 * s, ph, limit, abort_flag)) { ok = false; break; }
        tc_fence_after();
        if (elected) {
          const uint64_t a0 = desc0 + (uint64_t)(s * (STAGE_BYTES >> 4)), b0 = a0 + (OFF_B >> 4), a1 = a0 + 4, b1 = b0 + 4;      // the low parts lie 64 bytes along the row
#pragma unroll
          for (int k = 0; k < 2; k++) {                      // 16 contraction indices = 32 bytes per instruction
            const uint64_t adv = (uint64_t)(2 * k);
            if constexpr (MERGED) {
              // small terms first, so that they meet the accumulator before the large term of this group is added
              tc_mma_f16(acc_main, a1 + adv, b0 + adv, idesc, (i > 0 || k > 0) ? 1u : 0u);
              tc_mma_f16_same_a(acc_main, acc_main, a0 + adv, b1 + adv, b0 + adv, idesc, 1u, 1u);
            } else {
              tc_mma_f16(acc_cross, a1 + adv, b0 + adv, idesc, (i > 0 || k > 0) ? 1u : 0u);
              tc_mma_f16_same_a(acc_cross, acc_main, a0 + adv, b1 + adv, b0 + adv, idesc, 1u, (i > 0 || k > 0) ? 1u : 0u);
            }
          }
          tc_commit(empty0 + 8 * s);
          if (i == nkb - 1) tc_commit(tfull0 + 8 * slot);
        }
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
      if (ok && nkb == 0 && elected) tc_commit(tfull0 + 8 * slot);
    }
    if (!ok) {
      if (!*abort_flag) give_up(2);
      if (elected) { tc_commit(drain); mbar_wait(drain, 0, TC_DRAIN_LIMIT); }      // own instructions in flight must finish before TMEM is released
    }
    __syncwarp();
  } else {
    const int quad = warp & 3, cg = (warp - 2) >> 2; uint32_t lt = 0;
    float* stg = stg_all + (warp - 2) * 32 * Cfg::CC;
    int tile, half;
    for (int w = 0; work(w, tile, half); w++) {
      int m0, n0, z, kb0, nkb; if (!decode(tile, half, m0, n0, z, kb0, nkb)) continue;
      const uint32_t slot = lt & 1, u = lt >> 1; lt++;
      const int bw = half < 0 ? BN : BN / 2;
      const bool ok = tc_epilogue_tile<BN, OUT, MERGED>(ep, tmem_base, slot * SLOT_COLS, slot * SLOT_COLS + BN, m0, n0, z, quad, cg, lane, nkb, bw, stg, [&]() -> bool {
        int got = 1;
        if (lane == 0) got = mbar_wait(tfull0 + 8 * slot, u & 1, limit, abort_flag) ? 1 : 0;
        got = __shfl_sync(0xffffffffu, got, 0);
        tc_fence_after(); return got != 0;
      });
      if (!ok) { if (lane == 0 && !*abort_flag) give_up(3); break; }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty0 + 8 * slot);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0 && elected && *abort_flag) {
    // a wait gave up somewhere in this CTA: the producer's last copies may still be in flight and nobody consumes
    // them any more; the CTA must not exit (and hand its shared memory on) before they have landed
    const uint32_t n_back = issued < (uint32_t)STAGES ? issued : (uint32_t)STAGES;
    for (uint32_t j = issued - n_back; j < issued; j++) mbar_wait(full0 + 8 * (j % STAGES), (j / STAGES) & 1, TC_DRAIN_LIMIT);
  }
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

// ------------------------------------------------------------------ operand split (memory-bound)
// Batched, strided split: planes[z][r][c] (row stride ldp, c < ldp, zero beyond cols) of the source element
// (z, r, c) at p + (z / batch2) * b1 + (z % batch2) * b2 + r * s_r + c * s_c.  One of s_r, s_c is 1:
// s_c == 1 reads rows directly; s_r == 1 (the operand is the transpose of what is stored) goes through a shared tile.
// Two fp16 planes per operand, fp16(x s) and fp16(x s - fp16(x s)), interleaved (pl_off), and the inverse 1/s of every plane row's scale.
// Rows may consist of segments of `seg` elements (> 0, a multiple of 32), each `seg_stride` floats after the one before: column c at
// p + r * s_r + c % seg + (c / seg) * seg_stride.
// Problem z is left out if z % batch2 < first[z / batch2] (rows split as they lie only).
struct TcSrc { const float* p; long s_r, s_c, b1, b2; int batch2; int seg = 0; long seg_stride = 0; const int* first = nullptr; };
// One warp per plane row: first the row's largest magnitude (the row is read a second time from L1 / L2 afterwards),
// then eight elements per lane and step (two 16-byte loads, one 16-byte store per plane).  blockIdx.y = problem index.
// `rownorm` (may be null): receives the L2 norm of every row (a factor of the bound of a plane-output contraction).
__global__ void __launch_bounds__(256) split2_rows_kernel(TcSrc s, int rows, int cols, __half* __restrict__ pl, float* __restrict__ inv_scale, int ldp,
                                                          float* __restrict__ rownorm) {
  const int z = blockIdx.y, lane = threadIdx.x & 31;
  const long r = (long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= rows || (s.first && z % s.batch2 < s.first[z / s.batch2])) return;
  const float* src = s.p + (z / s.batch2) * s.b1 + (z % s.batch2) * s.b2 + r * s.s_r;
  const int seg = s.seg ? s.seg : cols; const long over = s.seg ? s.seg_stride - s.seg : 0;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | (uintptr_t)(over * 4)) & 15) == 0;
  const int cols8 = vec ? (cols & ~7) : 0;                  // columns handled with 16-byte loads
  float mx = 0.f, sq = 0.f;
#pragma unroll 2
  for (int c = lane * 8; c < cols8; c += 256) {
    const float* q = src + c + (over ? c / seg * over : 0);
    const float4 a = *reinterpret_cast<const float4*>(q), b = *reinterpret_cast<const float4*>(q + 4);
    mx = fmaxf(mx, fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))), fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w)))));
    sq += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w + b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
  }
  for (int c = cols8 + lane; c < cols; c += 32) { const float v = src[c + (over ? c / seg * over : 0)]; mx = fmaxf(mx, fabsf(v)); sq += v * v; }
  mx = warp_max(mx);
  if (rownorm) { sq = warp_sum(sq); if (lane == 0) rownorm[(long)z * rows + r] = sqrtf(sq) * 1.0001f; }
  float inv; const float sc = row_scale(mx, &inv);
  if (lane == 0) inv_scale[(long)z * rows + r] = inv;
  __half* o = pl + ((long)z * rows + r) * 2 * ldp;
#pragma unroll 2
  for (int c = lane * 8; c < ldp; c += 256) {
    float t[8]; const float* q = src + c + (over ? c / seg * over : 0);
    if (c + 7 < cols8) {
      const float4 a = *reinterpret_cast<const float4*>(q), b = *reinterpret_cast<const float4*>(q + 4);
      t[0] = a.x; t[1] = a.y; t[2] = a.z; t[3] = a.w; t[4] = b.x; t[5] = b.y; t[6] = b.z; t[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) t[j] = c + j < cols ? q[j] : 0.f;
    }
    uint4 a, b;
    split2_pair(t[0], t[1], sc, a.x, b.x); split2_pair(t[2], t[3], sc, a.y, b.y);
    split2_pair(t[4], t[5], sc, a.z, b.z); split2_pair(t[6], t[7], sc, a.w, b.w);
    *reinterpret_cast<uint4*>(o + pl_off(c)) = a;
    *reinterpret_cast<uint4*>(o + pl_off(c) + PL_LO) = b;
  }
}
// The same for few, long rows (the gradient of a head's output: 64 x 8192), where a warp per row leaves most SMs idle: a cluster of up to eight
// blocks per row, every thread holding up to 32 of the row's elements in registers between the maximum and the planes.  Bound by
// the latency of its loads and of one exchange through the cluster.  A training step of the small causal Transformer, which splits one such
// gradient (64 x 8192), went from 742 to 730 us.  From 2048 columns on, where a warp walks its row eight times, and up to as many rows as
// SMs.  us with cold caches, a warp per row -> this: 1 x 2048 6.2 -> 4.7, 148 x 2048 6.9 -> 4.8, 64 x 4096 10.8 -> 5.1, 64 x 8192 21 -> 5.4,
// 148 x 8192 21 -> 8.6, 148 x 16384 40 -> 14, 1 x 65536 133 -> 6, 148 x 65536 152 -> 21.
constexpr int SPLIT_W_CLUSTER = 8, SPLIT_W_MAX = SPLIT_W_CLUSTER * 256 * 32;
__global__ void __launch_bounds__(256) split2_wide_rows_kernel(TcSrc s, int rows, int cols, __half* __restrict__ pl, float* __restrict__ inv_scale, int ldp, float* __restrict__ rownorm, int cs) {
  __shared__ float red[2][8], part[2];
  const int z = blockIdx.y, rank = blockIdx.x % cs, lane = threadIdx.x & 31, warp = threadIdx.x >> 5; const long r = blockIdx.x / cs;
  if (s.first && z % s.batch2 < s.first[z / s.batch2]) return;
  const float* src = s.p + (z / s.batch2) * s.b1 + (z % s.batch2) * s.b2 + r * s.s_r;
  const int seg = s.seg ? s.seg : cols; const long over = s.seg ? s.seg_stride - s.seg : 0;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | (uintptr_t)(over * 4)) & 15) == 0;
  float t[4][8], mx = 0.f, sq = 0.f;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c = 8 * ((i * cs + rank) * 256 + (int)threadIdx.x); const float* q = src + c + (over ? c / seg * over : 0);
    if (vec && c + 7 < cols) {
      const float4 a = *reinterpret_cast<const float4*>(q), b = *reinterpret_cast<const float4*>(q + 4);
      t[i][0] = a.x; t[i][1] = a.y; t[i][2] = a.z; t[i][3] = a.w; t[i][4] = b.x; t[i][5] = b.y; t[i][6] = b.z; t[i][7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) t[i][j] = c + j < cols ? q[j] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) { mx = fmaxf(mx, fabsf(t[i][j])); sq = fmaf(t[i][j], t[i][j], sq); }
  }
  mx = warp_max(mx); sq = warp_sum(sq);
  if (lane == 0) { red[0][warp] = mx; red[1][warp] = sq; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; w++) { mx = fmaxf(mx, red[0][w]); sq += red[1][w]; }
    part[0] = mx; part[1] = sq;
  }
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  cluster.sync();
  mx = sq = 0.f;
  for (int k = 0; k < cs; k++) { const float* q = cluster.map_shared_rank(part, k); mx = fmaxf(mx, q[0]); sq += q[1]; }
  cluster.sync();                                           // (nobody leaves while its part is being read)
  float inv; const float sc = row_scale(mx, &inv);
  if (rank == 0 && threadIdx.x == 0) { inv_scale[(long)z * rows + r] = inv; if (rownorm) rownorm[(long)z * rows + r] = sqrtf(sq) * 1.0001f; }
  __half* o = pl + ((long)z * rows + r) * 2 * ldp;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int c = 8 * ((i * cs + rank) * 256 + (int)threadIdx.x);
    if (c < ldp) {
      uint4 a, b;
      split2_pair(t[i][0], t[i][1], sc, a.x, b.x); split2_pair(t[i][2], t[i][3], sc, a.y, b.y); split2_pair(t[i][4], t[i][5], sc, a.z, b.z); split2_pair(t[i][6], t[i][7], sc, a.w, b.w);
      *reinterpret_cast<uint4*>(o + pl_off(c)) = a;
      *reinterpret_cast<uint4*>(o + pl_off(c) + PL_LO) = b;
    }
  }
}
// Largest magnitude of every plane row of a transposed operand (= of every column of the stored matrix): a block covers
// 64 plane rows x 256 contraction indices, reads run along the stored matrix's fast index, one atomicMax per row and block
// on the bit pattern (non-negative floats order like integers).  `mx` must be zero on entry.
__global__ void __launch_bounds__(256) colmax_kernel(TcSrc s, int rows, int cols, int* __restrict__ mx) {
  __shared__ float red[4][64];
  const int z = blockIdx.z, r = blockIdx.x * 64 + (threadIdx.x & 63), cy = threadIdx.x >> 6;
  const float* src = s.p + (z / s.batch2) * s.b1 + (z % s.batch2) * s.b2;
  float m = 0.f;
  if (r < rows) for (int c = blockIdx.y * 256 + cy; c < min(cols, (int)(blockIdx.y + 1) * 256); c += 4) m = fmaxf(m, fabsf(src[r + (long)c * s.s_c]));
  red[cy][threadIdx.x & 63] = m;
  __syncthreads();
  if (threadIdx.x < 64 && r < rows) {
    m = fmaxf(fmaxf(red[0][threadIdx.x], red[1][threadIdx.x]), fmaxf(red[2][threadIdx.x], red[3][threadIdx.x]));
    if (!(m <= 3.0e38f)) m = 3.4e38f;                       // an infinity or a NaN in the column: row_scale() then uses s = 1
    atomicMax(mx + (long)z * rows + r, __float_as_int(m));
  }
}
// Transposing split: 64 x 64 source tile through shared memory; reads run along the source's fast index (r), each
// thread then writes two neighbouring contraction indices of one plane row as one 4-byte word.  `mx` = colmax_kernel's result.
__global__ void __launch_bounds__(256) split2_cols_kernel(TcSrc s, int rows, int cols, __half* __restrict__ pl, const int* __restrict__ mx,
                                                          float* __restrict__ inv_scale, int ldp) {
  __shared__ float t[64][65];
  const int z = blockIdx.z, c0 = blockIdx.x * 64, r0 = blockIdx.y * 64;
  const float* src = s.p + (z / s.batch2) * s.b1 + (z % s.batch2) * s.b2;
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
  for (int j = ty; j < 64; j += 4) { const int c = c0 + j, r = r0 + tx; t[j][tx] = (r < rows && c < cols) ? src[r + (long)c * s.s_c] : 0.f; }
  __syncthreads();
  const long zo = (long)z * rows * 2 * ldp;
  const int cx = (threadIdx.x & 31) * 2, ry = threadIdx.x >> 5;
  for (int j = ry; j < 64; j += 8) {
    const int r = r0 + j, c = c0 + cx;
    if (r < rows && c < ldp) {
      float inv; const float sc = row_scale(__int_as_float(mx[(long)z * rows + r]), &inv);
      if (c == 0) inv_scale[(long)z * rows + r] = inv;
      uint32_t a, b; split2_pair(t[cx][j], t[cx + 1][j], sc, a, b);
      __half* o = pl + zo + (long)r * 2 * ldp + pl_off(c);
      *reinterpret_cast<uint32_t*>(o) = a; *reinterpret_cast<uint32_t*>(o + PL_LO) = b;
    }
  }
}

// Both passes in one launch, the source read once: a cluster of up to eight blocks owns 32 plane rows, each block a run of
// contraction indices, kept in shared memory (rows of 33 floats: free of bank conflicts both ways) between the row maxima --
// combined through the cluster -- and the planes.  Memory-bound.  For contractions of up to SPLIT_T_MAX indices (the run has to fit);
// [1000, 1100] and [4096, 2816] transposed took 16 and 33 us in two passes and a memset.
constexpr int SPLIT_T_CLUSTER = 8, SPLIT_T_RUN = 1536, SPLIT_T_MAX = SPLIT_T_CLUSTER * SPLIT_T_RUN;
__global__ void __launch_bounds__(256) split2_cols_cluster_kernel(TcSrc s, int rows, int cols, __half* __restrict__ pl, float* __restrict__ inv_scale, int ldp, int per, int cs) {
  extern __shared__ float slab[];                           // [per][33]
  __shared__ float red[8][32], mxs[32];
  const int z = blockIdx.y, rank = blockIdx.x % cs, r0 = blockIdx.x / cs * 32, k0 = rank * per, k1 = min(ldp, k0 + per), t = threadIdx.x, lane = t & 31, w = t >> 5;
  const float* src = s.p + (z / s.batch2) * s.b1 + (z % s.batch2) * s.b2;
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | (uintptr_t)(s.s_c * 4)) & 15) == 0 && r0 + 32 <= rows;
  const int c4 = (t & 7) * 4, ko = t >> 3;                  // this thread: columns c4 .. c4 + 3 of stored rows k0 + ko + 32 i
  float m[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int k = k0 + ko; k < k1; k += 32) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < cols) {
      const float* q = src + (long)k * s.s_c + r0 + c4;
      if (vec) v = *reinterpret_cast<const float4*>(q);
      else { if (r0 + c4 < rows) v.x = q[0]; if (r0 + c4 + 1 < rows) v.y = q[1]; if (r0 + c4 + 2 < rows) v.z = q[2]; if (r0 + c4 + 3 < rows) v.w = q[3]; }
    }
    float* d = slab + (k - k0) * 33 + c4; d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    m[0] = fmaxf(m[0], fabsf(v.x)); m[1] = fmaxf(m[1], fabsf(v.y)); m[2] = fmaxf(m[2], fabsf(v.z)); m[3] = fmaxf(m[3], fabsf(v.w));
  }
#pragma unroll
  for (int j = 0; j < 4; j++) {
    m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], 8)); m[j] = fmaxf(m[j], __shfl_xor_sync(0xffffffffu, m[j], 16));
    if (lane < 8) red[w][c4 + j] = m[j];
  }
  __syncthreads();
  if (t < 32) { float v = red[0][t]; for (int q = 1; q < 8; q++) v = fmaxf(v, red[q][t]); mxs[t] = v; }
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  cluster.sync();
  if (t < 32) {
    float v = 0.f;
    for (int q = 0; q < cs; q++) v = fmaxf(v, cluster.map_shared_rank(mxs, q)[t]);
    if (!(v <= 3.0e38f)) v = 3.4e38f;                       // an infinity in the column: row_scale() then uses s = 1
    float inv; red[0][t] = row_scale(v, &inv);
    if (rank == 0 && r0 + t < rows) inv_scale[(long)z * rows + r0 + t] = inv;
  }
  cluster.sync();                                           // (also: nobody leaves while its maxima are being read)
  for (int kb = k0 + 32 * w; kb < k1; kb += 256)            // a warp per block of 32 contraction indices, four plane rows at a time
#pragma unroll 2
    for (int i = 0; i < 32; i += 4) {
      const int r = i + (lane >> 3), k = (lane & 7) * 4; const float sc = red[0][r]; const float* q = slab + (kb - k0 + k) * 33 + r;
      if (r0 + r >= rows) continue;
      uint2 a, b; split2_pair(q[0], q[33], sc, a.x, b.x); split2_pair(q[66], q[99], sc, a.y, b.y);
      __half* o = pl + ((long)z * rows + r0 + r) * 2 * ldp + pl_off(kb + k);
      *reinterpret_cast<uint2*>(o) = a; *reinterpret_cast<uint2*>(o + PL_LO) = b;
    }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                    CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// Operand planes of the contraction engine: two interleaved fp16 planes [nbatch][rows][2 ldp] (pl_off; ldp a multiple of 32, zero
// beyond K), and the inverse scale of every plane row [nbatch][rows].  koff (a multiple of 32): first contraction index used.
struct BfPlanes { __half* base; float* inv_scale; int rows, K, ldp, nbatch; int koff = 0; };
// Where a contraction's result goes when it is only ever used as the A operand of another contraction (the FFN's hidden
// activation and its gradient: half of all operand elements of a TransformerBlock).  A row's scale must be known before
// its first element is written, and a tile sees only 256 of the row's columns, so the scale comes from a bound instead of
// the row's maximum: |sum_k a_k b_k + bias| <= sqrt(|a|^2 + 1) * sqrt(K + 1) * max(|B|, |bias|) (Cauchy-Schwarz).  For
// random-sign data the bound is about 8-16 times the row's actual maximum, i.e. 3-4 of the planes' 22 bits; it can never
// be exceeded, so the fp16 planes cannot overflow.  `last`: fp32 copy of every sequence's last row (the only rows of
// these tensors that are read as numbers: ReLU gate and weight-gradient input of the reference's last-token rule).
struct TcPlaneOut { BfPlanes planes; const int* b_maxabs; float* last; int last_T; float* rowsum32 = nullptr; float* z_last = nullptr; bool scale = false; };
inline int tc_ldp(int K) { return ((K + 31) / 32) * 32; }           // plane row length: whole blocks of 32
inline size_t bf_plane_floats(long nbatch, long rows, long ldp) { return (size_t)nbatch * rows * ldp; }   // two fp16 planes = one float per element

// Per-context operand-plane scratch of the contraction engine (calls on a context are serialised by Ctx::run_mu).
struct TcScratch { DevBuf a, b, sa, sb, mx, part; const float* last_a = nullptr; int last_m = 0, last_k = 0; long last_ld = 0; };
inline TcScratch& tc_scratch(Ctx* ctx) { if (!ctx->tc_scratch) ctx->tc_scratch = ctx->own(new TcScratch()); return *static_cast<TcScratch*>(ctx->tc_scratch); }

// After a replayed graph the scratch no longer holds what the last directly issued call left there.
inline void forget_planes(Ctx* ctx) { if (ctx->tc_scratch) tc_scratch(ctx).last_a = nullptr; }
// Operand planes for `nbatch` problems of rows x K in the context's scratch (which = 0: A side, 1: B side).
inline int tc_planes(Ctx* ctx, int which, long nbatch, long rows, int K, BfPlanes* out) {
  TcScratch& sc = tc_scratch(ctx);
  const int ldp = tc_ldp(K); const size_t n = bf_plane_floats(nbatch, rows, ldp), ns = (size_t)nbatch * rows;
  if (rows > 0x7fffffffL || nbatch > 65535) return fail(GN_ERR_UNSUPPORTED, "tc_planes: operand too large");
  DevBuf& pl = which == 0 ? sc.a : sc.b; DevBuf& scl = which == 0 ? sc.sa : sc.sb;
  if (pl.n < n) { GN_CUDA(cudaStreamSynchronize(ctx->stream)); ctx->epoch++; GN_TRY(pl.alloc(n)); }
  if (scl.n < ns) { GN_CUDA(cudaStreamSynchronize(ctx->stream)); ctx->epoch++; GN_TRY(scl.alloc(ns + 1024)); }
  if (sc.mx.n < ns) { GN_CUDA(cudaStreamSynchronize(ctx->stream)); ctx->epoch++; GN_TRY(sc.mx.alloc(ns + 1024)); }
  if (which == 0) sc.last_a = nullptr;
  *out = BfPlanes{reinterpret_cast<__half*>(pl.p), scl.p, (int)rows, K, ldp, (int)nbatch}; return GN_OK;
}
inline int* tc_rowmax_buf(Ctx* ctx) { return reinterpret_cast<int*>(tc_scratch(ctx).mx.p); }

template <int BN, TcOut OUT> inline bool tc_set_smem1() { return cudaFuncSetAttribute(gemm_tc_persist_kernel<BN, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcCfg<BN, OUT == TC_OUT_PLANES>::SMEM_BYTES) == cudaSuccess; }
template <int BN> inline bool tc_set_smem() { return tc_set_smem1<BN, TC_OUT_VEC>() && tc_set_smem1<BN, TC_OUT_PLANES>() && tc_set_smem1<BN, TC_OUT_ROWS>(); }
inline void tc_init(Ctx* ctx) {
  ctx->tc_ok = false;
  void* fn = nullptr; cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn || q != cudaDriverEntryPointSuccess) { cudaGetLastError(); return; }
  if (!(tc_set_smem<64>() && tc_set_smem<128>() && tc_set_smem<256>())) { cudaGetLastError(); return; }
  ctx->encode_tiled = fn; ctx->tc_ok = true;
  if (const char* e = getenv("GONEURON_CUDA_TC_BN")) ctx->tc_force_bn = atoi(e);
  if (const char* e = getenv("GONEURON_CUDA_TC_KSLICE")) ctx->tc_kslice = atoi(e);
  if (const char* e = getenv("GONEURON_CUDA_TC_TAIL_SPLIT")) ctx->tc_tail_split = atoi(e) != 0;
  if (const char* e = getenv("GONEURON_CUDA_TC_TILE_QUEUE")) ctx->tc_tile_queue = atoi(e) != 0;
  if (!ctx->tc_queue_pool) {
    // (cleared on the legacy stream, which the context's non-blocking stream does not wait for: hence the device-wide wait)
    if (cudaMalloc(&ctx->tc_queue_pool, TC_QUEUE_POOL * sizeof(int)) != cudaSuccess || cudaMemset(ctx->tc_queue_pool, 0, TC_QUEUE_POOL * sizeof(int)) != cudaSuccess ||
        cudaDeviceSynchronize() != cudaSuccess) {
      cudaGetLastError(); ctx->tc_queue_pool = nullptr; ctx->tc_tile_queue = false;
    }
  }
}

// 16-bit plane [nbatch][rows][ld], `cols` valid columns, 64 columns (128 bytes, 128-byte swizzle) x box_rows per copy
inline int tc_make_map_f16(Ctx* ctx, CUtensorMap* map, const __half* base, int cols, int rows, long ld, int nbatch, int box_rows) {
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)nbatch};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)rows * ld * 2};
  cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = ((PFN_encodeTiled)ctx->encode_tiled)(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(GN_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d (rows %d columns %d ld %ld batch %d)", (int)r, rows, cols, ld, nbatch);
  return GN_OK;
}
// ... of a contraction operand: the interleaved blocks of K contraction indices from koff on
inline int tc_operand_map(Ctx* ctx, CUtensorMap* map, const BfPlanes& p, int box_rows) {
  return tc_make_map_f16(ctx, map, p.base + 2 * (long)p.koff, 2 * tc_ldp(p.K), p.rows, 2L * p.ldp, p.nbatch, box_rows);
}

// Writes the planes and inverse row scales of an operand.  `mx` (only used by the transposing variant): nbatch * rows ints.
inline int tc_split(Ctx* ctx, const TcSrc& src, const BfPlanes& p, int* mx, float* rownorm = nullptr) {
  if (rownorm && src.s_c != 1) return fail(GN_ERR_UNSUPPORTED, "tc_split: row norms are only formed by the row-wise split");
  if (src.s_c == 1) {
    if (p.nbatch > 65535) return fail(GN_ERR_UNSUPPORTED, "tc_split: more than 65535 problems in a batch");
    if ((long)p.rows * p.nbatch <= ctx->sm_count && p.ldp >= 2048 && p.ldp <= SPLIT_W_MAX) {
      int cs = 1; while (cs < SPLIT_W_CLUSTER && p.ldp > cs * 256 * 8) cs *= 2;      // eight elements a thread where that takes no more than eight blocks
      GN_CLUSTER_LAUNCH(ctx, split2_wide_rows_kernel, dim3(p.rows * cs, p.nbatch), 256, 0, cs, src, p.rows, p.K, p.base, p.inv_scale, p.ldp, rownorm, cs);
    } else GN_LAUNCH(ctx, split2_rows_kernel, dim3(cdiv(p.rows, 8), p.nbatch), 256, 0, src, p.rows, p.K, p.base, p.inv_scale, p.ldp, rownorm);
  } else if (src.s_r == 1) {
    if (p.nbatch > 65535 || cdiv(p.rows, 64) > 65535 || cdiv(p.K, 256) > 65535) return fail(GN_ERR_UNSUPPORTED, "tc_split: operand too large for the transposing split");
    if (p.ldp <= SPLIT_T_MAX) {
      int cs = 1; while (cs < SPLIT_T_CLUSTER && p.ldp > 64 * cs) cs *= 2;
      const int per = cdiv(cdiv(p.ldp, cs), 32) * 32, smem = per * 33 * (int)sizeof(float);
      if (smem > 40 * 1024) GN_CUDA(cudaFuncSetAttribute(split2_cols_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      GN_CLUSTER_LAUNCH(ctx, split2_cols_cluster_kernel, dim3(cdiv(p.rows, 32) * cs, p.nbatch), 256, smem, cs, src, p.rows, p.K, p.base, p.inv_scale, p.ldp, per, cs);
      ctx->split_bytes += 8.0 * (double)p.nbatch * p.rows * p.K;
      return check_launch("tc_split");
    }
    if (!mx) return fail(GN_ERR_INVALID_ARG, "tc_split: the transposing split needs a row-maximum buffer");
    GN_CUDA(stream_zero(ctx, mx, (size_t)p.nbatch * p.rows * sizeof(int)));
    GN_LAUNCH(ctx, colmax_kernel, dim3(cdiv(p.rows, 64), cdiv(p.K, 256), p.nbatch), 256, 0, src, p.rows, p.K, mx);
    GN_LAUNCH(ctx, split2_cols_kernel, dim3(cdiv(p.ldp, 64), cdiv(p.rows, 64), p.nbatch), 256, 0, src, p.rows, p.K, p.base, (const int*)mx, p.inv_scale, p.ldp);
  } else return fail(GN_ERR_UNSUPPORTED, "tc_split: neither stride of the operand is 1");
  ctx->split_bytes += 8.0 * (double)p.nbatch * p.rows * p.K;
  return check_launch("tc_split");
}

// SMs a persistent kernel spreads over.  With several ranks the gradient all-reduces run beside the backward pass; a
// persistent kernel that waits for the SMs their CTAs hold takes as long as the collective, so it leaves them some.
inline int persist_sms(const Ctx* ctx) { return std::max(1, ctx->sm_count - ctx->sm_reserve); }
// Number of left-over tiles of the last round that are run as two half tiles each (0: none): only when they would keep at
// most half of the CTAs busy, and not for the triangular products (their tiles differ in length anyway).
inline long tc_tail_halves(Ctx* ctx, long total_tiles, int bn, int flags) {
  if (!ctx->tc_tail_split || bn < 128 || total_tiles <= persist_sms(ctx) || (flags & (GEMM_SKIP_UPPER | GEMM_KBEG_AT_M0 | GEMM_KEND_AT_M0))) return 0;
  const long left = total_tiles % persist_sms(ctx);
  return 2 * left <= persist_sms(ctx) ? left : 0;
}
// A zeroed counter for one launch's tile queue, from a pool that is cleared when it has been used up (in stream order, so
// every earlier launch has finished with its counter by then).
inline int tc_next_queue(Ctx* ctx, int** out) {
  if (!ctx->tc_queue_pool) return fail(GN_ERR_CUDA, "tile-queue pool missing");
  if (ctx->tc_queue_used >= TC_QUEUE_POOL) { GN_CUDA(cudaMemsetAsync(ctx->tc_queue_pool, 0, TC_QUEUE_POOL * sizeof(int), ctx->stream)); ctx->tc_queue_used = 0; }
  *out = ctx->tc_queue_pool + ctx->tc_queue_used++; return GN_OK;
}
template <int BN>
inline int tc_launch_persist(Ctx* ctx, const BfPlanes& A, const BfPlanes& B, const TcParams& ep) {
  CUtensorMap mA, mB;
  // the B tile of a stage arrives as two copies of BN / 2 rows, so that a half tile (see the kernel's work list) is one of them
  GN_TRY(tc_operand_map(ctx, &mA, A, TC_BM)); GN_TRY(tc_operand_map(ctx, &mB, B, BN / 2));
  const int tiles_m = cdiv(ep.M, TC_BM), tiles_n = cdiv(ep.N, BN); const long total = (long)tiles_m * tiles_n * A.nbatch * ep.splits;
  if (total > 0x7fffffffL) return fail(GN_ERR_UNSUPPORTED, "too many output tiles");
  const unsigned grid = (unsigned)std::min<long>(total, persist_sms(ctx));
  const long left = tc_tail_halves(ctx, total, BN, ep.flags);
  const int full_end = (int)(total - left), n_half = (int)(2 * left);
  int* queue = nullptr;
  if (ctx->tc_tile_queue && total > grid) GN_TRY(tc_next_queue(ctx, &queue));
  ProfScope prof(ctx);
  if (ep.out_p) GN_LAUNCH(ctx, (gemm_tc_persist_kernel<BN, TC_OUT_PLANES>), grid, (TcCfg<BN, true>::THREADS), (TcCfg<BN, true>::SMEM_BYTES), mA, mB, ep, tiles_m, tiles_n, (int)total, full_end, n_half, queue);
  else if ((ep.flags & TC_FLAG_VEC) || ep.nchw_P > 0) GN_LAUNCH(ctx, (gemm_tc_persist_kernel<BN, TC_OUT_VEC>), grid, (TcCfg<BN, false>::THREADS), (TcCfg<BN, false>::SMEM_BYTES), mA, mB, ep, tiles_m, tiles_n, (int)total, full_end, n_half, queue);
  else GN_LAUNCH(ctx, (gemm_tc_persist_kernel<BN, TC_OUT_ROWS>), grid, (TcCfg<BN, false>::THREADS), (TcCfg<BN, false>::SMEM_BYTES), mA, mB, ep, tiles_m, tiles_n, (int)total, full_end, n_half, queue);
  return check_launch("gemm_tc_persist");
}
// Output tile width for a problem: 64 for narrow outputs; 256 (three quarters of the shared-memory traffic per MMA
// cycle of the 128-wide tile) when the problem still fills the SMs evenly with tiles of that size.
inline int tc_pick_bn(Ctx* ctx, int M, int N, long nbatch, int flags) {
  if (ctx->tc_force_bn == 64 || ctx->tc_force_bn == 128 || ctx->tc_force_bn == 256) return ctx->tc_force_bn;
  if (N <= 64) return 64;
  if (N <= 128 || (flags & (GEMM_SKIP_UPPER | GEMM_KBEG_AT_M0 | GEMM_KEND_AT_M0))) return 128;
  auto cost = [&](int bn, double rate) {
    const long tiles = (long)cdiv(M, TC_BM) * cdiv(N, bn) * nbatch;
    double waves = std::ceil((double)tiles / persist_sms(ctx));
    if (tc_tail_halves(ctx, tiles, bn, flags) > 0) waves -= 0.38;       // a half tile costs about 0.62 of a whole one
    return waves * bn / rate;
  };
  return cost(256, 1.3) < cost(128, 1.0) ? 256 : 128;
}
// C[z] = A[z] * B[z]^T from prepared planes, one accumulator run over the whole contraction.
inline int tc_launch(Ctx* ctx, const BfPlanes& A, const BfPlanes& B, const TcParams& ep_in, int bn) {
  if (!ctx->tc_ok) return fail(GN_ERR_UNSUPPORTED, "tcgen05 engine unavailable");
  TcParams ep = ep_in; ep.spin_limit = ctx->spin_limit; ep.isa = A.inv_scale; ep.isb = B.inv_scale;
  if (A.K != B.K || A.nbatch != B.nbatch || A.rows != ep.M || B.rows != ep.N || A.K != ep.K) return fail(GN_ERR_INVALID_ARG, "tc_launch: operand shapes disagree");
  auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  bool vec = ep.N % 4 == 0 && ep.ldc % 4 == 0 && ep.c_b1 % 4 == 0 && ep.c_b2 % 4 == 0 && a16(ep.C) && (!ep.bias || a16(ep.bias)) && a16(ep.isb);
  if (ep.R) vec = vec && ep.ldr % 4 == 0 && ep.r_b1 % 4 == 0 && ep.r_b2 % 4 == 0 && a16(ep.R);
  if (ep.n_seg) vec = vec && ep.c_seg % 4 == 0 && ep.bias_seg % 4 == 0;
  if (ep.mask) vec = vec && ep.mask_ld % 4 == 0 && a16(ep.mask);
  if (ep.nchw_P > 0) { if (ep.R || A.nbatch != 1) return fail(GN_ERR_UNSUPPORTED, "tc_launch: NCHW store with a residual or a batch"); vec = false; }
  if (ep.out_p) {
    if (!(ep.N % 32 == 0 && ep.out_ldp % 32 == 0 && (reinterpret_cast<uintptr_t>(ep.out_p) & 31) == 0 && (!ep.bias || a16(ep.bias)) && a16(ep.isb) && (!ep.mask || (ep.mask_ld % 4 == 0 && a16(ep.mask))) && (!ep.c_last || a16(ep.c_last)) && (!ep.z_last || a16(ep.z_last)) && (!ep.rowsum32 || a16(ep.rowsum32))))
      return fail(GN_ERR_INVALID_ARG, "tc_launch: plane output needs whole blocks of 32 columns and aligned operands");
    vec = true;
  }
  if (ep.zmax && !vec) return fail(GN_ERR_INVALID_ARG, "tc_launch: maxima need 16-byte aligned operands");
  if (vec) ep.flags |= TC_FLAG_VEC;
  {
    double by = 4.0 * ((double)ep.M + ep.N) * ep.K + 4.0 * (double)ep.M * ep.N * (ep.R ? 2 : 1);
    if (ep.flags & (GEMM_SKIP_UPPER | GEMM_KBEG_AT_M0 | GEMM_KEND_AT_M0)) by *= 0.5;
    ctx->gemm_bytes += by * A.nbatch;
  }
  if (bn == 64) return tc_launch_persist<64>(ctx, A, B, ep);
  if (bn == 256) return tc_launch_persist<256>(ctx, A, B, ep);
  return tc_launch_persist<128>(ctx, A, B, ep);
}
// The tensor core truncates when it adds a product group to the accumulator, so the error of one accumulator run grows
// with the number of MMA instructions that feed it (one per 16 contraction indices and term).  Long contractions (weight
// gradients over all tokens of a batch) are therefore cut into slices, each slice adding its result to C through the
// epilogue's residual path, i.e. in properly rounded fp32: 4096 indices per run with separate accumulators for the
// large and the small terms, 2048 with the single accumulator of the 256-wide tile.
inline int tc_run_rows(Ctx* ctx, const BfPlanes& A, const BfPlanes& B, const TcParams& ep, int bn, int slice = 0) {
  const int kslice = slice > 0 ? slice : ctx->tc_kslice > 0 ? ctx->tc_kslice : (bn == 256 ? 2048 : 4096);
  if (ep.K <= kslice || (ep.flags & (GEMM_KBEG_AT_M0 | GEMM_KEND_AT_M0))) return tc_launch(ctx, A, B, ep, bn);
  if (ep.out_p) return fail(GN_ERR_UNSUPPORTED, "a contraction that writes operand planes must fit one accumulator run (K = %d)", ep.K);
  for (int k0 = 0; k0 < ep.K; k0 += kslice) {
    const int kl = std::min(kslice, ep.K - k0); const bool first = k0 == 0, last = k0 + kl >= ep.K;
    BfPlanes As = A, Bs = B; As.koff = A.koff + k0; As.K = kl; Bs.koff = B.koff + k0; Bs.K = kl;
    TcParams es = ep; es.K = kl;
    if (!first) { es.bias = nullptr; es.R = ep.C; es.ldr = ep.ldc; es.r_b1 = ep.c_b1; es.r_b2 = ep.c_b2; }
    if (!last) { es.act = GN_ACT_LINEAR; es.mask = nullptr; }
    GN_TRY(tc_launch(ctx, As, Bs, es, bn));
  }
  return GN_OK;
}
// Few output tiles and a long contraction leave SMs idle for the whole contraction (the products of a head or of a block's token
// rows: 64 x 1024 over 4096 is eight tiles, 45 us with one tile per CTA), or make 128-wide tiles the only ones that fill them,
// whose main loop is bound by shared memory traffic.  The contraction can then be cut into slices, each a tile of its own with a
// partial result; a second kernel adds the partial results in slice order (fp32) and applies the epilogue.
// VEC: four columns per thread (N a multiple of four).  Whole product, us, with one kernel for both and the slices in a loop unrolled by four -> this: [700, 200] over 4096 13.4 -> 12.5,
// [128, 1024] over 8192 15.7 -> 14.7.
template <bool VEC>
__global__ void __launch_bounds__(256) tc_sum_slices_kernel(const float* __restrict__ part, int splits, int M, int N, const TcParams ep) {
  const long mn = (long)M * N;
  auto finish = [&](float x, int r, int c) {
    if (ep.bias) x += ep.bias[c];
    if (ep.R) x += ep.R[(long)r * ep.ldr + c];
    if (ep.act == GN_ACT_RELU) x = fmaxf(x, 0.f);
    if (ep.mask && !(ep.mask[(long)(r / ep.mask_group) * ep.mask_ld + c] > 0.f)) x = 0.f;
    return x;
  };
  if constexpr (VEC) {
    for (long i = 4 * (blockIdx.x * 256L + threadIdx.x); i < mn; i += gridDim.x * 1024L) {
      const int r = (int)(i / N), c = (int)(i - (long)r * N);
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int z = 0; z < splits; z += 4) {                   // four slices in flight together; where there are fewer left the last one again, not added
        float4 u[4];
#pragma unroll
        for (int q = 0; q < 4; q++) u[q] = *reinterpret_cast<const float4*>(part + min(z + q, splits - 1) * mn + i);
#pragma unroll
        for (int q = 0; q < 4; q++) if (z + q < splits) { t.x += u[q].x; t.y += u[q].y; t.z += u[q].z; t.w += u[q].w; }
      }
      float x[4] = {t.x, t.y, t.z, t.w};
      for (int k = 0; k < 4; k++) x[k] = finish(x[k], r, c + k);
      float* o = ep.C + (long)r * ep.ldc + c;
      if (((ep.ldc & 3) | (long)(reinterpret_cast<uintptr_t>(ep.C) & 15)) == 0) *reinterpret_cast<float4*>(o) = make_float4(x[0], x[1], x[2], x[3]);
      else for (int k = 0; k < 4; k++) o[k] = x[k];
    }
  } else {                                                    // four elements of a thread in flight together, a block apart
    for (long i0 = blockIdx.x * 1024L + threadIdx.x; i0 < mn; i0 += gridDim.x * 1024L) {
      float x[4] = {};
#pragma unroll 2
      for (int z = 0; z < splits; z++) {
#pragma unroll
        for (int k = 0; k < 4; k++) if (i0 + 256 * k < mn) x[k] += part[z * mn + i0 + 256 * k];
      }
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const long i = i0 + 256 * k; if (i >= mn) break;
        const int r = mn < (1L << 31) ? (int)i / N : (int)(i / N), c = (int)(i - (long)r * N);
        ep.C[(long)r * ep.ldc + c] = finish(x[k], r, c);
      }
    }
  }
}
// Slices and tile width by estimated time, from measured rates (us): 0.335 / 0.43 per 32 contraction indices of a 128 / 256 wide
// tile, 2.4 / 3.9 for the last tile's epilogue, 3 for the second launch and 4 TB/s for its partial results.  Slices keep at least 256
// indices, and have to win by a tenth.  Over 249 products with contractions of 512 to 32 000 (us, whole or in other slices -> as chosen): every choice below 1024 that differs from one
// launch wins, [5000, 33] over 768 14.6 -> 12.6 the least, [150, 768] over 1000 16.0 -> 11.3; [1000, 1000] over 1500 21.6 -> 17.4, [1024, 1024] over 2048 20.2 -> 18.7 (256 wide in four, by today's
// epilogues; with 3 / 5 for them 128 wide in two).  Rows that 16-byte pieces do not fit go by the same figures: their epilogue is longer, and slices win by more ([1100, 333] over 1000 30.8 -> 18.2).
inline int tc_split_count(Ctx* ctx, const TcParams& ep, long nbatch, int* bn) {
  if (nbatch != 1 || ep.out_p || ep.n_seg || ep.nchw_P || ep.flags || ep.K < 512 || ctx->tc_kslice > 0 || ctx->tc_force_bn) return 1;
  const long sms = persist_sms(ctx), tm = cdiv(ep.M, TC_BM); const double kb = cdiv(ep.K, TC_BK);
  auto cost = [&](int w, int sl) {
    const long tiles = tm * cdiv(ep.N, w); double rounds = std::ceil((double)tiles * sl / sms);
    if (sl == 1 && tc_tail_halves(ctx, tiles, w, 0) > 0) rounds -= 0.38;
    return rounds * (kb / sl) * (w == 256 ? 0.43 : 0.335) + (w == 256 ? 3.9 : 2.4) + (sl > 1 ? 3.0 + 1e-6 * ep.M * ep.N * (sl + 1) : 0.0);
  };
  double best = 0.9 * cost(tc_pick_bn(ctx, ep.M, ep.N, 1, 0) == 256 ? 256 : 128, 1); int splits = 1;
  for (int w : {128, 256}) if (w == 128 || ep.N > 128)
    for (int sl = std::max(2, (int)cdiv(ep.K, w == 256 ? 2048 : 4096)); sl <= 32 && sl * 256 <= ep.K; sl++) {
      if (tm * cdiv(ep.N, w) * (sl - 1) >= sms) break;
      const double c = cost(w, sl); if (c < best) { best = c; splits = sl; *bn = w; }
    }
  return splits;
}
inline int tc_slice_length(int K, int splits) { return cdiv(cdiv(K, splits), TC_BK) * TC_BK; }
// `part`: room for one partial result [M, N] per slice
inline int tc_run_slices(Ctx* ctx, const BfPlanes& A, const BfPlanes& B, const TcParams& ep, int splits, int bn, float* part) {
  TcParams es = ep;
  es.k_slice = tc_slice_length(ep.K, splits); es.splits = cdiv(ep.K, es.k_slice);
  es.C = part; es.ldc = ep.N; es.c_b1 = (long)ep.M * ep.N; es.c_b2 = 0; es.batch2 = 1; es.bias = nullptr; es.R = nullptr; es.mask = nullptr; es.act = GN_ACT_LINEAR;
  es.z_first = nullptr;                                     // goes by problems, and z counts the slices of the only one
  GN_TRY(tc_launch(ctx, A, B, es, ep.N <= 64 ? 64 : bn));
  GN_LAUNCH(ctx, ((ep.N & 3) == 0 ? tc_sum_slices_kernel<true> : tc_sum_slices_kernel<false>), (unsigned)std::min<long>(cdiv((long)ep.M * ep.N, 1024), 4L * ctx->sm_count), 256, 0, (const float*)part, es.splits, ep.M, ep.N, ep);
  return check_launch("tc_sum_slices");
}
inline int tc_run(Ctx* ctx, const BfPlanes& A, const BfPlanes& B, const TcParams& ep) {
  int bn = 128; const int splits = tc_split_count(ctx, ep, A.nbatch, &bn);
  if (splits > 1) {
    TcScratch& sc = tc_scratch(ctx); const size_t n = (size_t)splits * ep.M * ep.N;
    if (sc.part.n < n) { GN_CUDA(cudaStreamSynchronize(ctx->stream)); ctx->epoch++; GN_TRY(sc.part.alloc(n)); }
    return tc_run_slices(ctx, A, B, ep, splits, bn, sc.part.p);
  }
  // (Running the rows of a short last wave as a second launch with 128-wide tiles was measured at 16 384 rows: the second
  // launch's fixed cost ate the 9 % it should have saved, so every product is one tiling.)
  return tc_run_rows(ctx, A, B, ep, tc_pick_bn(ctx, ep.M, ep.N, A.nbatch, ep.flags));
}

// ------------------------------------------------------------------ prepared planes of weight matrices
// A weight matrix W [out, in] is an operand twice per training step: as stored (rows = out, contraction over in) in the
// forward product X W^T, and transposed (rows = in, contraction over out) in the input-gradient product dZ W.  Splitting it
// at each use costs two small launches per orientation and matrix, work that does not shrink when the batch is sharded over
// GPUs.  Instead all registered matrices are split once per parameter update, both orientations from one read, by two
// launches in all: the matrices get ONE power-of-two scale each (their entries are of similar size, unlike activation
// rows), found by wplanes_max_kernel, and wplanes_split_kernel writes every 64 x 64 tile as stored and transposed.
// A registered matrix may be a stack of several (Q, K and V projections; SwiGLU gate and up): rows [j part, (j + 1) part) come from
// src + j * stride.  Products may then use the whole stack or a run of its parts.
struct WPlaneJob { const float* src; const float* bias; int part; long stride; int out, in, ldp_r, ldp_c; __half *r, *c; float *inv_r, *inv_c; int tile0, tiles_in; };
__device__ __forceinline__ const float* wplane_row(const WPlaneJob& jb, int r) { const int j = r / jb.part; return jb.src + j * jb.stride + (long)(r - j * jb.part) * jb.in; }
__device__ __forceinline__ int wplane_find(const WPlaneJob* jobs, int njobs, int tile) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) { const int mid = (lo + hi + 1) >> 1; if (jobs[mid].tile0 <= tile) lo = mid; else hi = mid - 1; }
  return lo;
}
// (after a training step the parameter update has left the maxima behind, see adam_kernel: this pass is for other changes)
__global__ void __launch_bounds__(256) wplanes_max_kernel(const WPlaneJob* __restrict__ jobs, int njobs, int* __restrict__ mx, int tile_off) {
  __shared__ float red[33];
  const int tile = blockIdx.x + tile_off;
  const int j = wplane_find(jobs, njobs, tile); const WPlaneJob jb = jobs[j];
  const int t = tile - jb.tile0, r0 = (t / jb.tiles_in) * 64, c0 = (t % jb.tiles_in) * 64;
  float m = 0.f;
  for (int e = threadIdx.x; e < 4096; e += 256) { const int r = r0 + (e >> 6), c = c0 + (e & 63); if (r < jb.out && c < jb.in) m = fmaxf(m, fabsf(wplane_row(jb, r)[c])); }
  if (jb.bias && c0 == 0 && threadIdx.x < 64 && r0 + (int)threadIdx.x < jb.out) m = fmaxf(m, fabsf(jb.bias[(r0 + (int)threadIdx.x) / jb.part * jb.stride + (r0 + (int)threadIdx.x) % jb.part]));      // the layer's biases count towards the maximum (bounds of plane-output contractions)
  m = block_max(m, red);
  if (threadIdx.x == 0) { if (!(m <= 3.0e38f)) m = 3.4e38f; atomicMax(mx + j, __float_as_int(m)); }
}
// Memory-bound: 4 bytes read and 8 written per weight.  16-byte loads of a 64 x 64 tile, then four neighbouring contraction
// indices per thread and store in either orientation: whole 64-byte runs of each plane (two indices and 4-byte stores ran at 1.8 TB/s).
__global__ void __launch_bounds__(256) wplanes_split_kernel(const WPlaneJob* __restrict__ jobs, int njobs, const int* __restrict__ mx, int tile_off) {
  __shared__ float tl[64][65];
  const int tile = blockIdx.x + tile_off;
  const int j = wplane_find(jobs, njobs, tile); const WPlaneJob jb = jobs[j];
  const int t = tile - jb.tile0, r0 = (t / jb.tiles_in) * 64, c0 = (t % jb.tiles_in) * 64;
  float mxv = __int_as_float(mx[j]); if (!(mxv <= 3.0e38f)) mxv = 3.4e38f;
  float inv; const float sc = row_scale(mxv, &inv);
  const int x4 = (threadIdx.x & 15) * 4, y = threadIdx.x >> 4, c = c0 + x4;
  const bool vec = (((uintptr_t)jb.src | (uintptr_t)(jb.in * 4) | (uintptr_t)(jb.stride * 4)) & 15) == 0;
  float4 v[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int r = r0 + y + 16 * k;
    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < jb.out) {
      const float* q = wplane_row(jb, r) + c;
      if (vec) { if (c < jb.in) v[k] = *reinterpret_cast<const float4*>(q); }
      else { if (c < jb.in) v[k].x = q[0]; if (c + 1 < jb.in) v[k].y = q[1]; if (c + 2 < jb.in) v[k].z = q[2]; if (c + 3 < jb.in) v[k].w = q[3]; }
    }
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {                              // as stored: plane row = out index (a last group beyond `in` writes zeros: plane rows are whole blocks of 32)
    const int rr = y + 16 * k, r = r0 + rr;
    tl[rr][x4] = v[k].x; tl[rr][x4 + 1] = v[k].y; tl[rr][x4 + 2] = v[k].z; tl[rr][x4 + 3] = v[k].w;
    if (r < jb.out && c < jb.in) {
      uint2 a, b; split2_pair(v[k].x, v[k].y, sc, a.x, b.x); split2_pair(v[k].z, v[k].w, sc, a.y, b.y);
      __half* o = jb.r + (long)r * 2 * jb.ldp_r + pl_off(c);
      *reinterpret_cast<uint2*>(o) = a; *reinterpret_cast<uint2*>(o + PL_LO) = b;
      if (c == 0) jb.inv_r[r] = inv;
    }
  }
  __syncthreads();
  const int r = r0 + x4;
#pragma unroll
  for (int k = 0; k < 4; k++) {                              // transposed: plane row = in index
    const int cc = y + 16 * k, ci = c0 + cc;
    if (ci < jb.in && r < jb.out) {
      uint2 a, b; split2_pair(tl[x4][cc], tl[x4 + 1][cc], sc, a.x, b.x); split2_pair(tl[x4 + 2][cc], tl[x4 + 3][cc], sc, a.y, b.y);
      __half* o = jb.c + (long)ci * 2 * jb.ldp_c + pl_off(r);
      *reinterpret_cast<uint2*>(o) = a; *reinterpret_cast<uint2*>(o + PL_LO) = b;
      if (r == 0) jb.inv_c[ci] = inv;
    }
  }
}
// Host side of the table: one entry per registered matrix, looked up by the matrix's device address.
struct WeightPlaneEntry { const float* src; int out, in; BfPlanes rows, cols; int part = 0; long stride = 0;      // (part = out: a single matrix)
  const float* bias = nullptr; const int* maxabs = nullptr; int layer = -1; int tile0 = 0, tiles = 0; };
struct WeightPlaneTable {
  std::vector<WeightPlaneEntry> e; DevBuf planes, scales, mx, jobs, ranges; int total_tiles = 0;
  bool dirty = true, used = false, max_ok = false;          // used: some product has looked a matrix up; max_ok: `mx` holds the maxima of the current parameters
  // entries [j0, j1) that belong to model layer `layer` (they are registered layer by layer, so the range is contiguous)
  void layer_range(int layer, int* j0, int* j1) const {
    *j0 = *j1 = 0; bool in = false;
    for (int j = 0; j < (int)e.size(); j++) if (e[j].layer == layer) { if (!in) { *j0 = j; in = true; } *j1 = j + 1; }
  }
  const WeightPlaneEntry* find(const float* p, int* part) const {
    for (auto& x : e) for (int j = 0; j < x.out / x.part; j++) if (x.src + j * x.stride == p) { *part = j; return &x; }
    return nullptr;
  }
};
// The parameters a table entry covers (ascending; the biases count towards an entry's maximum).
struct PlaneRange { const float *b, *e; };
// Lays the table out for the matrices (src, out, in) and allocates its buffers (planes zeroed once: the padding columns
// of a plane row are never written afterwards and must read as zero).
inline int wplanes_build(Ctx* ctx, WeightPlaneTable& t, const std::vector<WeightPlaneEntry>& mats) {
  t.e = mats; size_t halves = 0, nscale = 0; int tiles = 0; std::vector<WPlaneJob> jobs;
  for (auto& x : t.e) {
    if (x.part == 0) { x.part = x.out; x.stride = 0; }
    const int lr = tc_ldp(x.in), lc = tc_ldp(x.out);
    halves += 2 * ((size_t)x.out * lr + (size_t)x.in * lc); nscale += (size_t)x.out + x.in + 8;
  }
  if (t.e.empty()) return GN_OK;
  GN_TRY(t.planes.alloc(halves / 2 + 64)); GN_TRY(t.scales.alloc(nscale)); GN_TRY(t.mx.alloc(t.e.size() + 4));
  GN_CUDA(cudaMemsetAsync(t.planes.p, 0, (halves / 2 + 64) * 4, ctx->stream));
  __half* hp = reinterpret_cast<__half*>(t.planes.p); float* sp = t.scales.p;
  for (auto& x : t.e) {
    const int lr = tc_ldp(x.in), lc = tc_ldp(x.out);
    x.rows = BfPlanes{hp, sp, x.out, x.in, lr, 1}; hp += 2 * (size_t)x.out * lr; sp += (x.out + 3) & ~3;
    x.cols = BfPlanes{hp, sp, x.in, x.out, lc, 1}; hp += 2 * (size_t)x.in * lc; sp += (x.in + 3) & ~3;
    x.maxabs = reinterpret_cast<const int*>(t.mx.p) + jobs.size();
    WPlaneJob jb{x.src, x.bias, x.part, x.stride, x.out, x.in, lr, lc, x.rows.base, x.cols.base, x.rows.inv_scale, x.cols.inv_scale, tiles, (int)cdiv(x.in, 64)};
    x.tile0 = tiles; x.tiles = (int)cdiv(x.out, 64) * (int)cdiv(x.in, 64);
    tiles += x.tiles; jobs.push_back(jb);
  }
  t.total_tiles = tiles;
  GN_TRY(t.jobs.alloc((jobs.size() * sizeof(WPlaneJob) + 3) / 4));
  GN_CUDA(copy_h2d(ctx, t.jobs.p, jobs.data(), jobs.size() * sizeof(WPlaneJob)));
  std::vector<PlaneRange> rg;
  for (auto& x : t.e) rg.push_back(PlaneRange{x.src, x.src + (x.out / x.part - 1) * x.stride + (size_t)x.part * x.in + (x.bias ? x.part : 0)});
  GN_TRY(t.ranges.alloc(rg.size() * sizeof(PlaneRange) / 4)); GN_CUDA(copy_h2d(ctx, t.ranges.p, rg.data(), rg.size() * sizeof(PlaneRange)));
  t.dirty = true; t.max_ok = false; return GN_OK;
}
// Re-splits every registered matrix if the parameters changed since the last call.
// Entries [j0, j1) only, on `stream`: used right behind a layer's parameter update when the update runs layer by layer.
inline int wplanes_max(Ctx* ctx, WeightPlaneTable& t, int j0, int j1, cudaStream_t stream) {
  const int tile_off = t.e[j0].tile0, ntiles = t.e[j1 - 1].tile0 + t.e[j1 - 1].tiles - tile_off;
  GN_CUDA(stream_zero(ctx, stream, reinterpret_cast<int*>(t.mx.p) + j0, (size_t)(j1 - j0) * sizeof(int)));
  GN_LAUNCH_ON(ctx, stream, wplanes_max_kernel, ntiles, 256, 0, reinterpret_cast<const WPlaneJob*>(t.jobs.p), (int)t.e.size(), reinterpret_cast<int*>(t.mx.p), tile_off);
  return check_launch("wplanes_max");
}
inline int wplanes_split(Ctx* ctx, WeightPlaneTable& t, int j0, int j1, cudaStream_t stream) {
  const int tile_off = t.e[j0].tile0, ntiles = t.e[j1 - 1].tile0 + t.e[j1 - 1].tiles - tile_off;
  GN_LAUNCH_ON(ctx, stream, wplanes_split_kernel, ntiles, 256, 0, reinterpret_cast<const WPlaneJob*>(t.jobs.p), (int)t.e.size(), reinterpret_cast<const int*>(t.mx.p), tile_off);
  double elems = 0; for (int j = j0; j < j1; j++) elems += (double)t.e[j].out * t.e[j].in;
  ctx->split_bytes += 12.0 * elems;
  return check_launch("wplanes_split");
}
inline int wplanes_refresh_range(Ctx* ctx, WeightPlaneTable& t, int j0, int j1, cudaStream_t stream) {
  if (j1 <= j0) return GN_OK;
  GN_TRY(wplanes_max(ctx, t, j0, j1, stream));
  return wplanes_split(ctx, t, j0, j1, stream);
}
// The maxima, where the last change of the parameters was not a training step's update.
inline int wplanes_need_max(Ctx* ctx, WeightPlaneTable& t) {
  if (t.e.empty() || !t.used || t.max_ok) return GN_OK;
  GN_TRY(wplanes_max(ctx, t, 0, (int)t.e.size(), ctx->stream));
  t.max_ok = true; return GN_OK;
}
inline int wplanes_refresh(Ctx* ctx, WeightPlaneTable& t) {
  if (t.e.empty() || !t.dirty) return GN_OK;
  if (!t.max_ok) { GN_TRY(wplanes_max(ctx, t, 0, (int)t.e.size(), ctx->stream)); t.max_ok = true; }
  GN_TRY(wplanes_split(ctx, t, 0, (int)t.e.size(), ctx->stream));
  t.dirty = false; return GN_OK;
}
// Prepared planes for B of this contraction, if B is a registered matrix used in one of its two orientations.
inline bool wplanes_lookup(Ctx* ctx, const GemmDesc& g, BfPlanes* p, const WeightPlaneEntry** entry = nullptr) {
  WeightPlaneTable* t = static_cast<WeightPlaneTable*>(ctx->weight_planes);
  if (!t || g.batch1 * g.batch2 != 1) return false;
  int part = 0; const WeightPlaneEntry* x = t->find(g.B, &part); if (!x) return false;
  const int r0 = part * x->part;
  const bool stored = g.sb_k == 1 && g.sb_n == x->in && g.K == x->in && g.N % x->part == 0 && r0 + g.N <= x->out;          // B(k, n) = W[r0 + n, k]
  const bool transposed = !stored && g.sb_n == 1 && g.sb_k == x->in && g.N == x->in && g.K % x->part == 0 && r0 + g.K <= x->out;      // B(k, n) = W[r0 + k, n]
  if (!stored && !transposed) return false;
  if (t->dirty && wplanes_refresh(ctx, *t) != GN_OK) return false;         // once per parameter update, when the first product asks
  t->used = true;
  if (entry) *entry = x;
  if (stored) { *p = x->rows; p->base += 2 * (long)r0 * p->ldp; p->inv_scale += r0; p->rows = g.N; }
  else { *p = x->cols; p->koff = r0; p->K = g.K; }
  return true;
}

// Can the engine run this contraction at all?  One of each operand's strides must be 1; LINEAR/RELU epilogue; alpha 1.
inline bool gemm_tc_supported(Ctx* ctx, const GemmDesc& g) {
  if (!ctx->tc_ok) return false;
  if (g.alpha != 1.f) return false;
  if (!(g.sa_k == 1 || g.sa_m == 1)) return false;
  if (!(g.sb_k == 1 || g.sb_n == 1)) return false;
  if (g.act != GN_ACT_LINEAR && g.act != GN_ACT_RELU && !(g.act == GN_ACT_GELU && g.plane_out)) return false;
  return g.M > 0 && g.N > 0 && g.K > 0;
}
// Is it worth it?  Small or skinny problems stay on the CUDA-core engine, which needs no operand planes: 1e8 multiply-adds take it
// about 8 us.  Products over many rows come here somewhat earlier: several of them share the planes of one input (Q, K and V).
inline bool gemm_tc_eligible(Ctx* ctx, const GemmDesc& g) {
  if (!gemm_tc_supported(ctx, g)) return false;
  const double work = (double)g.M * g.N * g.K * g.batch1 * g.batch2;
  return g.M >= 16 && g.N >= 32 && g.K >= 32 && work >= (g.M >= 512 ? 6.0e7 : 1.0e8);
}

// General entry: splits both operands into the context's scratch planes, then runs the contraction.
inline int gemm_tc(Ctx* ctx, const GemmDesc& g) {
  if (!gemm_tc_supported(ctx, g)) return fail(GN_ERR_UNSUPPORTED, "tcgen05 engine cannot run this contraction");
  TcScratch& sc = tc_scratch(ctx);
  const int nb = g.batch1 * g.batch2;
  const float* last_a = sc.last_a; const float* pa = sc.a.p; const float* psa = sc.sa.p;   // tc_planes() forgets the A planes' origin when it hands the buffer out
  BfPlanes A, B; GN_TRY(tc_planes(ctx, 0, nb, g.M, g.K, &A)); GN_TRY(tc_planes(ctx, 1, nb, g.N, g.K, &B));
  int* mx = tc_rowmax_buf(ctx);
  sc.last_a = (sc.a.p == pa && sc.sa.p == psa) ? last_a : nullptr;                          // still valid unless a buffer was replaced
  if (g.a_planes) {
    A = *static_cast<const BfPlanes*>(g.a_planes);
    if (A.rows != g.M || A.K != g.K || A.nbatch != nb) return fail(GN_ERR_INVALID_ARG, "gemm_tc: prepared planes of A do not match the contraction");
  } else if (g.m_seg) {
    // the rows of A (a transposed operand) come from M / m_seg arrays: as a batch, whose planes lie one after the other
    if (g.sa_m != 1 || nb != 1 || g.M % g.m_seg) return fail(GN_ERR_INVALID_ARG, "gemm_tc: row segments need a transposed A");
    BfPlanes S = A; S.rows = g.m_seg; S.nbatch = g.M / g.m_seg;
    GN_TRY(tc_split(ctx, TcSrc{g.A, g.sa_m, g.sa_k, g.a_seg, 0, 1}, S, mx)); sc.last_a = nullptr;
  } else if (g.k_seg) {
    if (g.sa_k != 1 || nb != 1 || g.k_seg % 32) return fail(GN_ERR_INVALID_ARG, "gemm_tc: contraction segments need a row-major A and a multiple of 32");
    GN_TRY(tc_split(ctx, TcSrc{g.A, g.sa_m, g.sa_k, g.a_b1, g.a_b2, g.batch2, g.k_seg, g.a_seg}, A, mx, g.a_rownorm)); sc.last_a = nullptr;
  } else if (!g.a_rownorm && g.reuse_a_planes && nb == 1 && sc.last_a == g.A && sc.last_m == g.M && sc.last_k == g.K && sc.last_ld == g.sa_m && g.sa_k == 1) {
    // same tensor as the previous call (the Q, K and V projections share their input): planes still valid
  } else {
    GN_TRY(tc_split(ctx, TcSrc{g.A, g.sa_m, g.sa_k, g.a_b1, g.a_b2, g.batch2, 0, 0, g.z_first}, A, mx, g.a_rownorm));
    sc.last_a = (nb == 1 && g.sa_k == 1) ? g.A : nullptr; sc.last_m = g.M; sc.last_k = g.K; sc.last_ld = g.sa_m;
  }
  if (g.b_planes) {
    B = *static_cast<const BfPlanes*>(g.b_planes);
    if (B.rows != g.N || B.K != g.K || B.nbatch != nb) return fail(GN_ERR_INVALID_ARG, "gemm_tc: prepared planes of B do not match the contraction");
  } else GN_TRY(tc_split(ctx, TcSrc{g.B, g.sb_n, g.sb_k, g.b_b1, g.b_b2, g.batch2, 0, 0, g.z_first}, B, mx));
  TcParams ep{g.C, g.ldc, g.c_b1, g.c_b2, g.bias, g.R, g.ldr, g.r_b1, g.r_b2, g.act, g.M, g.N, g.K, g.batch2, g.flags, ctx->d_status, g.mask, g.mask_ld, g.mask_group}; ep.z_first = g.z_first;
  if (g.n_seg) {
    if (g.n_seg % 32 || nb != 1 || g.R || g.plane_out) return fail(GN_ERR_INVALID_ARG, "gemm_tc: this contraction cannot write its columns in segments");
    ep.n_seg = g.n_seg; ep.c_seg = g.c_seg; ep.bias_seg = g.bias_seg;
    ep.zmax = g.zmax; ep.zmax_T = g.zmax_T; ep.zmax_H = g.n_seg / 64; ep.zmax_seg = 3L * (g.M / std::max(1, g.zmax_T)) * ep.zmax_H;
  }
  if (g.plane_out) {
    const TcPlaneOut& po = *static_cast<const TcPlaneOut*>(g.plane_out);
    if (nb != 1 || g.R || !g.a_rownorm || !po.b_maxabs || g.N % 32 || po.planes.rows != g.M || po.planes.K != g.N || (g.flags & (GEMM_SKIP_UPPER | GEMM_KBEG_AT_M0 | GEMM_KEND_AT_M0)))
      return fail(GN_ERR_INVALID_ARG, "gemm_tc: this contraction cannot write its result as operand planes");
    ep.out_p = po.planes.base; ep.out_inv = po.planes.inv_scale; ep.out_ldp = po.planes.ldp;
    ep.a_rownorm = g.a_rownorm; ep.b_maxabs = po.b_maxabs; ep.c_last = po.last; ep.last_T = po.last_T > 0 ? po.last_T : 1; ep.rowsum32 = po.rowsum32; ep.z_last = po.z_last;
    if (po.scale) ep.flags |= TC_FLAG_SCALE;
  }
  return tc_run(ctx, A, B, ep);
}

}  // namespace gn
