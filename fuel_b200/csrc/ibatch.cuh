// Integer matmul for a few to a few dozen activation rows (a dense batch, or the rows routed to one expert) on the integer
// tensor cores: every weight format, rows of whole 256-element stretches. One pass over the weights serves up to 64 rows.
//
// Arithmetic: the reference's vec_dot per (weight row, activation row) - exact integer dot products of the packed weights
// with the 8-bit activation blocks, combined per block in f32 (fuel-quantized/src/k_quants.rs:1388-1468 Q4_K, 1946-2003
// Q6_K, 674-692 Q8_0, 783-833 Q2_K, 1013-1133 Q3_K, 1626-1760 Q5_K, 252-533 the other 32-element formats). Only the f32
// summation order over blocks differs from the CPU path.
//
// Mapping: the WEIGHTS are the 16-row operand of mma.sync and 8 activation rows the other, so a 16-row weight tile is
// unpacked once per 256 elements (32 registers a lane) and used by all of the activation rows' 8-column tiles:
//   Q4_K, Q5_K   m16n8k32 u8 x s8, one per 32-element sub-block; S += scale * c in integers
//   Q6_K, Q3_K   m16n8k16 s8 x s8, one per 16-element group; the values minus their offset, left-justified in the byte
//                (4 * (q - 32), 32 * (q - 4)), which makes the offset a flipped top bit and costs only a power of two
//   Q2_K         m16n8k32, the 4-bit scale multiplied into the 2-bit values (at most 45): accumulates over the whole block
//   Q8_0, Q4_0, Q5_0, Q4_1, Q5_1   m16n8k32 per 32-element block, scaled in f32 (left-justified as above where signed)
// The minimums of Q4_K / Q5_K / Q2_K are one f16 MMA per 256 elements: minimums and 16-element activation sums (at most
// 2032 in magnitude) are exact in f16, their products' sum (below 2^24) in f32.
//
// What bounds it: HBM up to some 32 rows, above that the shared-memory reads of the activation fragments (2 KB per 16 x 8 x
// 256 tile, 16 cycles) and the integer multiply-adds (half rate), about 20 cycles a tile and SM; measured rates on this
// part: m16n8k32 s8 2.1 cycles a SM, m16n8k16 s8 2.1, m16n8k16 f16 2.2.
//
// Work split: a warp owns one 16-row tile and one contiguous share of k (`kp` shares) for a whole round, its accumulators in
// registers to the end; the shares' sums then meet in shared memory and are added in order. Warps stream their own weights
// with cp.async into private stages: no producer and no barrier between warps on that path (a bulk copy per row segment was
// bound by its issue rate, 60-90 ns each). The activations of a chunk (each share's next `bpc` blocks) are staged for the whole
// thread block by one bulk copy per block, double-buffered when k does not fit at once, with one barrier per chunk: they are
// as many bytes per SM as the weights (every SM needs all of them), and copied by the threads, 16 bytes each, they cost
// more instructions than the arithmetic.
#pragma once
#include "decode_regs.cuh"
#include "fq_common.cuh"

namespace fq {

constexpr int kIbMaxWarps = 16;
constexpr int kIbHeader = 128;    // barriers, at the start of shared memory
constexpr int kIbMaxRows = 64;    // activation rows per pass
constexpr int kIbGroupRows = 32;  // and of the grouped form

enum IbAct { kIbQ8K, kIbQ8_0, kIbQ8_1 };
__host__ __device__ constexpr int ib_rec(IbAct a) { return a == kIbQ8_1 ? kActRecordMin : kActRecord; }  // bytes per row of a slot

struct IbParams {
  const uint8_t* w;      // [n_groups][n][k] blocks
  ActPlanes act;         // activation planes of all rows
  const int* offsets;    // [n_groups + 1] row ranges, or null: one group holding rows [0, fixed_rows)
  const int* out_rows;   // row -> output row, or null for the identity
  float* y;              // [rows][n]
  int64_t group_bytes;   // n * row_bytes
  int64_t total_bytes;   // n_groups * group_bytes
  int fixed_rows;
  int64_t act_rows;      // rows of the records
  int early_w;           // one matrix: the weights are streamed before the wait for the preceding kernel
  int n, nblk, row_bytes, n_groups;
  int rows_cap;          // activation rows per pass (a multiple of 8, at most 8 * MT)
  int kp;                // shares of k; the warps of a tile
  int share_q, share_rem;  // blocks per share: share_q, one more in the first share_rem
  int tg;                // tiles per round (warps / kp)
  int bpc, n_chunks;     // blocks of every share per chunk of activations
  int stages;            // weight stages per warp
  int act_off, act_buf;  // shared-memory offset of the activation buffers, bytes of one
  int part_off;          // and of the partial sums
};

// Launches the kernel of a weight type for mt 8-row tiles (ibatch.cu)
cudaError_t ibatch_launch(int type, int mt, bool grouped, const IbParams& p, unsigned grid, int warps, size_t smem, int max_smem, cudaStream_t stream);
cudaError_t ibatch_device_error(int* code, bool clear);  // the error word of these kernels

// ---- small pieces
__device__ __forceinline__ void ib_cp16(uint32_t dst, const void* src, uint32_t bytes) {  // bytes past `bytes` become zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ib_cp4(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ib_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void ib_wait(int pending) {  // until at most `pending` of this thread's newest groups are in flight
  switch (pending) {
    case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
  }
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
// The MMA wrappers are pure functions of their operands: not volatile, so the compiler may schedule them among the
// surrounding arithmetic; the shared-memory loads stay volatile and keep their order against the barriers.
// kFresh: c = A * B, else c += A * B.
#define FQ_IB_MMA_K32(NAME, TYPE)                                                                                            \
  template <bool kFresh>                                                                                                     \
  __device__ __forceinline__ void NAME(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {                      \
    if constexpr (kFresh)                                                                                                    \
      asm("mma.sync.aligned.m16n8k32.row.col.s32." TYPE ".s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"  \
          : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])                                                                   \
          : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));                                           \
    else                                                                                                                     \
      asm("mma.sync.aligned.m16n8k32.row.col.s32." TYPE ".s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"      \
          : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])                                                                   \
          : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));                                                   \
  }
FQ_IB_MMA_K32(mma_u8_k32, "u8")
FQ_IB_MMA_K32(mma_s8_k32, "s8")
#undef FQ_IB_MMA_K32
__device__ __forceinline__ void mma_s8_k16(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
      : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}
__device__ __forceinline__ void mma_f16_k16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t lds_u32_2b_addr(uint32_t a) {
  const uint32_t base = a & ~3u;
  uint32_t lo, hi;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(lo) : "r"(base));
  asm volatile("ld.shared.u32 %0, [%1+4];" : "=r"(hi) : "r"(base));
  return __funnelshift_r(lo, hi, (a & 2u) * 8u);
}
__device__ __forceinline__ uint32_t lds_u16_addr(uint32_t a) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void ib_sums16(uint32_t dst, const int16_t* src) {  // eight sums of the plane as f16
  const int4 v = *reinterpret_cast<const int4*>(src);
  const int in[4] = {v.x, v.y, v.z, v.w};
  uint32_t h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __half2 p = __halves2half2(__int2half_rn((int16_t)in[i]), __int2half_rn(in[i] >> 16));
    h[i] = *reinterpret_cast<const uint32_t*>(&p);
  }
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]) : "memory");
}
__device__ __forceinline__ int ib_byte(uint32_t w, int i) { return (int)((w >> (8 * i)) & 0xffu); }
__device__ __forceinline__ int ib_sbyte(uint32_t w, int i) { return (int)(int8_t)((w >> (8 * i)) & 0xffu); }
__device__ __forceinline__ uint32_t ib_h2(int a, int b) {  // two small integers as packed f16
  const __half2 h = __floats2half2_rn((float)a, (float)b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Cost of a tile for a group of r rows, in 8-row tiles: its unpacking and streaming weigh about as much as three of them
__device__ __forceinline__ int ib_group_cost(int r, int rows_cap) {
  return r > 0 ? 3 * ((r + rows_cap - 1) / rows_cap) + ((r + 7) >> 3) : 0;
}

// Where a warp's operands are: shared addresses
struct IbCtx {
  uint32_t r0, r1;   // weight rows gid and gid + 8 of the tile, at this block (skew included)
  uint32_t lm;       // ldmatrix row address of this lane (rows (lane & 7) + 8 * bit 3, byte 16 * bit 4), aligned formats
  uint32_t act;      // this block's activation slot: one record per row
  int lane, gid, tig, nt;
};

// The activation tiles of a step, in parts that run together: with a branch around each tile, none of one tile's loads and
// products can be issued under the latency of another's (Q4_K 11008 x 4096, 48 rows: 45 us, with parts 35); with all of eight,
// or three of the sixteen-group formats at the sixteen-warp form's 128 registers, the registers spill (64 rows: 51 and 77 us).
__host__ __device__ constexpr int ib_part(int nt, int small, int large) {
  return nt <= 2 ? nt : nt <= 4 ? (small < nt ? small : nt) : nt <= 6 ? nt : large;
}
#define FQ_IB_TILES(SMALL, LARGE)                                                                                  \
  _Pragma("unroll") for (int mq = 0; mq < NT; mq += ib_part(NT, SMALL, LARGE)) if (mq == 0 || mq < cx.nt) \
      _Pragma("unroll") for (int mt = mq; mt < NT && mt < mq + ib_part(NT, SMALL, LARGE); ++mt)

// Quant fragments of activation tile mt for 64 elements from element 64 * g: b[0..1] the first 32, b[2..3] the second
template <int kRec = kActRecord>
__device__ __forceinline__ void ib_b64(const IbCtx& cx, int mt, int g, uint32_t (&b)[4]) {
  ldmatrix_x4(b, cx.act + (uint32_t)(8 * mt + (cx.lane & 7)) * (uint32_t)kRec + 64u * g + 16u * (cx.lane >> 3));
}

// facc += y_d * (d * S - dmin * (minimums . 16-element sums)) of one block; am = the minimums as an f16 A fragment
template <int MT>
__device__ __forceinline__ void ib_finish_min(const IbCtx& cx, int mt, const uint32_t (&am)[4], const int (&S)[4], float d0, float dm0,
                                              float d1, float dm1, float (&facc)[MT][4]) {
  const uint32_t ba = cx.act + (uint32_t)(8 * mt + cx.gid) * kActRecord + kActRecAux + 4u * cx.tig;
  float t[4];
  mma_f16_k16(t, am, lds32(ba), lds32(ba + 16u));
  const uint32_t da = cx.act + (uint32_t)(8 * mt + 2 * cx.tig) * kActRecord + kActRecD;
  const float ya = __uint_as_float(lds32(da)), yb = __uint_as_float(lds32(da + kActRecord));
  facc[mt][0] += ya * (d0 * (float)S[0] - dm0 * t[0]);
  facc[mt][1] += yb * (d0 * (float)S[1] - dm0 * t[1]);
  facc[mt][2] += ya * (d1 * (float)S[2] - dm1 * t[2]);
  facc[mt][3] += yb * (d1 * (float)S[3] - dm1 * t[3]);
}

// ------------------------------------------------------------------------------------------------ Q4_K / Q5_K
template <bool kFive>
struct IbQ45K {
  static constexpr int kBytes256 = kFive ? 176 : 144, kPitch = kBytes256;  // 144 and 176 both spread eight rows over the banks
  static constexpr bool kAligned = true;
  static constexpr IbAct kAct = kIbQ8K;
  static constexpr bool kSums = true;  // reads the 16-element sums
  template <int NT, int MT>
  __device__ __forceinline__ static void block(const IbCtx& cx, float (&facc)[MT][4]) {
    // Eight 6-bit scales per row as bytes of two words (get_scale_min_k4, fuel-quantized/src/utils.rs:50-60). The rest of the
    // block's first 16 bytes is read again behind the loop: held across it, it takes registers that the two-tile form spills
    // (4096 x 11008, 16 rows: 20.6 us, read again 19.9).
    uint32_t sc0[2], sc1[2];
    {
      const uint4 h0 = lds128(cx.r0), h1 = lds128(cx.r1);
      sc0[0] = h0.y & 0x3f3f3f3fu, sc0[1] = (h0.w & 0x0f0f0f0fu) | (((h0.y >> 6) & 0x03030303u) << 4);
      sc1[0] = h1.y & 0x3f3f3f3fu, sc1[1] = (h1.w & 0x0f0f0f0fu) | (((h1.y >> 6) & 0x03030303u) << 4);
    }
    uint32_t hq[4];
    if constexpr (kFive) ldmatrix_x4(hq, cx.lm + 16u);
    int S[NT][4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {  // 64 elements: low nibbles = sub-block 2g, high nibbles = 2g + 1
      uint32_t r[4], lo[4], hi[4];
      ldmatrix_x4(r, cx.lm + (kFive ? 48u : 16u) + 32u * g);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        lo[i] = r[i] & 0x0f0f0f0fu, hi[i] = (r[i] >> 4) & 0x0f0f0f0fu;
        if constexpr (kFive) {
          lo[i] |= ((hq[i] >> (2 * g)) & 0x01010101u) << 4;
          hi[i] |= ((hq[i] >> (2 * g + 1)) & 0x01010101u) << 4;
        }
      }
      const int s0l = ib_byte(sc0[g >> 1], 2 * (g & 1)), s0h = ib_byte(sc0[g >> 1], 2 * (g & 1) + 1);
      const int s1l = ib_byte(sc1[g >> 1], 2 * (g & 1)), s1h = ib_byte(sc1[g >> 1], 2 * (g & 1) + 1);
      FQ_IB_TILES(4, 4) {
        uint32_t b[4];
        ib_b64(cx, mt, g, b);
        int cl[4], ch[4];
        mma_u8_k32<true>(cl, lo, b[0], b[1]);
        mma_u8_k32<true>(ch, hi, b[2], b[3]);
        int (&T)[4] = S[mt];
        // one product at a time where many tiles run together: fewer registers (48 rows: 33.0 -> 32.5 us, 32 rows 28.8 -> 27.7;
        // the two-tile form 19.9 -> 21.2)
        if constexpr (NT > 2) {
          if (g == 0) T[0] = cl[0] * s0l, T[1] = cl[1] * s0l, T[2] = cl[2] * s1l, T[3] = cl[3] * s1l;
          else T[0] += cl[0] * s0l, T[1] += cl[1] * s0l, T[2] += cl[2] * s1l, T[3] += cl[3] * s1l;
          T[0] += ch[0] * s0h, T[1] += ch[1] * s0h, T[2] += ch[2] * s1h, T[3] += ch[3] * s1h;
        } else if (g == 0) {
          T[0] = cl[0] * s0l + ch[0] * s0h, T[1] = cl[1] * s0l + ch[1] * s0h;
          T[2] = cl[2] * s1l + ch[2] * s1h, T[3] = cl[3] * s1l + ch[3] * s1h;
        } else {
          T[0] += cl[0] * s0l + ch[0] * s0h, T[1] += cl[1] * s0l + ch[1] * s0h;
          T[2] += cl[2] * s1l + ch[2] * s1h, T[3] += cl[3] * s1l + ch[3] * s1h;
        }
      }
    }
    const uint4 h0 = lds128(cx.r0), h1 = lds128(cx.r1);
    const uint32_t mn0[2] = {h0.z & 0x3f3f3f3fu, ((h0.w >> 4) & 0x0f0f0f0fu) | (((h0.z >> 6) & 0x03030303u) << 4)};
    const uint32_t mn1[2] = {h1.z & 0x3f3f3f3fu, ((h1.w >> 4) & 0x0f0f0f0fu) | (((h1.z >> 6) & 0x03030303u) << 4)};
    const float d0 = h2f_bits(h0.x & 0xffffu), dm0 = h2f_bits(h0.x >> 16);
    const float d1 = h2f_bits(h1.x & 0xffffu), dm1 = h2f_bits(h1.x >> 16);
    uint32_t am[4];  // minimum of 16-element group i = minimum of sub-block i / 2: this lane's groups 2 tig, + 1, + 8, + 9
    {
      const int a = ib_byte(mn0[0], cx.tig), b = ib_byte(mn1[0], cx.tig), c = ib_byte(mn0[1], cx.tig), e = ib_byte(mn1[1], cx.tig);
      am[0] = ib_h2(a, a), am[1] = ib_h2(b, b), am[2] = ib_h2(c, c), am[3] = ib_h2(e, e);
    }
    FQ_IB_TILES(4, 4)
      ib_finish_min(cx, mt, am, S[mt], d0, dm0, d1, dm1, facc);
  }
};
using IbQ4K = IbQ45K<false>;
using IbQ5K = IbQ45K<true>;

// ------------------------------------------------------------------------------------------------ Q6_K, Q3_K
// Sixteen groups of 16 elements, each with a signed scale (bytes of sc0 / sc1 for rows gid / gid + 8): step g takes groups
// 4g .. 4g + 3, A[i] = the left-justified values of group 4g + i
template <int NT>
__device__ __forceinline__ void ib_groups16_step(const IbCtx& cx, int g, const uint32_t (&A)[4][2], uint32_t sc0, uint32_t sc1, int (&S)[NT][4]) {
  int s0[4], s1[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) s0[i] = ib_sbyte(sc0, i), s1[i] = ib_sbyte(sc1, i);
  FQ_IB_TILES(2, 4) {
    uint32_t b[4];
    ib_b64(cx, mt, g, b);
    int (&T)[4] = S[mt];
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      int c[4], e[4];
      mma_s8_k16(c, A[i][0], A[i][1], b[i]);
      mma_s8_k16(e, A[i + 1][0], A[i + 1][1], b[i + 1]);
      if (g == 0 && i == 0) T[0] = c[0] * s0[i], T[1] = c[1] * s0[i], T[2] = c[2] * s1[i], T[3] = c[3] * s1[i];
      else T[0] += c[0] * s0[i], T[1] += c[1] * s0[i], T[2] += c[2] * s1[i], T[3] += c[3] * s1[i];
      T[0] += e[0] * s0[i + 1], T[1] += e[1] * s0[i + 1], T[2] += e[2] * s1[i + 1], T[3] += e[3] * s1[i + 1];
    }
  }
}
template <int NT, int MT>
__device__ __forceinline__ void ib_groups16_finish(const IbCtx& cx, const int (&S)[NT][4], float d0, float d1, float (&facc)[MT][4]) {
  FQ_IB_TILES(2, 4) {
    const uint32_t da = cx.act + (uint32_t)(8 * mt + 2 * cx.tig) * kActRecord + kActRecD;
    const float ya = __uint_as_float(lds32(da)), yb = __uint_as_float(lds32(da + kActRecord));
    facc[mt][0] += (d0 * ya) * (float)S[mt][0];
    facc[mt][1] += (d0 * yb) * (float)S[mt][1];
    facc[mt][2] += (d1 * ya) * (float)S[mt][2];
    facc[mt][3] += (d1 * yb) * (float)S[mt][3];
  }
}

struct IbQ6K {
  static constexpr int kBytes256 = 210, kPitch = 240;  // fetched as 14 16-byte pieces (skew 0..14)
  static constexpr bool kAligned = false;
  static constexpr IbAct kAct = kIbQ8K;
  static constexpr bool kSums = false;
  template <int NT, int MT>
  __device__ __forceinline__ static void block(const IbCtx& cx, float (&facc)[MT][4]) {
    int S[NT][4];
    // 4 * (q - 32) of quadrant q of half h: elements 128 h + 32 q + l (k_quants.rs:2170-2185), l = 16 s + 4 tig .. + 3
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t qa[2][2], qb[2][2], qh[2][2];  // [s][row]
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint32_t row = (r ? cx.r1 : cx.r0) + 16u * s + 4u * cx.tig;
          qa[s][r] = lds_u32_2b_addr(row + 64u * h), qb[s][r] = lds_u32_2b_addr(row + 64u * h + 32u);
          qh[s][r] = lds_u32_2b_addr(row + 128u + 32u * h);
        }
#pragma unroll
      for (int u = 0; u < 2; ++u) {  // quadrants 2u, 2u + 1: the low nibbles, then the high ones
        uint32_t A[4][2];
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const uint32_t a = u ? qa[s][r] >> 2 : qa[s][r] << 2, b = u ? qb[s][r] >> 2 : qb[s][r] << 2;
            const uint32_t ha = u ? qh[s][r] << 2 : qh[s][r] << 6, hb = u ? qh[s][r] : qh[s][r] << 4;
            A[s][r] = ((a & 0x3c3c3c3cu) ^ 0x80808080u) ^ (ha & 0xc0c0c0c0u);
            A[2 + s][r] = ((b & 0x3c3c3c3cu) ^ 0x80808080u) ^ (hb & 0xc0c0c0c0u);
          }
        const int g = 2 * h + u;
        ib_groups16_step<NT>(cx, g, A, lds_u32_2b_addr(cx.r0 + 192u + 4u * g), lds_u32_2b_addr(cx.r1 + 192u + 4u * g), S);
      }
    }
    const float d0 = 0.25f * h2f_bits(lds_u16_addr(cx.r0 + 208u)), d1 = 0.25f * h2f_bits(lds_u16_addr(cx.r1 + 208u));
    ib_groups16_finish<NT>(cx, S, d0, d1, facc);
  }
};

struct IbQ3K {
  static constexpr int kBytes256 = 110, kPitch = 144;  // fetched as eight pieces
  static constexpr bool kAligned = false;
  static constexpr IbAct kAct = kIbQ8K;
  static constexpr bool kSums = false;
  __device__ __forceinline__ static void scales(uint32_t row, uint32_t (&sc)[4]) {  // k_quants.rs:1095-1103, minus 32 per byte
    const uint32_t a = lds_u32_2b_addr(row + 96u), b = lds_u32_2b_addr(row + 100u), c = lds_u32_2b_addr(row + 104u);
    sc[0] = (a & 0x0f0f0f0fu) | ((c & 0x03030303u) << 4);
    sc[1] = (b & 0x0f0f0f0fu) | (((c >> 2) & 0x03030303u) << 4);
    sc[2] = ((a >> 4) & 0x0f0f0f0fu) | (((c >> 4) & 0x03030303u) << 4);
    sc[3] = ((b >> 4) & 0x0f0f0f0fu) | (((c >> 6) & 0x03030303u) << 4);
#pragma unroll
    for (int i = 0; i < 4; ++i) sc[i] = ((sc[i] | 0x80808080u) - 0x20202020u) ^ 0x80808080u;
  }
  template <int NT, int MT>
  __device__ __forceinline__ static void block(const IbCtx& cx, float (&facc)[MT][4]) {
    uint32_t sc0[4], sc1[4], hm[2][2];  // hm: [s][row]
    scales(cx.r0, sc0);
    scales(cx.r1, sc1);
    int S[NT][4];
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int r = 0; r < 2; ++r) hm[s][r] = lds_u32_2b_addr((r ? cx.r1 : cx.r0) + 16u * s + 4u * cx.tig);
    // 32 * (q - 4): element 128 c + 32 j + b has its low bits in qs[32 c + b] at 2 j, its high bit in hmask[b] at 4 c + j
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t q[2][2];
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int r = 0; r < 2; ++r) q[s][r] = lds_u32_2b_addr((r ? cx.r1 : cx.r0) + 32u + 32u * c + 16u * s + 4u * cx.tig);
#pragma unroll
      for (int u = 0; u < 2; ++u) {  // bit pairs 2u, 2u + 1
        uint32_t A[4][2];
#pragma unroll
        for (int jj = 0; jj < 2; ++jj)
#pragma unroll
          for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int j = 2 * u + jj;
              A[2 * jj + s][r] = (((q[s][r] >> (2 * j)) & 0x03030303u) << 5) ^ ((((hm[s][r] >> (4 * c + j)) & 0x01010101u) << 7) ^ 0x80808080u);
            }
        ib_groups16_step<NT>(cx, 2 * c + u, A, sc0[2 * c + u], sc1[2 * c + u], S);
      }
    }
    const float d0 = 0.03125f * h2f_bits(lds_u16_addr(cx.r0 + 108u)), d1 = 0.03125f * h2f_bits(lds_u16_addr(cx.r1 + 108u));
    ib_groups16_finish<NT>(cx, S, d0, d1, facc);
  }
};

// ------------------------------------------------------------------------------------------------ Q2_K
struct IbQ2K {
  static constexpr int kBytes256 = 84, kPitch = 112;  // fetched as six or seven pieces (skew 0, 4, 8, 12)
  static constexpr bool kAligned = false;
  static constexpr IbAct kAct = kIbQ8K;
  static constexpr bool kSums = true;
  template <int NT, int MT>
  __device__ __forceinline__ static void block(const IbCtx& cx, float (&facc)[MT][4]) {
    uint32_t am[4], sw[2][4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const uint32_t row = r ? cx.r1 : cx.r0;
#pragma unroll
      for (int i = 0; i < 4; ++i) sw[r][i] = lds32(row + 4u * i);  // scale (low nibble) and minimum (high) of 16 groups
      const uint32_t ma = lds_u16_addr(row + 2u * cx.tig), mb = lds_u16_addr(row + 8u + 2u * cx.tig);
      am[r] = ib_h2((int)((ma >> 4) & 0xfu), (int)(ma >> 12)), am[2 + r] = ib_h2((int)((mb >> 4) & 0xfu), (int)(mb >> 12));
    }
    int S[NT][4];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      uint32_t q[2][2];  // [s][row]
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int r = 0; r < 2; ++r) q[s][r] = lds32((r ? cx.r1 : cx.r0) + 16u + 32u * c + 16u * s + 4u * cx.tig);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        uint32_t A[2][4];
#pragma unroll
        for (int jj = 0; jj < 2; ++jj)
#pragma unroll
          for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              const int j = 2 * u + jj, gr = 8 * c + 2 * j + s;
              A[jj][2 * s + r] = ((q[s][r] >> (2 * j)) & 0x03030303u) * (uint32_t)(ib_byte(sw[r][gr >> 2], gr & 3) & 0xf);  // at most 45 a byte
            }
        FQ_IB_TILES(4, 4) {
          uint32_t b[4];
          ib_b64(cx, mt, 2 * c + u, b);
          if (c == 0 && u == 0) mma_u8_k32<true>(S[mt], A[0], b[0], b[1]);
          else mma_u8_k32<false>(S[mt], A[0], b[0], b[1]);
          mma_u8_k32<false>(S[mt], A[1], b[2], b[3]);
        }
      }
    }
    const uint32_t dd0 = lds32(cx.r0 + 80u), dd1 = lds32(cx.r1 + 80u);
    const float d0 = h2f_bits(dd0 & 0xffffu), dm0 = h2f_bits(dd0 >> 16), d1 = h2f_bits(dd1 & 0xffffu), dm1 = h2f_bits(dd1 >> 16);
    FQ_IB_TILES(4, 4)
      ib_finish_min(cx, mt, am, S[mt], d0, dm0, d1, dm1, facc);
  }
};

// ------------------------------------------------------------------------------------------------ the 32-element formats
// kBits 8: f16 scale, 32 signed bytes. 4 / 5: scale (and minimum m when kMin), for 5 the fifth bits qh, 16 bytes of nibbles -
// byte t holds element t (low) and 16 + t (high). Values minus their offset left-justified: 16 (q - 8) or 8 (q - 16).
template <int kBits, bool kMin>
struct Ib32 {
  static constexpr int kBlk = kBits == 8 ? 34 : 2 + (kMin ? 2 : 0) + (kBits == 5 ? 4 : 0) + 16;
  static constexpr int kBytes256 = 8 * kBlk;  // 272, 144, 160, 176 or 192: rows and blocks start on 16-byte boundaries
  static constexpr int kPitch = kBytes256 % 128 == 32 || kBytes256 % 128 == 64 ? kBytes256 + 16 : kBytes256;
  static constexpr bool kAligned = true;
  static constexpr IbAct kAct = kMin ? kIbQ8_1 : kIbQ8_0;
  static constexpr float kUnit = kBits == 8 || kMin ? 1.0f : kBits == 5 ? 0.125f : 0.0625f;
  __device__ __forceinline__ static uint32_t spread4(uint32_t bits) {  // bit i of a nibble -> bit 0 of byte i
    return ((bits & 0xFu) * 0x00204081u) & 0x01010101u;
  }
  // one 32-element block of one row: operand words lo (elements 4 tig ..) and hi (16 + 4 tig ..), scale, minimum
  __device__ __forceinline__ static void row_block(uint32_t p, int tig, uint32_t& lo, uint32_t& hi, float& d, float& mn) {
    auto word = [](uint32_t a) -> uint32_t {
      if constexpr (kBlk % 4 == 0) return lds32(a);
      else return lds_u32_2b_addr(a);
    };
    d = kUnit * h2f_bits(lds_u16_addr(p));
    mn = kMin ? h2f_bits(lds_u16_addr(p + 2u)) : 0.f;
    if constexpr (kBits == 8) {
      lo = word(p + 2u + 4u * tig), hi = word(p + 18u + 4u * tig);
    } else {
      const uint32_t w = word(p + (uint32_t)kBlk - 16u + 4u * tig);
      uint32_t h = 0;
      if constexpr (kBits == 5) h = word(p + (uint32_t)kBlk - 20u);  // bit t belongs to element t
      if constexpr (kMin) {
        lo = w & 0x0f0f0f0fu, hi = (w >> 4) & 0x0f0f0f0fu;
        if constexpr (kBits == 5) lo |= spread4(h >> (4 * tig)) << 4, hi |= spread4(h >> (16 + 4 * tig)) << 4;
      } else if constexpr (kBits == 4) {
        lo = ((w << 4) & 0xf0f0f0f0u) ^ 0x80808080u, hi = (w & 0xf0f0f0f0u) ^ 0x80808080u;
      } else {
        lo = ((w << 3) & 0x78787878u) ^ ((spread4(h >> (4 * tig)) << 7) ^ 0x80808080u);
        hi = ((w >> 1) & 0x78787878u) ^ ((spread4(h >> (16 + 4 * tig)) << 7) ^ 0x80808080u);
      }
    }
  }
  template <int NT, int MT>
  __device__ __forceinline__ static void block(const IbCtx& cx, float (&facc)[MT][4]) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {  // two 32-element blocks at a time
      uint32_t A[2][4];
      float d0[2], d1[2], m0[2], m1[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        row_block(cx.r0 + (uint32_t)(kBlk * (2 * g + h)), cx.tig, A[h][0], A[h][2], d0[h], m0[h]);
        row_block(cx.r1 + (uint32_t)(kBlk * (2 * g + h)), cx.tig, A[h][1], A[h][3], d1[h], m1[h]);
      }
      FQ_IB_TILES(4, 4) {
        uint32_t b[4];
        constexpr int kRec = ib_rec(kAct);
        ib_b64<kRec>(cx, mt, g, b);
        const uint32_t da = cx.act + (uint32_t)(8 * mt + 2 * cx.tig) * kRec + kActRecAux + 8u * g;
        const uint2 ya = lds64(da), yb = lds64(da + kRec);
        uint2 sa = make_uint2(0, 0), sb = sa;
        if constexpr (kMin) sa = lds64(da + 32u), sb = lds64(da + 32u + kRec);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          int c[4];
          if constexpr (kMin) mma_u8_k32<true>(c, A[h], b[2 * h], b[2 * h + 1]);
          else mma_s8_k32<true>(c, A[h], b[2 * h], b[2 * h + 1]);
          const float fa = __uint_as_float(h ? ya.y : ya.x), fb = __uint_as_float(h ? yb.y : yb.x);
          facc[mt][0] += (d0[h] * fa) * (float)c[0];
          facc[mt][1] += (d0[h] * fb) * (float)c[1];
          facc[mt][2] += (d1[h] * fa) * (float)c[2];
          facc[mt][3] += (d1[h] * fb) * (float)c[3];
          if constexpr (kMin) {
            const float ga = __uint_as_float(h ? sa.y : sa.x), gb = __uint_as_float(h ? sb.y : sb.x);
            facc[mt][0] += m0[h] * ga, facc[mt][1] += m0[h] * gb, facc[mt][2] += m1[h] * ga, facc[mt][3] += m1[h] * gb;
          }
        }
      }
    }
  }
};
using IbQ8_0 = Ib32<8, false>;
using IbQ4_0 = Ib32<4, false>;
using IbQ5_0 = Ib32<5, false>;
using IbQ4_1 = Ib32<4, true>;
using IbQ5_1 = Ib32<5, true>;

// ------------------------------------------------------------------------------------------------ kernel
// The step's block times the first cx.nt tiles, whose number is a constant in the arithmetic
template <class F, int NT, int MT>
__device__ __forceinline__ void ib_block(const IbCtx& cx, float (&facc)[MT][4]) {
  if constexpr (NT < MT) {
    if (cx.nt > NT) {
      ib_block<F, NT + 1>(cx, facc);
      return;
    }
  }
  F::template block<NT>(cx, facc);
}

// kGrouped: the rows of many matrices' groups; else one matrix
template <class F, int MT, bool kGrouped>
__global__ void __launch_bounds__(32 * (MT > 4 ? kIbMaxWarps / 2 : kIbMaxWarps), 1) ibatch_kernel(const IbParams p) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw);  // [2]: an activation buffer's copies have landed
  const uint32_t smem = smem_u32(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = (p.n + 15) >> 4;
  const bool early = !kGrouped && p.early_w;
  if (threadIdx.x == 0) {
    mbar_init(&full[0], 1);
    mbar_init(&full[1], 1);
    mbar_init_fence();
  }
  __syncthreads();
  pdl_launch_dependents();
  if (!early) pdl_wait();

  // This block's share of the work: whole 16-row tiles of one matrix, or of several groups' (a segment each), equal in cost
  // to every other block's. `base` is the cost before group grp, per tile of every group; lo and hi are in cost * n_tiles.
  int grp = 0, m_begin = 0, m_count = p.fixed_rows, t_begin, t_end;
  int base = 0, cost = 0;
  int64_t lo = 0, hi = 0;
  bool whole = false;  // few groups: every group has blocks of its own, in proportion to its cost, and a block one segment
  if constexpr (!kGrouped) {
    t_begin = (int)((int64_t)n_tiles * blockIdx.x / gridDim.x), t_end = (int)((int64_t)n_tiles * (blockIdx.x + 1) / gridDim.x);
  } else {
    int total = 0, live = 0;
    for (int g = lane; g < p.n_groups; g += 32) {
      const int c = ib_group_cost(p.offsets[g + 1] - p.offsets[g], p.rows_cap);
      total += c, live += c > 0;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) total += __shfl_xor_sync(0xffffffffu, total, off), live += __shfl_xor_sync(0xffffffffu, live, off);
    // from five blocks a group on, rounding to whole blocks costs less than a second segment
    const int n_blocks = (int)gridDim.x;
    whole = n_blocks >= 5 * live;
    lo = (int64_t)total * n_tiles * blockIdx.x / n_blocks, hi = (int64_t)total * n_tiles * (blockIdx.x + 1) / n_blocks;
    for (;; grp += 32) {  // the group that this block, or lo, falls into
      if (grp >= p.n_groups) return;
      int mine = grp + lane < p.n_groups ? ib_group_cost(p.offsets[grp + lane + 1] - p.offsets[grp + lane], p.rows_cap) : 0;
      if (whole && mine > 0) mine = 1 + (int)((int64_t)(n_blocks - live) * mine / total);
      int upto = mine;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, off);
        if (lane >= off) upto += v;
      }
      const unsigned past = __ballot_sync(0xffffffffu, whole ? base + upto > (int)blockIdx.x : (int64_t)(base + upto) * n_tiles > lo);
      if (past) {
        const int l = __ffs((int)past) - 1;
        base += __shfl_sync(0xffffffffu, upto - mine, l);
        grp += l;
        if (whole) {
          const int part = (int)blockIdx.x - base, parts = __shfl_sync(0xffffffffu, mine, l);
          t_begin = (int)((int64_t)n_tiles * part / parts), t_end = (int)((int64_t)n_tiles * (part + 1) / parts);
        }
        break;
      }
      base += __shfl_sync(0xffffffffu, upto, 31);
    }
  }
  // the next segment with tiles in it, from group grp on
  auto segment = [&]() -> bool {
    if constexpr (!kGrouped) {
      return t_begin < t_end;
    } else {
      if (whole) {
        m_begin = p.offsets[grp], m_count = p.offsets[grp + 1] - m_begin;
        return t_begin < t_end;
      }
      for (; grp < p.n_groups && (int64_t)base * n_tiles < hi; ++grp, base += cost) {
        m_begin = p.offsets[grp], m_count = p.offsets[grp + 1] - m_begin;
        cost = ib_group_cost(m_count, p.rows_cap);
        if (cost == 0) continue;
        const int64_t l = lo - (int64_t)base * n_tiles, h = hi - (int64_t)base * n_tiles;
        t_begin = l <= 0 ? 0 : (int)((l + cost - 1) / cost);
        const int64_t e = (h + cost - 1) / cost;
        t_end = e < n_tiles ? (int)e : n_tiles;
        if (t_begin < t_end) return true;
      }
      return false;
    }
  };
  if (!segment()) {
    pdl_wait();
    return;
  }
  const int kpart = warp % p.kp, slot = warp / p.kp;  // warps past kp * tg have no tile but stage activations
  const int b_begin = kpart * p.share_q + (kpart < p.share_rem ? kpart : p.share_rem), b_end = b_begin + p.share_q + (kpart < p.share_rem);
  const bool has_slot = slot < p.tg;

  IbCtx cx;
  cx.lane = lane, cx.gid = lane >> 2, cx.tig = lane & 3;

  // ---- weight stream of this warp: its tiles' blocks, round after round, pass after pass
  const uint32_t stage_bytes = 16u * F::kPitch;
  const uint32_t wst = smem + kIbHeader + (uint32_t)(warp * p.stages) * stage_bytes;
  const int nb = b_end - b_begin;
  int64_t gbase;
  int n_pass, rounds;
  int f_tile, f_b, f_stage = 0, f_left;  // next block to fetch
  constexpr int kPieces = F::kAligned ? F::kBytes256 / 16 : F::kPitch / 16 - 1, kCopies = (16 * kPieces + 31) / 32;
  // This lane's pieces, lane + 32 i. Formats on 16-byte boundaries: their offsets from the tile's first row, at the block to
  // fetch, kept for the tile (worked out for every block, they took a tenth of the kernel's instructions), and where they
  // go: a constant apart where rows are stored without gaps. Others: row | piece << 8.
  constexpr bool kGapless = F::kAligned && F::kPitch == F::kBytes256;
  const uint8_t* f_src;
  uint32_t so[kCopies], rc[kCopies];
#pragma unroll
  for (int i = 0; i < kCopies; ++i) {
    const int q = lane + 32 * i, r = q / kPieces;
    rc[i] = F::kAligned ? (kGapless ? 16 * q : r * F::kPitch + 16 * (q - r * kPieces)) : r | (q - r * kPieces) << 8;
  }
  auto open_tile = [&]() {  // f_tile from block f_b on
    f_src = p.w + gbase + (int64_t)f_tile * 16 * p.row_bytes + (int64_t)f_b * F::kBytes256;
    if constexpr (F::kAligned) {
      const int last = p.n - 1 - f_tile * 16;  // the last tile repeats row n - 1
#pragma unroll
      for (int i = 0; i < kCopies; ++i) {
        const int q = lane + 32 * i, r = q / kPieces;
        so[i] = (uint32_t)(r < last ? r : last) * (uint32_t)p.row_bytes + 16u * (uint32_t)(q - r * kPieces);
      }
    }
  };
  auto start_stream = [&]() {  // for the segment's tiles slot, slot + tg, ...
    gbase = kGrouped ? (int64_t)grp * p.group_bytes : 0;
    n_pass = (m_count + p.rows_cap - 1) / p.rows_cap;
    rounds = (t_end - t_begin + p.tg - 1) / p.tg;
    const int mine = has_slot && t_end - t_begin > slot ? (t_end - t_begin - slot + p.tg - 1) / p.tg : 0;
    f_tile = t_begin + slot, f_b = b_begin, f_left = mine * nb * n_pass;
    open_tile();
  };
  auto fetch = [&]() {  // one block of this warp's tile into the next stage; always one commit group
    if (f_left > 0) {
      --f_left;
      const uint32_t dst = wst + (uint32_t)f_stage * stage_bytes;
      if constexpr (F::kAligned) {
#pragma unroll
        for (int i = 0; i < kCopies; ++i)
          if (32 * i + 32 <= 16 * kPieces || lane + 32 * i < 16 * kPieces) ib_cp16(dst + rc[i], f_src + so[i], 16u);
      } else if (f_tile + 1 < n_tiles) {
#pragma unroll
        for (int i = 0; i < kCopies; ++i) {
          if (32 * i + 32 <= 16 * kPieces || lane + 32 * i < 16 * kPieces) {
            const int r = rc[i] & 255, c = rc[i] >> 8;
            const uint8_t* row = f_src + r * p.row_bytes;
            const int skew = (int)(reinterpret_cast<uintptr_t>(row) & 15);  // the matrix starts on a 16-byte boundary
            if (16 * (kPieces - 1) < F::kBytes256 || 16 * c < skew + F::kBytes256)
              ib_cp16(dst + (uint32_t)(r * F::kPitch + 16 * c), row - skew + 16 * c, 16u);
          }
        }
      } else {  // the matrix may end inside a 16-byte piece: read only what it has
#pragma unroll 1
        for (int q = lane; q < 16 * kPieces; q += 32) {
          const int r = q / kPieces, c = q - r * kPieces;
          const int row = f_tile * 16 + r < p.n ? f_tile * 16 + r : p.n - 1;
          const int64_t b0 = gbase + (int64_t)row * p.row_bytes + (int64_t)f_b * F::kBytes256, at = (b0 & ~(int64_t)15) + 16 * c;
          const int64_t left = p.total_bytes - at;
          if (at < b0 + F::kBytes256) ib_cp16(dst + (uint32_t)(r * F::kPitch + 16 * c), p.w + at, left >= 16 ? 16u : (uint32_t)left);
        }
      }
      if (++f_stage == p.stages) f_stage = 0;
      f_src += F::kBytes256;
      if (++f_b == b_end) {
        f_b = b_begin;
        f_tile += p.tg;
        if (f_tile >= t_end) f_tile = t_begin + slot;  // next pass over the rows
        open_tile();
      }
    }
    ib_commit();
  };

  // ---- activation staging: chunk c of the pass that starts at row a0 into buffer `buf`. Slot s holds the s % bpc-th block of
  // the chunk of share s / bpc: the rows' records, one bulk copy (a lane of warp 0 each). Rows past `ac` keep whatever is
  // there: a row is a column of the MMAs' results, and theirs are not stored.
  constexpr int kRec = ib_rec(F::kAct);
  // Planes hold a single row, so the forms for many tiles have no code for them. The two-tile form needs none either, but its
  // registers came out worse without: Q4_K 4096 x 11008 at 16 rows 19.9 -> 20.3 us.
  auto records = [&]() -> bool { return MT > 2 || p.act.rec; };
  int slot_bytes, bpc, n_chunks;
  auto stage_acts = [&](int a0, int ac, int c, int buf) {
    const uint32_t base = (uint32_t)(p.act_off + buf * p.act_buf);
    const int slots = p.kp * bpc;
    auto slot_block = [&](int s) -> int {  // or -1
      const int sh = s / bpc, b0 = sh * p.share_q + (sh < p.share_rem ? sh : p.share_rem), j = c * bpc + s - sh * bpc;
      return j < p.share_q + (sh < p.share_rem) ? b0 + j : -1;
    };
    if (records()) {
      if (warp == 0) {
        int mine = 0;
        for (int s = lane; s < slots; s += 32) mine += slot_block(s) >= 0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, off);
        if (lane == 0) mbar_arrive_expect_tx(&full[buf], (uint32_t)(mine * ac * kRec));
        __syncwarp();
        for (int s = lane; s < slots; s += 32) {
          const int b = slot_block(s);
          if (b >= 0) bulk_g2s(smem_raw + base + s * slot_bytes, p.act.rec + ((size_t)b * p.act_rows + a0) * kRec, (uint32_t)(ac * kRec), &full[buf]);
        }
      }
    } else {  // one row, as planes: sixteen threads a slot, in this thread's newest cp.async group
      const int piece = threadIdx.x & 15;
      for (int s = threadIdx.x >> 4; s < slots; s += blockDim.x >> 4) {
        const int b = slot_block(s);
        if (b < 0) continue;
        const uint32_t dst = smem + base + (uint32_t)(s * slot_bytes);
        ib_cp16(dst + 16u * piece, p.act.qs + b * 256 + 16 * piece, 16u);
        if constexpr (F::kAct == kIbQ8K) {
          if (F::kSums && piece < 2) ib_sums16(dst + kActRecAux + 16u * piece, p.act.bsums + b * 16 + 8 * piece);
          else if (piece == 2) ib_cp4(dst + kActRecD, p.act.d + b, 4u);
        } else {
          if (piece < 2) ib_cp16(dst + kActRecAux + 16u * piece, p.act.d + b * 8 + 4 * piece, 16u);
          else if (F::kAct == kIbQ8_1 && piece < 4)
            ib_cp16(dst + kActRecAux + 16u * piece, reinterpret_cast<const float*>(p.act.bsums) + b * 8 + 4 * (piece - 2), 16u);
        }
      }
    }
    ib_commit();
  };
  uint32_t phases = 0;  // bit b: parity of buffer b's next fill
  auto acts_landed = [&](int buf) {
    if (records()) {
      if (!mbar_wait_bounded(&full[buf], (phases >> buf) & 1u)) record_dev_error(kErrFullWait);  // carries on: the host sees the code
      phases ^= 1u << buf;
    }
  };

  float* part = reinterpret_cast<float*>(smem_raw + p.part_off);
  int step_stage = 0;
  for (bool first = true;; first = false) {
    start_stream();
    // all but one stage of weights (before the wait for the predecessor where allowed), then the first activations
    for (int i = 0; i < p.stages - 1; ++i) fetch();
    if (first && early) pdl_wait();
    // the plan's chunks are for rows_cap rows: fewer need fewer chunks
    slot_bytes = (kGrouped && n_pass == 1 ? (m_count + 7) & ~7 : p.rows_cap) * kRec;
    bpc = p.bpc, n_chunks = p.n_chunks;
    if (kGrouped && n_chunks > 1) {
      const int share = p.share_q + (p.share_rem > 0);
      if (p.kp * share * slot_bytes <= 2 * p.act_buf) bpc = share, n_chunks = 1;
      else bpc = p.act_buf / (p.kp * slot_bytes), n_chunks = (share + bpc - 1) / bpc;
    }
    for (int pass = 0; pass < n_pass; ++pass) {
      const int a0 = m_begin + pass * p.rows_cap;
      const int ac = m_count - pass * p.rows_cap < p.rows_cap ? m_count - pass * p.rows_cap : p.rows_cap;
      cx.nt = (ac + 7) >> 3;
      if (pass > 0 || !first) __syncthreads();  // the previous pass's activations are done with
      stage_acts(a0, ac, 0, 0);
      if (!records()) {
        ib_wait(0);
        __syncthreads();
      }
      acts_landed(0);
      int buf = 0;
      for (int round = 0; round < rounds; ++round) {
        float facc[MT][4];
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int i = 0; i < 4; ++i) facc[mt][i] = 0.f;
        const int tile = t_begin + round * p.tg + slot;
        const bool live = has_slot && tile < t_end;
        for (int c = 0; c < n_chunks; ++c) {
          const bool last_chunk = c + 1 == n_chunks, more = n_chunks > 1 && !(last_chunk && round + 1 == rounds);
          // the next chunk, into the buffer that the barrier at the end of the previous chunk freed
          if (more) stage_acts(a0, ac, last_chunk ? 0 : c + 1, buf ^ 1);
          const uint32_t abase = smem + (uint32_t)(p.act_off + buf * p.act_buf);
          const int j_end = nb - c * bpc < bpc ? nb - c * bpc : bpc;
          for (int j = 0; j < j_end && live; ++j) {
            fetch();
            // groups newer than this step's weights: the stages - 1 fetches after it (a staged chunk among them only helps)
            ib_wait(p.stages - 1);
            __syncwarp();
            const uint32_t st = wst + (uint32_t)step_stage * stage_bytes;
            if (++step_stage == p.stages) step_stage = 0;
            uint32_t k0 = 0, k1 = 0;
            if constexpr (!F::kAligned) {  // rows past n repeat row n - 1
              const int b = b_begin + c * bpc + j;
              const int ra = tile * 16 + cx.gid < p.n ? tile * 16 + cx.gid : p.n - 1;
              const int rb = tile * 16 + cx.gid + 8 < p.n ? tile * 16 + cx.gid + 8 : p.n - 1;
              const uint32_t o = (uint32_t)gbase + (uint32_t)b * F::kBytes256;
              k0 = (o + (uint32_t)ra * (uint32_t)p.row_bytes) & 15u, k1 = (o + (uint32_t)rb * (uint32_t)p.row_bytes) & 15u;
            }
            cx.r0 = st + (uint32_t)(cx.gid * F::kPitch) + k0;
            cx.r1 = st + (uint32_t)((cx.gid + 8) * F::kPitch) + k1;
            cx.lm = st + (uint32_t)(((lane & 7) + (lane & 8)) * F::kPitch) + 16u * (lane >> 4);
            cx.act = abase + (uint32_t)((kpart * bpc + j) * slot_bytes);
            ib_block<F, kGrouped ? 1 : MT>(cx, facc);
            __syncwarp();  // every lane has read the stage before any lane refills it
          }
          if (more) {
            if (!records()) ib_wait(0);
            __syncthreads();
            buf ^= 1;
            acts_landed(buf);
          }
        }
        // the shares' sums, two 8-row tiles at a time; a single share stores straight from its registers
        const int row0 = tile * 16;
        if (p.kp == 1) {
          if (live) {
#pragma unroll
            for (int mt = 0; mt < MT; ++mt)
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int m = 8 * mt + 2 * cx.tig + (i & 1), col = cx.gid + 8 * (i >> 1);
                if (m < ac && row0 + col < p.n) {
                  const int orow = kGrouped && p.out_rows ? p.out_rows[a0 + m] : a0 + m;
                  p.y[(size_t)orow * p.n + row0 + col] = facc[mt][i];
                }
              }
          }
        } else {
#pragma unroll
          for (int m2 = 0; m2 < MT; m2 += 2) {
            if (m2 < cx.nt) {
              constexpr int kW = (MT > 1 ? 2 : 1) * 128;  // floats per warp
              if (live) {
#pragma unroll
                for (int q = 0; q < (MT > 1 ? 2 : 1); ++q)
#pragma unroll
                  for (int i = 0; i < 4; ++i) if (m2 + q < MT) part[warp * kW + (q * 4 + i) * 32 + lane] = facc[m2 + q][i];
              }
              __syncthreads();
              const int tiles_here = t_end - (t_begin + round * p.tg) < p.tg ? t_end - (t_begin + round * p.tg) : p.tg;
              for (int i = threadIdx.x; i < tiles_here * kW; i += blockDim.x) {
                const int ts = i / kW, o = i - ts * kW, ml = o >> 4, col = o & 15;
                const int m = 8 * m2 + ml, gr = (t_begin + round * p.tg + ts) * 16 + col;
                if (m < ac && gr < p.n) {
                  // fragment position of (activation row ml, weight row col)
                  const int src = (((ml >> 3) * 4 + ((ml & 1) | ((col >> 3) << 1))) << 5) + ((col & 7) << 2) + ((ml & 7) >> 1);
                  const float* q = part + (size_t)(ts * p.kp) * kW + src;
                  float sum = q[0];
                  for (int s = 1; s < p.kp; ++s) sum += q[s * kW];
                  const int orow = kGrouped && p.out_rows ? p.out_rows[a0 + m] : a0 + m;
                  p.y[(size_t)orow * p.n + gr] = sum;
                }
              }
              __syncthreads();
            }
          }
        }
      }
    }
    if (!kGrouped || whole) break;
    ++grp, base += cost;
    if (!segment()) break;
  }
}

#undef FQ_IB_TILES
}  // namespace fq
