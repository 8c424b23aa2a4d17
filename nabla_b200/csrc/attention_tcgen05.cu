// Flash attention for sm_100a on tcgen05 tensor cores with TMEM accumulators.
//
//   O = softmax(Q K^T * scale [+ mask] [+ causal mask]) V     per (batch, head), never materialising
//                                                             the (seq_q, seq_k) score matrix
//
// Replaces the reference's composed attention (matmul, mul, tril, where, softmax, matmul:
// nabla/nn/functional/layers.py:106-153), whose memory is O(seq^2).
//
// Three kernels, all with the same warp roles (384 threads, one CTA per SM):
//   warp 0      TMA producer (4-D tensor maps over strided (B, H, S, D) views, so q/k/v sliced out
//               of a packed projection are read in place)
//   warp 1      MMA issuer (one elected thread)
//   warp 2      TMEM allocator
//   warps 4-11  two math warpgroups of 128 threads; thread r of a group owns TMEM lane r
//
// The probabilities never touch shared memory: the math threads write P (bf16, two values per
// 32-bit TMEM column) over the score columns they have just read, and the second MMA takes its A
// operand from TMEM. Shared memory then only feeds Q / K / V / dO, which halves the operand
// traffic of the PV-type products.
//
// forward (attn_fwd_kernel): one CTA owns TWO query tiles (2 x 128 rows; one where the grid has an
//   SM for every tile) that share the K / V stream. Group A works on the softmax of tile A while the tensor core runs tile B's products
//   and vice versa (S_A, S_B, O_A, O_B = 512 TMEM columns at head_dim 128).
// backward, dK / dV (attn_bwd_dkdv_kernel): one CTA owns 128 keys and walks over the query
//   tiles: S^T = K Q^T, dP^T = V dO^T, P^T and dS^T written back into TMEM as A operands of
//   dV += P^T dO and dK += dS^T Q. The two groups split the 128 query columns of a tile.
// backward, dQ (attn_bwd_dq_kernel): one CTA owns 128 queries and walks over the key tiles:
//   S = Q K^T (double buffered), dP = dO V^T, dS into TMEM, dQ += dS K accumulated in TMEM and
//   stored once as bf16: no atomics, no fp32 scratch, deterministic.
// A small kernel before the backward computes delta = rowsum(dO * O) and log2-domain row
// statistics padded to whole tiles.
#include <cooperative_groups.h>

#include "sm100_ptx.cuh"
#include "launch.cuh"
#include "nb_debug.cuh"

namespace nba {
using namespace nb;

// named_bar_sync whose threads also learn whether `any` holds in one of them.
__device__ __forceinline__ bool named_bar_or(int id, int nthreads, bool any) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %3, 0;\n\t"
      "barrier.cta.red.or.pred p, %1, %2, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(nthreads), "r"((uint32_t)any)
      : "memory");
  return r != 0;
}

constexpr int BT = 128;          // tile edge, queries and keys
constexpr int NTHREADS = 384;
constexpr float LOG2E = 1.4426950408889634f;

// Tile load at (column c0, row c1, head c2, batch c3) of a [batch][heads][rows][head_dim] bf16 tensor.
// Debug build: the origin lies inside the tensor and c0 starts on a 16-byte boundary, else the copy is
// not issued (the consumer's bounded wait then ends the kernel with an error status).
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1, int c2,
                                            int c3, int rows, int heads, int batch) {
  if (!(NB_ALIGNED(NB_SITE_ATTN_TMA_COORD, c0 * 2, 16) && NB_IN_BOUNDS(NB_SITE_ATTN_TMA_COORD, c1, rows) &&
        NB_IN_BOUNDS(NB_SITE_ATTN_TMA_COORD, c2, heads) && NB_IN_BOUNDS(NB_SITE_ATTN_TMA_COORD, c3, batch)))
    return;
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6}], [%2];"
      :
      : "r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2),
        "r"(c3)
      : "memory");
}
// Untiled bulk copy global -> shared; both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(smem_dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
// tcgen05.wait::ld that names the 32 loaded registers as in/out operands: everything that reads
// them afterwards depends on the wait, so the compiler cannot schedule a use above it. This lets a
// loop issue the load of the next chunk before it works on the current one.
__device__ __forceinline__ void tmem_ld_wait32(uint32_t (&v)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                 "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                 "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]),
                 "+r"(v[24]), "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]), "+r"(v[30]), "+r"(v[31])
               :
               : "memory");
}
// Register split between the four service warps (loads, MMA issue) and the eight math warps. The shares add
// up to 80 * 128 + 208 * 256 = 63488 of the 168 * 384 = 64512 registers that a block is launched with, so
// the increase never waits.
__device__ __forceinline__ void service_registers() { asm volatile("setmaxnreg.dec.sync.aligned.u32 80;"); }
__device__ __forceinline__ void math_registers() { asm volatile("setmaxnreg.inc.sync.aligned.u32 208;"); }
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float2 f2(uint32_t a, uint32_t b) { return make_float2(__uint_as_float(a), __uint_as_float(b)); }

// 32 values of a row times `mul` as bf16. vec32: the address is 32-byte aligned, and a lane writes whole sectors (in
// 16-byte pieces of 32 different rows the end of a dK / dV block took 5200 clocks, 3000 this way).
__device__ __forceinline__ void store_row32(__nv_bfloat16* p, const uint32_t (&v)[32], float mul, int vec32) {
  uint32_t w[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) w[e] = pack_bf16(__uint_as_float(v[2 * e]) * mul, __uint_as_float(v[2 * e + 1]) * mul);
  if (vec32) {
    st_global_v8(p, w);
    st_global_v8(p + 16, w + 8);
  } else {
#pragma unroll
    for (int u = 0; u < 4; ++u) reinterpret_cast<uint4*>(p)[u] = make_uint4(w[4 * u], w[4 * u + 1], w[4 * u + 2], w[4 * u + 3]);
  }
}

// D[128 x 128] = A[128 x HD] B[128 x HD]^T : both operands K-major tiles of HD / 64 swizzled chunks.
template <int HD>
__device__ __forceinline__ void mma_scores(uint32_t d_tmem, uint32_t a0, uint32_t b0) {
  constexpr uint32_t idesc = make_idesc_bf16(BT, BT, 0, 0);
#pragma unroll
  for (int k = 0; k < HD / 16; ++k) {
    const uint64_t da = make_smem_desc_sw128(a0 + (k >> 2) * (BT * 128) + (k & 3) * 32, 16, 1024);
    const uint64_t db = make_smem_desc_sw128(b0 + (k >> 2) * (BT * 128) + (k & 3) * 32, 16, 1024);
    umma_f16_ss(d_tmem, da, db, idesc, k != 0);
  }
}
// D[128 x HD] (+)= A[128 x 128] B[128 x HD] : A (bf16 pairs) in TMEM, B in shared memory with the
// reduction index as rows and HD contiguous. `split`: the A columns of k-steps 4-7 start 64 TMEM
// columns after those of k-steps 0-3 (each math group writes inside the columns it has read).
template <int HD>
__device__ __forceinline__ void mma_accum(uint32_t d_tmem, uint32_t a_tmem, bool split, uint32_t b0, bool accumulate) {
  constexpr uint32_t idesc = make_idesc_bf16(BT, HD, 0, 1);
#pragma unroll
  for (int k = 0; k < BT / 16; ++k) {
    const uint64_t db = make_smem_desc_sw128(b0 + k * (16 * 128), BT * 128, 1024);
    const uint32_t a = a_tmem + (split ? 64 * (k >> 2) + 8 * (k & 3) : 8 * k);
    umma_f16_ts(d_tmem, a, db, idesc, (accumulate || k != 0) ? 1u : 0u);
  }
}

// Optional additive mask (fp32, natural-log domain), element (b, h, q, key) at
// mask[b * sb + h * sh + q * sq + key]; strides of 0 broadcast.
struct MaskArg {
  const float* ptr;
  long long sb, sh, sq;
};
// The kinds a kernel is compiled for. KEYS: one mask row for all queries (padding masks). ROWS: a row per query, read
// by the threads that own the rows. Both in one kernel, told apart at run time, keep a row mask's loads from being in
// flight together (backward of 64 heads x 2048 x 128 with a row mask: 2.6 -> 4.0 ms).
enum UserMask { MASK_NONE, MASK_KEYS, MASK_ROWS };

// Order of the CTAs of a launch. Causal: the tile index is the slow one, so that the long tiles start first and
// the short ones fill the end of the grid (a head's tiles one after the other: at 64 heads x 8 forward tiles the
// busiest SM had 1.3 times the mean); the (batch, head) pairs are taken in chunks whose shared operands,
// `chunk` at a time, stay in L2. Otherwise all tiles are alike, and chunk = 1 keeps a head's tiles, which read
// the same operands, together. rank 0 is the longest tile. Causal forward, head_dim 128: 113 -> 97 us at 64 heads
// of 2048, 311 -> 254 us at 16 heads of 8192; chunks of 64 MB, or this order without causality (152 -> 158 us),
// are slower.
__device__ __forceinline__ void tile_order(int bid, int nbh, int chunk, int tiles, int& bh, int& rank) {
  const int c = bid / (chunk * tiles), r = bid - c * (chunk * tiles), n = min(chunk, nbh - c * chunk);
  rank = r / n;
  bh = c * chunk + (r - rank * n);
}

// ====================================================================== forward
struct FwdArgs {
  int B, H, Sq, Skv;
  float scale_log2;   // softmax scale * log2(e)
  int causal;
  __nv_bfloat16* O;
  long long o_sb, o_sh, o_ss;   // element strides of O for batch, head, row
  float* lse;                   // [B][H][Sq]
  MaskArg mask;
  int* status;
  int vec32;                    // rows of O start on 32-byte boundaries
  int q_tiles;                  // query tiles of a CTA: 2, or 1 where those of 2 would leave SMs without a CTA
  int bh_chunk;                 // see tile_order
  int nsplit;                   // the keys are cut into this many ranges, one CTA each (1: no split)
  float* part_o;                // nsplit > 1: [nsplit][B][H][Sq][HD] output over each range, fp32
  float* part_lse;              //             [nsplit][B][H][Sq] natural-log sum of exponentials of each range
};

template <int HD, bool KEYS>
struct FwdSmem {
  static constexpr int TILE_BYTES = BT * HD * 2;
  static constexpr int OFF_Q = 0;                          // 2 query tiles
  static constexpr int OFF_K = OFF_Q + 2 * TILE_BYTES;     // 2 stages
  static constexpr int OFF_V = OFF_K + 2 * TILE_BYTES;     // 2 stages
  static constexpr int OFF_MASK = OFF_V + 2 * TILE_BYTES;  // key mask: [2 math groups][2][128] values of a key tile. Not for
  static constexpr int OFF_BAR = OFF_MASK + (KEYS ? 4 * BT * 4 : 0);   // the others: at 196 KB (head_dim 128) the 2 KB cost
                                                           // half of the L1 that holds a row mask's lines
  static constexpr int RAW = OFF_BAR + 20 * 8 + 16 + 1024;
  static constexpr int TOTAL = RAW < 120 * 1024 ? 120 * 1024 : RAW;   // one CTA per SM (it takes all of TMEM)
};
static_assert(FwdSmem<128, false>::TOTAL + 1024 <= 196 * 1024, "with a row mask or none 60 KB of L1 are left");

// MASK_KEYS: a user mask with one row for all queries (padding). Its kernel reads a row's scores once and keeps them in
// registers for the mask, the maximum and the exponentials; without a mask, reading them twice (maximum,
// exponentials), each load under the work on the one before, measured 5 % faster at head_dim 128. 96 heads x 777 x
// 64 with a key mask: forward 134 -> 84 us, backward 318 -> 199 us.
// MASK_ROWS: a mask row per query, 128 loads per thread and key tile. They are added in the pass that hides keys, the
// kernel otherwise that without a mask: with the scores in registers fewer of those loads are in flight
// (96 x 777 x 64: 243 us that way, 212 this way; 16 heads x 300 x 128: 74 and 47, the L1 space included).
// SPARE (head_dim 64 but for MASK_ROWS): the two outputs take 128 columns of tensor memory, which leaves 128 of the 512 for
// the probabilities. A tile's scores are read into registers at once and the next key tile's QK^T overwrites them while
// the exponentials run, so the softmax does not wait for a product.
template <int HD, UserMask MASK>
__global__ void __launch_bounds__(NTHREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const FwdArgs args) {
  using L = FwdSmem<HD, MASK == MASK_KEYS>;
  constexpr bool SPARE = HD == 64 && MASK != MASK_ROWS;
  constexpr bool REGS = SPARE || MASK == MASK_KEYS;      // a row's 128 scores stay in registers
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + L::OFF_Q;
  uint8_t* sK = smem + L::OFF_K;
  uint8_t* sV = smem + L::OFF_V;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* q_full = bars + 0;     // [2] per query tile
  uint64_t* k_full = bars + 2;     // [2]
  uint64_t* k_empty = bars + 4;    // [2]
  uint64_t* v_full = bars + 6;     // [2]
  uint64_t* v_empty = bars + 8;    // [2]
  uint64_t* s_full = bars + 10;    // [2] per query tile: scores of the next key tile are in TMEM
  uint64_t* p_full = bars + 12;    // [2] per query tile: probabilities are in TMEM (128 arrivals)
  uint64_t* o_done = bars + 14;    // [2] per query tile: last PV product has retired (SPARE: every PV product)
  uint64_t* s_read = bars + 16;    // [2] per query tile, SPARE: scores are in registers (128 arrivals)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // an earlier bounded wait on this device already failed, as far as is known before the grid ahead has ended: leave (uniformly)
  if (__syncthreads_or(threadIdx.x == 0 ? *reinterpret_cast<volatile int*>(args.status) : 0)) return follow_grid();
  const int nqt = (args.Sq + args.q_tiles * BT - 1) / (args.q_tiles * BT);
  int bh_, rank;
  tile_order(blockIdx.x, args.H * args.B * args.nsplit, args.bh_chunk, nqt, bh_, rank);
  const int qt = nqt - 1 - rank;          // the late tiles of a causal problem see the most keys
  const int sp = bh_ % args.nsplit;
  bh_ /= args.nsplit;
  const int h = bh_ % args.H;
  const int b = bh_ / args.H;
  const int q0 = qt * args.q_tiles * BT;
  const int off = args.Skv - args.Sq;     // causal: row i sees keys <= i + off
  int n_t[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int q0t = q0 + t * BT;
    int n = (args.Skv + BT - 1) / BT;
    if (args.causal) {
      const int last_key = min(args.Skv - 1, q0t + BT - 1 + off);
      n = last_key < 0 ? 0 : last_key / BT + 1;
    }
    n_t[t] = t < args.q_tiles && q0t < args.Sq ? n : 0;
  }
  // this CTA's range of key tiles: [kt0, kt0 + n_t[t]) of query tile t
  const int per = (max(n_t[0], n_t[1]) + args.nsplit - 1) / args.nsplit;
  const int kt0 = sp * per;
  n_t[0] = min(max(n_t[0] - kt0, 0), per);
  n_t[1] = min(max(n_t[1] - kt0, 0), per);
  const int n_max = max(n_t[0], n_t[1]);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], SPARE ? 2 : 1);       // SPARE: one arrival per query tile
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], SPARE ? 2 : 1);
      mbar_init(&s_full[i], 1);
      mbar_init(&p_full[i], 128);
      mbar_init(&o_done[i], 1);
      mbar_init(&s_read[i], 128);
    }
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  follow_grid();
  // tile t: scores (and P over their first 64 columns) at t * 128, output accumulator at 256 + t * HD; SPARE: P at 384 + t * 64

  if (warp < 4) {
  if (REGS) service_registers();
  if (warp == 0) {
    if (n_max > 0 && elect_one()) {
      for (int t = 0; t < 2; ++t) {
        if (n_t[t] == 0) continue;
        mbar_arrive_expect_tx(&q_full[t], L::TILE_BYTES);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          tma_load_4d(sQ + t * L::TILE_BYTES + c * (BT * 128), &tmQ, &q_full[t], c * 64, q0 + t * BT, h, b, args.Sq, args.H, args.B);
      }
      for (int j = 0; j < n_max; ++j) {
        const int st = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        if (!mbar_wait(&k_empty[st], ph)) { atomicExch(args.status, NB_ERR_TIMEOUT_PRODUCER); break; }
        mbar_arrive_expect_tx(&k_full[st], L::TILE_BYTES);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          tma_load_4d(sK + st * L::TILE_BYTES + c * (BT * 128), &tmK, &k_full[st], c * 64, (kt0 + j) * BT, h, b, args.Skv, args.H, args.B);
        if (!mbar_wait(&v_empty[st], ph)) { atomicExch(args.status, NB_ERR_TIMEOUT_PRODUCER); break; }
        mbar_arrive_expect_tx(&v_full[st], L::TILE_BYTES);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          tma_load_4d(sV + st * L::TILE_BYTES + c * (BT * 128), &tmV, &v_full[st], c * 64, (kt0 + j) * BT, h, b, args.Skv, args.H, args.B);
      }
    }
  } else if (SPARE) {
    // warps 1 and 3 issue for one query tile each, so that neither group's softmax waits for the other's
    const int t = warp >> 1;
    if (warp != 2 && n_max > 0 && elect_one()) {
      bool ok = n_t[t] == 0 || mbar_wait(&q_full[t], 0);
      for (int j = 0; j <= n_max && ok; ++j) {
        if (j < n_max) {                   // scores of key tile j, as soon as those before are in registers
          const int st = j & 1;
          ok = mbar_wait(&k_full[st], (j >> 1) & 1);
          if (ok && j < n_t[t]) {
            ok = j == 0 || mbar_wait(&s_read[t], (j - 1) & 1);
            if (!ok) break;
            tc_fence_after();
            mma_scores<HD>(tmem_base + t * BT, smem_u32(sQ + t * L::TILE_BYTES), smem_u32(sK + st * L::TILE_BYTES));
            umma_commit(&s_full[t]);
            umma_commit(&k_empty[st]);
          } else if (ok) {
            mbar_arrive(&k_empty[st]);     // this query tile sees no key of the tile
          }
        }
        if (ok && j > 0) {                 // PV of key tile j - 1
          const int i = j - 1, st = i & 1;
          ok = mbar_wait(&v_full[st], (i >> 1) & 1);
          if (ok && i < n_t[t]) {
            ok = mbar_wait(&p_full[t], i & 1);
            if (!ok) break;
            tc_fence_after();
            mma_accum<HD>(tmem_base + 256 + t * HD, tmem_base + 384 + t * 64, false, smem_u32(sV + st * L::TILE_BYTES), i != 0);
            umma_commit(&o_done[t]);
            umma_commit(&v_empty[st]);
          } else if (ok) {
            mbar_arrive(&v_empty[st]);
          }
        }
      }
      if (!ok) atomicExch(args.status, NB_ERR_TIMEOUT_MMA);
    }
  } else if (warp == 1) {
    if (n_max > 0 && elect_one()) {
      bool ok = true;
      auto qk = [&](int t, int j) {
        mma_scores<HD>(tmem_base + t * BT, smem_u32(sQ + t * L::TILE_BYTES), smem_u32(sK + (j & 1) * L::TILE_BYTES));
        umma_commit(&s_full[t]);
      };
      auto pv = [&](int t, int j) {
        mma_accum<HD>(tmem_base + 256 + t * HD, tmem_base + t * BT, false, smem_u32(sV + (j & 1) * L::TILE_BYTES), j != 0);
        if (j == n_t[t] - 1) umma_commit(&o_done[t]);
      };
      for (int t = 0; t < 2 && ok; ++t)
        if (n_t[t] > 0) ok = mbar_wait(&q_full[t], 0);
      ok = ok && mbar_wait(&k_full[0], 0);
      if (ok) {
        tc_fence_after();
        if (n_t[0] > 0) qk(0, 0);
        if (n_t[1] > 0) qk(1, 0);
        umma_commit(&k_empty[0]);
      }
      for (int j = 0; j < n_max && ok; ++j) {
        const bool more = j + 1 < n_max;
        if (!mbar_wait(&v_full[j & 1], (j >> 1) & 1)) { ok = false; break; }
        if (more && !mbar_wait(&k_full[(j + 1) & 1], ((j + 1) >> 1) & 1)) { ok = false; break; }
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j < n_t[t]) {
            if (!mbar_wait(&p_full[t], j & 1)) { ok = false; break; }
            tc_fence_after();
            pv(t, j);
          }
          if (t == 1) umma_commit(&v_empty[j & 1]);
          if (j + 1 < n_t[t]) qk(t, j + 1);
        }
        if (!ok) break;
        if (more) umma_commit(&k_empty[(j + 1) & 1]);
      }
      if (!ok) atomicExch(args.status, NB_ERR_TIMEOUT_MMA);
    }
  }
  } else {
    if (REGS) math_registers();
    const int t = (warp - 4) >> 2;          // query tile of this math group
    const int wq = warp & 3;
    const int r = wq * 32 + lane;
    const int q_idx = q0 + t * BT + r;
    const int n = n_t[t];
    const uint32_t lane_addr = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t t_s = tmem_base + t * BT + lane_addr;
    const uint32_t t_o = tmem_base + 256 + t * HD + lane_addr;
    const uint32_t t_p = SPARE ? tmem_base + 384 + t * 64 + lane_addr : t_s;
    // user mask: one row for all queries (padding masks) goes through shared memory, 128 coalesced values
    // per key tile; a row per query is read by its own thread
    const float* mrow = nullptr;
    constexpr bool mshared = MASK == MASK_KEYS;
    if (mshared || (MASK == MASK_ROWS && q_idx < args.Sq))
      mrow = args.mask.ptr + b * args.mask.sb + h * args.mask.sh + (mshared ? 0ll : (long long)q_idx * args.mask.sq);
    float* smask = reinterpret_cast<float*>(smem + L::OFF_MASK) + t * 2 * BT;
    const float mask_mul = LOG2E / args.scale_log2;
    float mnext = 0.f;
    if (mshared && n > 0 && kt0 * BT + r < args.Skv) mnext = mrow[kt0 * BT + r];
    float m_used = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      const int kv0 = (kt0 + j) * BT;
      bool masked = false;                 // a tile whose 128 mask values are all zero (most of a padded batch) adds nothing
      if (mshared) {
        smask[(j & 1) * BT + r] = mnext;
        masked = named_bar_or(2 + t, 128, mnext != 0.f);
        mnext = j + 1 < n && kv0 + BT + r < args.Skv ? mrow[kv0 + BT + r] : 0.f;
      }
      if (ok && !mbar_wait(&s_full[t], j & 1)) {
        atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (mshared) continue;             // keep the group's barrier participation uniform
        break;
      }
      tc_fence_after();
      const bool edge = kv0 + BT > args.Skv || (args.causal && kv0 + BT - 1 > q0 + t * BT + off);
      float mxa[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      uint32_t v4[REGS ? 4 : 2][32];     // the row's 128 scores, or two chunks of 32, one of them in flight
      if constexpr (REGS) {
        auto& v = v4;
        if constexpr (SPARE) {
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_32x32(t_s + c * 32, v[c]);
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld_wait32(v[c]);
          tc_fence_before();
          mbar_arrive(&s_read[t]);
        } else {
          tmem_ld_32x32(t_s, v[0]);        // the load of the next 32 columns runs under the work on the current ones
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if constexpr (!SPARE) {
            tmem_ld_wait32(v[c]);
            if (c < 3) tmem_ld_32x32(t_s + (c + 1) * 32, v[c + 1]);
          }
          if (mshared && masked) {
            const float4* m4 = reinterpret_cast<const float4*>(smask + (j & 1) * BT + c * 32);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 mv = m4[i];
              uint32_t* w = &v[c][i * 4];
              w[0] = __float_as_uint(fmaf(mv.x, mask_mul, __uint_as_float(w[0])));
              w[1] = __float_as_uint(fmaf(mv.y, mask_mul, __uint_as_float(w[1])));
              w[2] = __float_as_uint(fmaf(mv.z, mask_mul, __uint_as_float(w[2])));
              w[3] = __float_as_uint(fmaf(mv.w, mask_mul, __uint_as_float(w[3])));
            }
          }
          if (edge) {
            // diagonal or tail tile: -inf where a key is not visible
            const int last = args.causal ? min(args.Skv - 1, q_idx + off) : args.Skv - 1;      // this row's last visible key
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i > last - kv0) v[c][i] = __float_as_uint(-INFINITY);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i) mxa[i & 3] = max3(mxa[i & 3], __uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1]));
        }
      } else {
        uint32_t (&va)[32] = v4[0], (&vb)[32] = v4[1];
        if (edge || MASK == MASK_ROWS) {
          // diagonal or tail tile, or a mask: rewrite the scores in place, -inf where a key is
          // not visible, so that the two passes below carry no mask logic. Its bounds live in here alone: two registers
          // more across the whole loop cost it 1.5 % (4 queries x 16384 keys x 128 heads: 234.5 us, 238.6 with them)
          const int last = args.causal ? min(args.Skv - 1, q_idx + off) : args.Skv - 1;      // this row's last visible key
#pragma unroll 1
          for (int c = 0; c < BT / 32; ++c) {
            uint32_t v[32];
            tmem_ld_32x32(t_s + c * 32, v);
            tmem_ld_wait32(v);
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const int kc = kv0 + c * 32 + i;
              float x = __uint_as_float(v[i]);
              if (MASK == MASK_ROWS && mrow != nullptr && kc < args.Skv) x = fmaf(mrow[kc], mask_mul, x);
              v[i] = __float_as_uint(kc <= last ? x : -INFINITY);
            }
            tmem_st_32x32(t_s + c * 32, v);
          }
          tmem_st_wait();
        }
        // pass 1: row maximum. The load of the next 32 columns is in flight while the current ones
        // are reduced (four independent chains of three-input max).
        tmem_ld_32x32(t_s, va);
#pragma unroll
        for (int c = 0; c < BT / 32; ++c) {
          uint32_t (&v)[32] = (c & 1) ? vb : va;
          uint32_t (&nx)[32] = (c & 1) ? va : vb;
          tmem_ld_wait32(v);
          tmem_ld_32x32(t_s + ((c + 1) & 3) * 32, nx);       // after the last chunk: chunk 0 again, for pass 2
#pragma unroll
          for (int i = 0; i < 16; ++i) mxa[i & 3] = max3(mxa[i & 3], __uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
        }
      }
      const float mx = fmaxf(fmaxf(mxa[0], mxa[1]), fmaxf(mxa[2], mxa[3])) * args.scale_log2;
      // lazy rescale: keep the old reference maximum unless the new one exceeds it by 2^8
      float alpha = 1.f;
      bool resc = false;
      if (m_used == -INFINITY) {
        m_used = mx;                       // may stay -inf: every key so far is masked for this row
      } else if (mx > m_used + 8.f) {
        alpha = ex2(m_used - mx);
        m_used = mx;
        resc = true;
      }
      const float m_sub = m_used == -INFINITY ? 0.f : m_used;
      if (SPARE && j > 0) {
        // the previous PV product has read P and written O
        if (!mbar_wait(&o_done[t], (j - 1) & 1)) {
          atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
          ok = false;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (mshared) continue;
          break;
        }
        tc_fence_after();
      }
      if (__any_sync(0xffffffffu, resc)) {
        // O is not being written now (without SPARE s_full of this tile also tracks the previous PV product)
#pragma unroll 1
        for (int c = 0; c < HD / 32; ++c) {
          uint32_t o[32];
          tmem_ld_32x32(t_o + c * 32, o);
          tmem_ld_wait32(o);
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32(t_o + c * 32, o);
        }
      }
      // pass 2: probabilities (bf16 pairs) written over the first 64 score columns; packed fp32x2
      // arithmetic: per pair one FFMA2, two EX2, one FADD2, one pack
      const float2 sc2 = make_float2(args.scale_log2, args.scale_log2), nm2 = make_float2(-m_sub, -m_sub);
      float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
      for (int c = 0; c < BT / 32; ++c) {
        uint32_t (&v)[32] = v4[REGS ? c : c & 1];
        if constexpr (!REGS) {
          tmem_ld_wait32(v);
          if (c + 1 < BT / 32) tmem_ld_32x32(t_s + (c + 1) * 32, v4[(c + 1) & 1]);
        }
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float2 x = __ffma2_rn(f2(v[2 * i], v[2 * i + 1]), sc2, nm2);
          const float2 pr = make_float2(ex2(x.x), ex2(x.y));
          acc[i & 1] = __fadd2_rn(acc[i & 1], pr);
          pk[i] = pack_bf16(pr.x, pr.y);
        }
        tmem_st_32x16(t_p + c * 16, pk);
      }
      const float sum = (acc[0].x + acc[0].y) + (acc[1].x + acc[1].y);
      l = l * alpha + sum;
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full[t]);
    }
    if (ok && n > 0) {
      if (!mbar_wait(&o_done[t], SPARE ? (n - 1) & 1 : 0)) {
        atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok && t < args.q_tiles && q0 + t * BT < args.Sq) {
      tc_fence_after();
      const bool have = n > 0 && l > 0.f;
      const float inv = have ? 1.f / l : 0.f;
      __nv_bfloat16* orow = args.O + (long long)b * args.o_sb + (long long)h * args.o_sh + (long long)q_idx * args.o_ss;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t v[32];
        if (n > 0) {
          tmem_ld_32x32(t_o + c * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0;
        }
        if (q_idx < args.Sq && args.nsplit > 1) {
          float4* prow = reinterpret_cast<float4*>(args.part_o + ((((long long)sp * args.B + b) * args.H + h) * args.Sq + q_idx) * HD + c * 32);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            prow[u] = make_float4(__uint_as_float(v[4 * u]) * inv, __uint_as_float(v[4 * u + 1]) * inv,
                                  __uint_as_float(v[4 * u + 2]) * inv, __uint_as_float(v[4 * u + 3]) * inv);
        } else if (q_idx < args.Sq) {
          store_row32(orow + c * 32, v, inv, args.vec32);
        }
      }
      if (q_idx < args.Sq) {
        const long long row = ((long long)b * args.H + h) * args.Sq + q_idx;
        float* dst = args.nsplit > 1 ? args.part_lse + (long long)sp * args.B * args.H * args.Sq + row : args.lse + row;
        *dst = have ? (m_used + log2f(l)) * 0.6931471805599453f : -INFINITY;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// O = sum_s w_s O_s with w_s = exp(lse_s - lse): joins the key ranges of a split forward pass. One warp per row; a range
// in which the row sees no key has lse = -inf and weight 0.
template <int HD>
__global__ void __launch_bounds__(128) attn_fwd_combine_kernel(const FwdArgs args) {
  follow_grid();
  constexpr int E = HD / 32;
  const long long rows = (long long)args.B * args.H * args.Sq;
  const long long row = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= rows) return;
  float mx = -INFINITY;
  bool nan = false;                                  // a NaN range makes the row NaN (fmaxf would drop it)
  for (int s = lane; s < args.nsplit; s += 32) {
    const float v = args.part_lse[s * rows + row];
    mx = fmaxf(mx, v);
    nan |= v != v;
  }
  if (__any_sync(0xffffffffu, nan)) mx = NAN;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float v = __shfl_xor_sync(0xffffffffu, mx, o);
    mx = mx != mx ? mx : fmaxf(mx, v);
  }
  float acc[E], sum = 0.f;
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
  if (mx != -INFINITY) {
    for (int s = 0; s < args.nsplit; ++s) {
      const float w = ex2((args.part_lse[s * rows + row] - mx) * LOG2E);
      const float* p = args.part_o + (s * rows + row) * HD + lane * E;
      sum += w;
#pragma unroll
      for (int e = 0; e < E; ++e) acc[e] = fmaf(w, p[e], acc[e]);
    }
  }
  const bool have = !(sum <= 0.f);
  const float inv = have ? 1.f / sum : 0.f;
  const int q = (int)(row % args.Sq);
  const long long bh = row / args.Sq;
  if (!NB_IN_BOUNDS(NB_SITE_ATTN_STORE, bh, (long long)args.B * args.H)) return;
  __nv_bfloat16* orow = args.O + (bh / args.H) * args.o_sb + (bh % args.H) * args.o_sh + q * args.o_ss + lane * E;
#pragma unroll
  for (int e = 0; e < E; e += 2) *reinterpret_cast<uint32_t*>(orow + e) = pack_bf16(acc[e] * inv, acc[e + 1] * inv);
  if (lane == 0) args.lse[row] = have ? mx + logf(sum) : -INFINITY;
}

// A few queries (at most 4 per head: decoding) against many keys, without a user mask. The work is one read of K
// and V: no tile of 128 query rows, no tensor core; K and V go from global memory to registers, 16 bytes per
// lane, HD / 8 lanes per key, DEC_U keys of K and of V in flight per lane, and every group of lanes keeps its
// own running maximum, sum and output (fp32), joined at the end of the block and, over the key ranges
// (gridDim.x), over the cluster or by attn_fwd_combine_kernel. 592 blocks (four per SM) of 4 x 16 B x 8 x 32 lanes hold the bytes
// in flight that HBM needs. 64 heads, 1 query, 4001 keys of 128: 68 us with the tile kernel, 42 here with the join
// (3.1 TB/s); 16 heads, 8000 keys: 120 -> 36 us.
struct DecodeArgs {
  FwdArgs f;
  const __nv_bfloat16 *q, *k, *v;
  long long q_sb, q_sh, q_ss, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss;
};
constexpr int DEC_MAX_Q = 4, DEC_U = 4;

// AHEAD (one query, blocks of four warps): the next keys and values are on their way while the current ones are worked on, for which four
// blocks fit an SM instead of seven: for grids that need no more (dec_ahead). Of eight warps with so many registers fewer clusters of 16 fit
// the chip (16 x 8000 18.1, 24.2), and two queries have the registers no more.
template <int HD, int NQ, int WARPS, bool CLUSTER, bool AHEAD>
__global__ void __launch_bounds__(32 * WARPS, NQ == 1 ? (WARPS == 4 ? (AHEAD ? 4 : 7) : 3) : NQ == 2 ? (WARPS == 4 ? 5 : 2) : 1) attn_decode_kernel(const DecodeArgs a) {
  follow_grid();
  constexpr int LPK = HD / 8, KPW = 32 / LPK, G = WARPS * KPW;      // lanes per key, keys per warp, lane groups per block
  const FwdArgs& f = a.f;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane / LPK, d0 = (lane % LPK) * 8;
  const int grp = warp * KPW + sub;
  const int sp = blockIdx.x, h = blockIdx.y % f.H, b = blockIdx.y / f.H;
  const int per = (f.Skv + f.nsplit - 1) / f.nsplit;
  const int k0 = sp * per, k1 = min(f.Skv, k0 + per);
  float q[NQ][8], acc[NQ][8], m[NQ], l[NQ];
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    m[i] = -INFINITY;
    l[i] = 0.f;
    uint4 raw = make_uint4(0, 0, 0, 0);
    if (i < f.Sq) raw = *reinterpret_cast<const uint4*>(a.q + b * a.q_sb + h * a.q_sh + i * a.q_ss + d0);
    const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      q[i][e] = __uint_as_float(e & 1 ? w[e >> 1] & 0xffff0000u : w[e >> 1] << 16) * f.scale_log2;
      acc[i][e] = 0.f;
    }
  }
  const __nv_bfloat16* kp = a.k + b * a.k_sb + h * a.k_sh + d0;
  const __nv_bfloat16* vp = a.v + b * a.v_sb + h * a.v_sh + d0;
  auto fetch = [&](int kb, uint4 (&kr)[DEC_U], uint4 (&vr)[DEC_U]) {
#pragma unroll
    for (int u = 0; u < DEC_U; ++u) {
      const int k = kb + u * G;
      kr[u] = vr[u] = make_uint4(0, 0, 0, 0);
      if (k < k1 && NB_IN_BOUNDS(NB_SITE_ATTN_TMA_COORD, k, f.Skv)) {
        kr[u] = *reinterpret_cast<const uint4*>(kp + k * a.k_ss);
        vr[u] = *reinterpret_cast<const uint4*>(vp + k * a.v_ss);
      }
    }
  };
  uint4 kr[DEC_U], vr[DEC_U], kn[DEC_U], vn[DEC_U];
  if (AHEAD) fetch(k0 + grp, kn, vn);
  for (int kb = k0 + grp; kb - grp < k1; kb += G * DEC_U) {
    if (AHEAD) {
#pragma unroll
      for (int u = 0; u < DEC_U; ++u) { kr[u] = kn[u]; vr[u] = vn[u]; }
      fetch(kb + G * DEC_U, kn, vn);
    } else {
      fetch(kb, kr, vr);
    }
    float s[NQ][DEC_U];
#pragma unroll
    for (int u = 0; u < DEC_U; ++u) {
      const uint32_t w[4] = {kr[u].x, kr[u].y, kr[u].z, kr[u].w};
#pragma unroll
      for (int i = 0; i < NQ; ++i) s[i][u] = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float x = __uint_as_float(e & 1 ? w[e >> 1] & 0xffff0000u : w[e >> 1] << 16);
#pragma unroll
        for (int i = 0; i < NQ; ++i) s[i][u] = fmaf(q[i][e], x, s[i][u]);
      }
    }
#pragma unroll
    for (int o = LPK / 2; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < NQ; ++i)
#pragma unroll
        for (int u = 0; u < DEC_U; ++u) s[i][u] += __shfl_xor_sync(0xffffffffu, s[i][u], o);
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      const int lim = min(k1, f.causal ? f.Skv - f.Sq + i + 1 : f.Skv);      // keys below lim are visible
      float mx = m[i];
#pragma unroll
      for (int u = 0; u < DEC_U; ++u) {
        if (kb + u * G >= lim) s[i][u] = -INFINITY;
        mx = fmaxf(mx, s[i][u]);
      }
      const float ms = mx == -INFINITY ? 0.f : mx;
      const float corr = ex2(m[i] - ms);
      m[i] = mx;
      l[i] *= corr;
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[i][e] *= corr;
#pragma unroll
      for (int u = 0; u < DEC_U; ++u) {
        s[i][u] = ex2(s[i][u] - ms);
        l[i] += s[i][u];
      }
    }
#pragma unroll
    for (int u = 0; u < DEC_U; ++u) {
      const uint32_t w[4] = {vr[u].x, vr[u].y, vr[u].z, vr[u].w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float x = __uint_as_float(e & 1 ? w[e >> 1] & 0xffff0000u : w[e >> 1] << 16);
#pragma unroll
        for (int i = 0; i < NQ; ++i) acc[i][e] = fmaf(s[i][u], x, acc[i][e]);
      }
    }
  }
  __shared__ float sm[G][NQ], sl[G][NQ], so[G][NQ][HD];
#pragma unroll
  for (int i = 0; i < NQ; ++i) {
    if (d0 == 0) { sm[grp][i] = m[i]; sl[grp][i] = l[i]; }
#pragma unroll
    for (int e = 0; e < 8; ++e) so[grp][i][d0 + e] = acc[i][e];
  }
  __shared__ float to[NQ][HD], tl[NQ];               // this block's range: output and log-sum-exp
  __syncthreads();
  const long long rows = (long long)f.B * f.H * f.Sq;
  for (int t = threadIdx.x; t < NQ * HD; t += 32 * WARPS) {
    const int i = t / HD, d = t % HD;
    if (i >= f.Sq) break;
    float mx = -INFINITY, sum = 0.f, o = 0.f;
#pragma unroll
    for (int g = 0; g < G; ++g) mx = fmaxf(mx, sm[g][i]);
    const float ms = mx == -INFINITY ? 0.f : mx;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const float w = ex2(sm[g][i] - ms);
      sum = fmaf(w, sl[g][i], sum);
      o = fmaf(w, so[g][i][d], o);
    }
    const bool have = !(sum <= 0.f);                 // NaN counts: it has to show
    o = have ? o / sum : 0.f;
    const float lse = have ? (mx + log2f(sum)) * 0.6931471805599453f : -INFINITY;
    const long long row = ((long long)b * f.H + h) * f.Sq + i;
    if (!NB_IN_BOUNDS(NB_SITE_ATTN_STORE, row, rows) || !NB_IN_BOUNDS(NB_SITE_ATTN_STORE, sp, f.nsplit)) continue;
    if (CLUSTER) {
      to[i][d] = o;
      if (d == 0) tl[i] = lse;
    } else if (f.nsplit > 1) {
      f.part_o[(sp * rows + row) * HD + d] = o;
      if (d == 0) f.part_lse[sp * rows + row] = lse;
    } else {
      f.O[b * f.o_sb + h * f.o_sh + i * f.o_ss + d] = __float2bfloat16(o);
      if (d == 0) f.lse[row] = lse;
    }
  }
  if (CLUSTER) {
    // the ranges of a (batch, head) are the blocks of a cluster: every block joins its share of the outputs, as
    // attn_fwd_combine_kernel does from memory
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    cluster.sync();
    for (int t = sp * 32 * WARPS + threadIdx.x; t < NQ * HD; t += f.nsplit * 32 * WARPS) {
      const int i = t / HD, d = t % HD;
      if (i >= f.Sq) break;
      float mx = -INFINITY;
      bool nan = false;                              // a NaN range makes the row NaN (fmaxf would drop it)
      for (int r = 0; r < f.nsplit; ++r) {
        const float v = *cluster.map_shared_rank(&tl[i], r);
        mx = fmaxf(mx, v);
        nan |= v != v;
      }
      if (nan) mx = NAN;
      float acc = 0.f, sum = 0.f;
      if (mx != -INFINITY)
        for (int r = 0; r < f.nsplit; ++r) {
          const float w = ex2((*cluster.map_shared_rank(&tl[i], r) - mx) * LOG2E);
          sum += w;
          acc = fmaf(w, *cluster.map_shared_rank(&to[i][d], r), acc);
        }
      const bool have = !(sum <= 0.f);
      const long long row = ((long long)b * f.H + h) * f.Sq + i;
      if (!NB_IN_BOUNDS(NB_SITE_ATTN_STORE, row, rows)) continue;
      f.O[b * f.o_sb + h * f.o_sh + i * f.o_ss + d] = __float2bfloat16(have ? acc / sum : 0.f);
      if (d == 0) f.lse[row] = have ? mx + logf(sum) : -INFINITY;
    }
    cluster.sync();                                  // a block's shared memory is read until here
  }
}

// ====================================================================== backward
struct BwdArgs {
  int B, H, Sq, Skv, Sq_pad;
  float scale, scale_log2;
  int causal;
  const float* nlse2;   // [B][H][Sq_pad]  -(log-sum-exp) in the log2 domain; -inf on padding rows and rows without keys
  const float* ndelta;  // [B][H][Sq_pad]  -rowsum(dO * O), 0 on padding rows
  __nv_bfloat16 *dQ, *dK, *dV;
  long long dq_sb, dq_sh, dq_ss, dk_sb, dk_sh, dk_ss, dv_sb, dv_sh, dv_ss;
  MaskArg mask;
  int* status;
  int vec32;               // rows of dQ, dK and dV start on 32-byte boundaries
  int q_chunk, kv_chunk;   // see tile_order: of the dK / dV kernel (Q and dO shared) and of the dQ kernel (K and V)
};

// ---------------------------------------------------------------------- dK / dV
template <int HD>
struct DkvSmem {
  static constexpr int TILE_BYTES = BT * HD * 2;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = OFF_K + TILE_BYTES;
  static constexpr int QST = 3;                           // Q stages: a Q tile is held from S^T until dK has read it,
                                                          // so two would leave its load half a tile's time
                                                          // (forward and backward at 64 heads x 2048: 461 -> 453 us)
  static constexpr int OFF_Q = OFF_V + TILE_BYTES;        // QST stages
  static constexpr int OFF_DO = OFF_Q + QST * TILE_BYTES; // 2 stages
  static constexpr int OFF_STAT = OFF_DO + 2 * TILE_BYTES;   // lse2[QST][128], delta[2][128]
  static constexpr int OFF_BAR = OFF_STAT + (QST + 2) * BT * 4;
  static constexpr int RAW = OFF_BAR + 18 * 8 + 16;       // no slack: the kernel's shared memory is 1024-byte aligned
  static constexpr int TOTAL = RAW < 120 * 1024 ? 120 * 1024 : RAW;
};

// Tensor memory: dV, dK and NREG regions of 128 columns (three where head_dim 64 leaves room, else two), which S^T and dP^T
// of the tiles take in turn. P^T and dS^T (bf16, 32 columns each per group) go over the score columns that their own threads
// have read. So a region that held dP^T is free once that is in registers: S^T of the next tile is multiplied while dS^T is
// made (three regions: from when P^T is written); dP^T of the next tile follows dK in the issue order and is ready before
// its exponentials are. With S^T and dP^T in fixed places a thread waited 1700 of 4050 clocks per tile for
// scores, 850 of 3250 this way (64 heads x 2048 x 128, causal: dK and dV 177 -> 149 us, with the 32-byte stores).
template <int HD, UserMask MASK>
__global__ void __launch_bounds__(NTHREADS, 1)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                     const BwdArgs args) {
  using L = DkvSmem<HD>;
  constexpr int QST = L::QST;
  extern __shared__ __align__(1024) uint8_t smem_tiles[];
  uint8_t* smem = smem_tiles;
  uint8_t* sK = smem + L::OFF_K;
  uint8_t* sV = smem + L::OFF_V;
  uint8_t* sQ = smem + L::OFF_Q;
  uint8_t* sDO = smem + L::OFF_DO;
  float* s_nlse2 = reinterpret_cast<float*>(smem + L::OFF_STAT);   // [QST][128]
  float* s_ndelta = s_nlse2 + QST * BT;                            // [2][128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;     // [QST] Q_i and its lse2 landed in stage i % QST
  uint64_t* q_empty = bars + 4;    // [QST]
  uint64_t* do_full = bars + 7;    // [2]  dO_i and its delta landed
  uint64_t* do_empty = bars + 9;   // [2]  dV has read dO_i, and all threads their deltas of it
  uint64_t* s_full = bars + 11;    //      S^T of the current tile is in TMEM
  uint64_t* dp_full = bars + 12;   //      dP^T of the current tile is in TMEM
  uint64_t* p_full = bars + 13;    //      P^T written back (256 arrivals)
  uint64_t* ds_full = bars + 14;   //      dS^T written back (256 arrivals)
  uint64_t* all_done = bars + 15;
  uint64_t* dp_read = bars + 16;   //      two regions: dP^T of the current tile is in registers (256 arrivals)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // an earlier bounded wait on this device already failed, as far as is known before the grid ahead has ended: leave (uniformly)
  if (__syncthreads_or(threadIdx.x == 0 ? *reinterpret_cast<volatile int*>(args.status) : 0)) return follow_grid();
  if (smem_u32(smem) & 1023u) {     // the swizzled tiles need it, and the size above leaves no room to align
    if (threadIdx.x == 0) atomicExch(args.status, NB_ERR_TIMEOUT_PRODUCER);
    return follow_grid();
  }
  int bh_, jt;             // key tile 0 sees every query tile, the last one only a few
  tile_order(blockIdx.x, args.H * args.B, args.q_chunk, (args.Skv + BT - 1) / BT, bh_, jt);
  const int h = bh_ % args.H;
  const int b = bh_ / args.H;
  const int k0 = jt * BT;
  const int off = args.Skv - args.Sq;
  const int nqt = (args.Sq + BT - 1) / BT;
  int i_start = 0;
  if (args.causal) {
    const int first_q = k0 - off;             // first query row that sees key k0
    i_start = first_q <= 0 ? 0 : first_q / BT;
  }
  const int n_it = max(0, nqt - i_start);
  const long long bh = (long long)b * args.H + h;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
    mbar_init(kv_full, 1);
    for (int i = 0; i < QST; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
    }
    mbar_init(s_full, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, 256);
    mbar_init(ds_full, 256);
    mbar_init(all_done, 1);
    mbar_init(dp_read, 256);
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  follow_grid();
  constexpr int NREG = HD == 64 ? 3 : 2;
  const uint32_t t_dv = tmem_base + NREG * 128, t_dk = t_dv + HD;
  auto t_s = [&](int it) { return tmem_base + (NREG == 3 ? 2 * it % 3 : it & 1) * 128; };            // S^T of tile it
  auto t_dp = [&](int it) { return tmem_base + (NREG == 3 ? (2 * it + 1) % 3 : (it + 1) & 1) * 128; };

  if (warp == 0) {
    if (n_it > 0 && elect_one()) {
      mbar_arrive_expect_tx(kv_full, 2 * L::TILE_BYTES);
#pragma unroll
      for (int c = 0; c < HD / 64; ++c) {
        tma_load_4d(sK + c * (BT * 128), &tmK, kv_full, c * 64, k0, h, b, args.Skv, args.H, args.B);
        tma_load_4d(sV + c * (BT * 128), &tmV, kv_full, c * 64, k0, h, b, args.Skv, args.H, args.B);
      }
      for (int it = 0; it < n_it; ++it) {
        const int st = it & 1, qs = it % QST;
        const uint32_t ph = ((it >> 1) & 1) ^ 1;
        const int q0 = (i_start + it) * BT;
        if (!mbar_wait(&q_empty[qs], ((it / QST) & 1) ^ 1)) { atomicExch(args.status, NB_ERR_TIMEOUT_PRODUCER); break; }
        mbar_arrive_expect_tx(&q_full[qs], L::TILE_BYTES + BT * 4);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          tma_load_4d(sQ + qs * L::TILE_BYTES + c * (BT * 128), &tmQ, &q_full[qs], c * 64, q0, h, b, args.Sq, args.H, args.B);
        if (!NB_IN_BOUNDS(NB_SITE_ATTN_STAT_INDEX, q0 + BT - 1, args.Sq_pad)) break;   // debug build only
        bulk_load_1d(s_nlse2 + qs * BT, args.nlse2 + bh * args.Sq_pad + q0, BT * 4, &q_full[qs]);
        if (!mbar_wait(&do_empty[st], ph)) { atomicExch(args.status, NB_ERR_TIMEOUT_PRODUCER); break; }
        mbar_arrive_expect_tx(&do_full[st], L::TILE_BYTES + BT * 4);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          tma_load_4d(sDO + st * L::TILE_BYTES + c * (BT * 128), &tmDO, &do_full[st], c * 64, q0, h, b, args.Sq, args.H, args.B);
        bulk_load_1d(s_ndelta + st * BT, args.ndelta + bh * args.Sq_pad + q0, BT * 4, &do_full[st]);
      }
    }
  } else if (warp == 1) {
    if (n_it > 0 && elect_one()) {
      bool ok = mbar_wait(kv_full, 0) && mbar_wait(&q_full[0], 0);
      if (ok) {
        tc_fence_after();
        mma_scores<HD>(t_s(0), smem_u32(sK), smem_u32(sQ));          // S^T_0 = K Q_0^T
        umma_commit(s_full);
        ok = mbar_wait(&do_full[0], 0);
      }
      if (ok) {
        tc_fence_after();
        mma_scores<HD>(t_dp(0), smem_u32(sV), smem_u32(sDO));        // dP^T_0 = V dO_0^T
        umma_commit(dp_full);
      }
      for (int it = 0; it < n_it && ok; ++it) {
        const int st = it & 1, qs = it % QST, qn = (it + 1) % QST;
        const bool more = it + 1 < n_it;
        // Scores of the next tile: their region held dP^T of this tile (two regions: free once all threads have read it) or
        // of the one before (three). Never before all have written P^T of this tile, so that none can arrive a second time
        // on a barrier where another has yet to arrive, or where this thread has yet to look.
        if (!mbar_wait(p_full, it & 1)) { ok = false; break; }
        if (more) {
          if (!(mbar_wait(&q_full[qn], ((it + 1) / QST) & 1) && (NREG == 3 || mbar_wait(dp_read, it & 1)))) { ok = false; break; }
          tc_fence_after();
          mma_scores<HD>(t_s(it + 1), smem_u32(sK), smem_u32(sQ + qn * L::TILE_BYTES));
          umma_commit(s_full);
        }
        tc_fence_after();
        mma_accum<HD>(t_dv, t_s(it), true, smem_u32(sDO + st * L::TILE_BYTES), it != 0);         // dV += P^T dO_i
        if (!mbar_wait(ds_full, it & 1)) { ok = false; break; }
        umma_commit(&do_empty[st]);        // behind ds_full: dS^T is made with the deltas that the next load into this stage replaces
        tc_fence_after();
        mma_accum<HD>(t_dk, t_s(it) + 32, true, smem_u32(sQ + qs * L::TILE_BYTES), it != 0);     // dK += dS^T Q_i
        umma_commit(&q_empty[qs]);
        if (more) {
          if (!mbar_wait(&do_full[st ^ 1], ((it + 1) >> 1) & 1)) { ok = false; break; }
          tc_fence_after();
          mma_scores<HD>(t_dp(it + 1), smem_u32(sV), smem_u32(sDO + (st ^ 1) * L::TILE_BYTES));
          umma_commit(dp_full);
        }
      }
      if (ok) umma_commit(all_done);
      else atomicExch(args.status, NB_ERR_TIMEOUT_MMA);
    }
  } else if (warp >= 4) {
    const int grp = (warp - 4) >> 2;        // query columns [64 grp, 64 grp + 64) of every tile
    const int wq = warp & 3;
    const int r = wq * 32 + lane;           // key row inside the tile
    const int key = k0 + r;
    const bool key_ok = key < args.Skv;
    const uint32_t lane_addr = static_cast<uint32_t>(wq * 32) << 16;
    const float* mbase = MASK == MASK_NONE ? nullptr : args.mask.ptr + b * args.mask.sb + h * args.mask.sh + key;
    // a mask with one row for all queries is one number per key here: added on the way into the exponent, no mask
    // pass, with the forward's roundings ((s + mask / scale) * scale_log2 - lse: where all keys of a row share
    // a large offset, any other order rounds the offset and the log-sum-exp apart)
    constexpr bool mkey = MASK == MASK_KEYS;
    const float mval = mkey && key_ok ? mbase[0] : 0.f;
    const float mask_mul = LOG2E / args.scale_log2;
    const float2 mval2 = make_float2(mval, mval), mul2 = make_float2(mask_mul, mask_mul);
    bool ok = true;
    for (int it = 0; it < n_it; ++it) {
      const int st = it & 1, qs = it % QST;
      const int q0 = (i_start + it) * BT + grp * 64;
      // (dO and its delta have landed by the time the scores are there)
      if (ok && !(mbar_wait(&q_full[qs], (it / QST) & 1) && mbar_wait(&do_full[st], (it >> 1) & 1) && mbar_wait(s_full, it & 1))) {
        atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const uint32_t a_s = t_s(it) + lane_addr + grp * 64, a_dp = t_dp(it) + lane_addr + grp * 64;
      const bool general = (args.causal && (k0 + BT - 1 > q0 + off)) || (k0 + BT > args.Skv) || MASK == MASK_ROWS;
      if (MASK == MASK_ROWS) {
        // rewrite S^T in place with the mask, -inf where (key, query) is not visible
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(a_s + c * 32, v);
          tmem_ld_wait32(v);
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int q = q0 + c * 32 + i;
            float x = __uint_as_float(v[i]);
            if (key_ok && q < args.Sq) x = fmaf(mbase[(long long)q * args.mask.sq], mask_mul, x);
            if (!key_ok || (args.causal && key > q + off)) x = -INFINITY;
            v[i] = __float_as_uint(x);
          }
          tmem_st_32x32(a_s + c * 32, v);
        }
        tmem_st_wait();
      }
      const float2* nl2 = reinterpret_cast<const float2*>(s_nlse2 + qs * BT + grp * 64);
      const float2 sc2 = make_float2(args.scale_log2, args.scale_log2);
      float2 p[32];
      uint32_t va[32], vb[32];
      tmem_ld_32x32(a_s, va);
      tmem_ld_32x32(a_s + 32, vb);
      tmem_ld_wait32(va);
      tmem_ld_wait32(vb);
      if (MASK != MASK_ROWS && general) {
        // diagonal or tail tile: -inf below the first query of this group that sees the key (one bound, so that the
        // compiler selects; two conditions per element became branches, 3400 clocks a tile)
        const int first = !key_ok ? 64 : args.causal ? key - off - q0 : 0;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t (&v)[32] = c ? vb : va;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            float x = __uint_as_float(v[i]);
            if (mkey) x = fmaf(mval, mask_mul, x);
            v[i] = __float_as_uint(c * 32 + i < first ? -INFINITY : x);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t (&v)[32] = c ? vb : va;
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float2 x = f2(v[2 * i], v[2 * i + 1]);
          if (mkey && !general) x = __ffma2_rn(mval2, mul2, x);      // else the mask pass has added it, under the -inf
          x = __ffma2_rn(x, sc2, nl2[c * 16 + i]);
          p[c * 16 + i] = make_float2(ex2(x.x), ex2(x.y));
          pk[i] = pack_bf16(p[c * 16 + i].x, p[c * 16 + i].y);
        }
        tmem_st_32x16(a_s + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(p_full);
      if (!mbar_wait(dp_full, it & 1)) {
        atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float2* nd2 = reinterpret_cast<const float2*>(s_ndelta + st * BT + grp * 64);
      tmem_ld_32x32(a_dp, va);
      tmem_ld_32x32(a_dp + 32, vb);
      tmem_ld_wait32(va);
      tmem_ld_wait32(vb);
      if (NREG == 2) {
        tc_fence_before();
        mbar_arrive(dp_read);
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t (&v)[32] = c ? vb : va;
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          // dS^T / scale = P^T * (dP^T - delta); the scale is applied once, to dK, in the epilogue
          const float2 d = __fmul2_rn(p[c * 16 + i], __fadd2_rn(f2(v[2 * i], v[2 * i + 1]), nd2[c * 16 + i]));
          pk[i] = pack_bf16(d.x, d.y);
        }
        tmem_st_32x16(a_s + 32 + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(ds_full);
    }
    if (ok && n_it > 0) {
      if (!mbar_wait(all_done, 0)) {
        atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (ok) tc_fence_after();
    }
    if (ok) {
      // group 0 writes this key's dK row, group 1 its dV row
      __nv_bfloat16* dst = grp == 0
          ? args.dK + (long long)b * args.dk_sb + (long long)h * args.dk_sh + (long long)key * args.dk_ss
          : args.dV + (long long)b * args.dv_sb + (long long)h * args.dv_sh + (long long)key * args.dv_ss;
      const uint32_t src = (grp == 0 ? t_dk : t_dv) + lane_addr;
      const float mul = grp == 0 ? args.scale : 1.f;
#pragma unroll
      for (int c = 0; c < HD / 32; ++c) {
        uint32_t v[32];
        if (n_it > 0) {
          tmem_ld_32x32(src + c * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0;
        }
        if (key_ok) {
          store_row32(dst + c * 32, v, mul, args.vec32);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------- dQ
template <int HD>
struct DqSmem {
  static constexpr int TILE_BYTES = BT * HD * 2;
  static constexpr int KST = 3;                             // K stages (a K tile is held until its dQ product retires)
  static constexpr int OFF_Q = 0;
  static constexpr int OFF_DO = OFF_Q + TILE_BYTES;
  static constexpr int OFF_K = OFF_DO + TILE_BYTES;
  static constexpr int OFF_V = OFF_K + KST * TILE_BYTES;    // 2 stages
  static constexpr int OFF_MASK = OFF_V + 2 * TILE_BYTES;   // [2 math groups][2][64] mask values of a key tile
  static constexpr int OFF_BAR = OFF_MASK + 4 * 64 * 4;
  static constexpr int RAW = OFF_BAR + 21 * 8 + 16 + 1024;
  static constexpr int TOTAL = RAW < 120 * 1024 ? 120 * 1024 : RAW;
};

// dS goes over the score columns that its own threads have read, so dP of the next tile needs its region only after dP was
// read, and S of the tile after next follows dQ in the issue order: with dS over dP a thread waited 1200 of 3100 clocks per
// tile for scores, 300 of 2190 this way (64 heads x 2048 x 128, causal: 127 -> 111 us).
template <int HD, UserMask MASK>
__global__ void __launch_bounds__(NTHREADS, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                   const BwdArgs args) {
  using L = DqSmem<HD>;
  constexpr int KST = L::KST;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem + L::OFF_Q;
  uint8_t* sDO = smem + L::OFF_DO;
  uint8_t* sK = smem + L::OFF_K;
  uint8_t* sV = smem + L::OFF_V;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::OFF_BAR);
  uint64_t* q_full = bars + 0;
  uint64_t* k_full = bars + 1;     // [3]
  uint64_t* k_empty = bars + 4;    // [3]
  uint64_t* v_full = bars + 7;     // [2]
  uint64_t* v_empty = bars + 9;    // [2]
  uint64_t* s_full = bars + 11;    // [2]  score buffer j & 1 holds S_j
  uint64_t* dp_full = bars + 13;   //      dP_j is in TMEM
  uint64_t* ds_full = bars + 18;   // [2]  dS_j written back (256 arrivals); two, because dP_j+1 may let a thread come here again
                                   //      before another has arrived for dS_j
  uint64_t* dq_done = bars + 15;
  uint64_t* dp_read = bars + 16;   //      dP_j is in registers (256 arrivals)
  uint64_t* do_full = bars + 17;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 20);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // an earlier bounded wait on this device already failed, as far as is known before the grid ahead has ended: leave (uniformly)
  if (__syncthreads_or(threadIdx.x == 0 ? *reinterpret_cast<volatile int*>(args.status) : 0)) return follow_grid();
  const int nqt = (args.Sq + BT - 1) / BT;
  int bh_, rank;
  tile_order(blockIdx.x, args.H * args.B, args.kv_chunk, nqt, bh_, rank);
  const int qt = nqt - 1 - rank;          // the late tiles of a causal problem see the most keys
  const int h = bh_ % args.H;
  const int b = bh_ / args.H;
  const int q0 = qt * BT;
  const int off = args.Skv - args.Sq;
  int n = (args.Skv + BT - 1) / BT;
  if (args.causal) {
    const int last_key = min(args.Skv - 1, q0 + BT - 1 + off);
    n = last_key < 0 ? 0 : last_key / BT + 1;
  }
  const long long bh = (long long)b * args.H + h;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
    mbar_init(q_full, 1);
    mbar_init(do_full, 1);
    for (int i = 0; i < KST; ++i) {
      mbar_init(&k_full[i], 1);
      mbar_init(&k_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&v_full[i], 1);
      mbar_init(&v_empty[i], 1);
      mbar_init(&s_full[i], 1);
    }
    mbar_init(dp_full, 1);
    mbar_init(&ds_full[0], 256);
    mbar_init(&ds_full[1], 256);
    mbar_init(dq_done, 1);
    mbar_init(dp_read, 256);
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == 2) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // (An exception to the rule, see launch.cuh.) The dK / dV kernel ahead writes nothing that is read here, and it lets this grid begin only when the statistics and all before them
  // are in memory: so the blocks work beside its last ones and wait for its end before their own. (Reads go to L2, past lines that this SM
  // may hold; a mask of rows is read through them.) us: 2 x 8 heads x 1001 x 64 causal 184 -> 176 in
  // a block's training step, 8 x 12 x 777 x 64 with a mask of keys 200 -> 198 and 4 x 16 x 2048 x 128 397 -> 394, both with their forward pass.
  constexpr bool BESIDE = MASK != MASK_ROWS;
  if (BESIDE) let_next_grid_start();
  else follow_grid();
  const uint32_t t_dp = tmem_base + 256, t_dq = tmem_base + 384;   // S buffers at 0 and 128

  if (warp == 0) {
    if (n > 0 && elect_one()) {
      mbar_arrive_expect_tx(q_full, L::TILE_BYTES);
#pragma unroll
      for (int c = 0; c < HD / 64; ++c)
        tma_load_4d(sQ + c * (BT * 128), &tmQ, q_full, c * 64, q0, h, b, args.Sq, args.H, args.B);
      for (int j = 0; j < n; ++j) {
        const int ks = j % KST, vs = j & 1;
        if (!mbar_wait(&k_empty[ks], ((j / KST) & 1) ^ 1)) { atomicExch(args.status, NB_ERR_TIMEOUT_PRODUCER); break; }
        mbar_arrive_expect_tx(&k_full[ks], L::TILE_BYTES);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          tma_load_4d(sK + ks * L::TILE_BYTES + c * (BT * 128), &tmK, &k_full[ks], c * 64, j * BT, h, b, args.Skv, args.H, args.B);
        if (j == 0) {                      // behind Q and K, which the first scores wait for
          mbar_arrive_expect_tx(do_full, L::TILE_BYTES);
#pragma unroll
          for (int c = 0; c < HD / 64; ++c)
            tma_load_4d(sDO + c * (BT * 128), &tmDO, do_full, c * 64, q0, h, b, args.Sq, args.H, args.B);
        }
        if (!mbar_wait(&v_empty[vs], ((j >> 1) & 1) ^ 1)) { atomicExch(args.status, NB_ERR_TIMEOUT_PRODUCER); break; }
        mbar_arrive_expect_tx(&v_full[vs], L::TILE_BYTES);
#pragma unroll
        for (int c = 0; c < HD / 64; ++c)
          tma_load_4d(sV + vs * L::TILE_BYTES + c * (BT * 128), &tmV, &v_full[vs], c * 64, j * BT, h, b, args.Skv, args.H, args.B);
      }
    }
  } else if (warp == 1) {
    if (n > 0 && elect_one()) {
      auto scores = [&](int j) {          // S_j = Q K_j^T into buffer j & 1
        mma_scores<HD>(tmem_base + (j & 1) * BT, smem_u32(sQ), smem_u32(sK + (j % KST) * L::TILE_BYTES));
        umma_commit(&s_full[j & 1]);
      };
      auto dprobs = [&](int j) {          // dP_j = dO V_j^T
        mma_scores<HD>(t_dp, smem_u32(sDO), smem_u32(sV + (j & 1) * L::TILE_BYTES));
        umma_commit(dp_full);
        umma_commit(&v_empty[j & 1]);
      };
      bool ok = mbar_wait(q_full, 0) && mbar_wait(&k_full[0], 0);
      if (ok) {
        tc_fence_after();
        scores(0);
        ok = mbar_wait(do_full, 0) && mbar_wait(&v_full[0], 0);
      }
      if (ok) {
        tc_fence_after();
        dprobs(0);
        if (n > 1) {
          ok = mbar_wait(&k_full[1], 0);
          if (ok) {
            tc_fence_after();
            scores(1);
          }
        }
      }
      for (int j = 0; j < n && ok; ++j) {
        if (j + 1 < n) {
          if (!(mbar_wait(&v_full[(j + 1) & 1], ((j + 1) >> 1) & 1) && mbar_wait(dp_read, j & 1))) { ok = false; break; }
          tc_fence_after();
          dprobs(j + 1);
        }
        if (!mbar_wait(&ds_full[j & 1], (j >> 1) & 1)) { ok = false; break; }
        tc_fence_after();
        mma_accum<HD>(t_dq, tmem_base + (j & 1) * BT, true, smem_u32(sK + (j % KST) * L::TILE_BYTES), j != 0);   // dQ += dS_j K_j
        umma_commit(&k_empty[j % KST]);
        if (j + 2 < n) {
          if (!mbar_wait(&k_full[(j + 2) % KST], ((j + 2) / KST) & 1)) { ok = false; break; }
          tc_fence_after();
          scores(j + 2);
        }
      }
      if (ok) umma_commit(dq_done);
      else atomicExch(args.status, NB_ERR_TIMEOUT_MMA);
    }
  } else if (warp >= 4) {
    const int grp = (warp - 4) >> 2;        // key columns [64 grp, 64 grp + 64) of every tile
    const int wq = warp & 3;
    const int r = wq * 32 + lane;
    const int q_idx = q0 + r;
    const uint32_t lane_addr = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t a_dp = t_dp + lane_addr + grp * 64;
    // padded to whole tiles, so always in range (the debug build checks it and reads nothing otherwise)
    const bool stat_ok = NB_IN_BOUNDS(NB_SITE_ATTN_STAT_INDEX, q_idx, args.Sq_pad);
    const float nlse2 = stat_ok ? __ldcg(args.nlse2 + bh * args.Sq_pad + q_idx) : -INFINITY;
    const float ndelta = stat_ok ? __ldcg(args.ndelta + bh * args.Sq_pad + q_idx) : 0.f;
    // user mask: one row for all queries goes through shared memory (64 values per group and key tile) and is
    // added on the way into the exponent, with the forward's roundings (see the dK / dV kernel); a row per query is
    // read by its own thread in the mask pass
    const float* mrow = nullptr;
    constexpr bool mkey = MASK == MASK_KEYS;
    const float* mkeys = mkey ? args.mask.ptr + b * args.mask.sb + h * args.mask.sh : nullptr;
    if (MASK == MASK_ROWS && q_idx < args.Sq)
      mrow = args.mask.ptr + b * args.mask.sb + h * args.mask.sh + (long long)q_idx * args.mask.sq;
    float* smask = reinterpret_cast<float*>(smem + L::OFF_MASK) + grp * 128;
    const float mask_mul = LOG2E / args.scale_log2;
    const float2 mul2 = make_float2(mask_mul, mask_mul);
    float mnext = mkey && r < 64 && grp * 64 + r < args.Skv ? __ldcg(mkeys + grp * 64 + r) : 0.f;
    const int lim = args.causal ? min(args.Skv - 1, q_idx + off) : args.Skv - 1;
    bool ok = true;
    for (int j = 0; j < n; ++j) {
      const int kv0 = j * BT + grp * 64;
      bool masked = false;
      if (mkey) {
        if (r < 64) smask[(j & 1) * 64 + r] = mnext;
        masked = named_bar_or(2 + grp, 128, mnext != 0.f);
        mnext = j + 1 < n && r < 64 && kv0 + BT + r < args.Skv ? __ldcg(mkeys + kv0 + BT + r) : 0.f;
      }
      if (ok && !mbar_wait(&s_full[j & 1], (j >> 1) & 1)) {
        atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (mkey) continue;                // keep the group's barrier participation uniform
        break;
      }
      tc_fence_after();
      const bool general = (kv0 + 64 > args.Skv) || (args.causal && (kv0 + 63 > q0 + off)) || MASK == MASK_ROWS;
      const uint32_t a_s = tmem_base + (j & 1) * BT + lane_addr + grp * 64;
      if (MASK == MASK_ROWS) {
        // rewrite the scores in place with the mask, -inf where the key is not visible
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(a_s + c * 32, v);
          tmem_ld_wait32(v);
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            const int kc = kv0 + c * 32 + i;
            float x = __uint_as_float(v[i]);
            if (mrow != nullptr && kc < args.Skv) x = fmaf(mrow[kc], mask_mul, x);
            v[i] = __float_as_uint(kc <= lim ? x : -INFINITY);
          }
          tmem_st_32x32(a_s + c * 32, v);
        }
        tmem_st_wait();
      }
      const float2 sc2 = make_float2(args.scale_log2, args.scale_log2), nl2 = make_float2(nlse2, nlse2);
      float2 p[32];
      uint32_t va[32], vb[32];
      tmem_ld_32x32(a_s, va);
      tmem_ld_32x32(a_s + 32, vb);
      tmem_ld_wait32(va);
      tmem_ld_wait32(vb);
      if (mkey && masked) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t (&v)[32] = c ? vb : va;
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            const float2 x = __ffma2_rn(*reinterpret_cast<const float2*>(smask + (j & 1) * 64 + c * 32 + i), mul2, f2(v[i], v[i + 1]));
            v[i] = __float_as_uint(x.x);
            v[i + 1] = __float_as_uint(x.y);
          }
        }
      }
      if (MASK != MASK_ROWS && general) {
        // diagonal or tail tile: -inf where the key is not visible
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t (&v)[32] = c ? vb : va;
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (c * 32 + i > lim - kv0) v[i] = __float_as_uint(-INFINITY);
        }
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t (&v)[32] = c ? vb : va;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          float2 x = f2(v[2 * i], v[2 * i + 1]);
          x = __ffma2_rn(x, sc2, nl2);
          p[c * 16 + i] = make_float2(ex2(x.x), ex2(x.y));
        }
      }
      if (!mbar_wait(dp_full, j & 1)) {
        atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) {
        if (mkey) continue;
        break;
      }
      tc_fence_after();
      const float2 nd2 = make_float2(ndelta, ndelta);
      tmem_ld_32x32(a_dp, va);
      tmem_ld_32x32(a_dp + 32, vb);
      tmem_ld_wait32(va);
      tmem_ld_wait32(vb);
      tc_fence_before();
      mbar_arrive(dp_read);
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t (&v)[32] = c ? vb : va;
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          // dS / scale = P * (dP - delta); the scale is applied once, to dQ, in the epilogue
          const float2 d = __fmul2_rn(p[c * 16 + i], __fadd2_rn(f2(v[2 * i], v[2 * i + 1]), nd2));
          pk[i] = pack_bf16(d.x, d.y);
        }
        tmem_st_32x16(a_s + c * 16, pk);
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&ds_full[j & 1]);
    }
    if (ok && n > 0) {
      if (!mbar_wait(dq_done, 0)) {
        atomicExch(args.status, NB_ERR_TIMEOUT_EPILOGUE);
        ok = false;
      }
      ok = __all_sync(0xffffffffu, ok);
      if (ok) tc_fence_after();
    }
    if (ok) {
      // each group stores half of the head dim of its query row
      constexpr int HALF = HD / 2;
      __nv_bfloat16* dst = args.dQ + (long long)b * args.dq_sb + (long long)h * args.dq_sh + (long long)q_idx * args.dq_ss +
                           grp * HALF;
#pragma unroll
      for (int c = 0; c < HALF / 32; ++c) {
        uint32_t v[32];
        if (n > 0) {
          tmem_ld_32x32(t_dq + lane_addr + grp * HALF + c * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = 0;
        }
        if (q_idx < args.Sq) {
          store_row32(dst + c * 32, v, args.scale, args.vec32);
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (BESIDE) wait_for_previous_grid();
}

// ndelta[b][h][q] = -sum_d dO * O and nlse2 = -lse * log2(e), both padded to Sq_pad rows per
// (b, h): padding rows and rows whose lse is -inf (no visible key) get nlse2 = -inf (probability 0)
// and ndelta = 0. D / 8 lanes per row, 16-byte loads, PREP_U rows per group of lanes on their way; a block's rows lie in
// one (b, h) (they divide a tile of 128), so there is one division per block; the heads of the same rows, which lie side by side in
// memory, are neighbouring blocks. Whole backward pass, us, with 4 rows and the rows of a head as neighbours, and so: 4 x 16 x 2048 x
// 128 259.6, 256.7; 8 x 12 x 777 x 64 86.1, 84.4; 2 x 8 x 1001 x 64 23.0, 21.9; 4 x 16 x 4096 x 64 672, 662.
constexpr int PREP_U = 2;
template <int D>
__global__ void __launch_bounds__(256) attn_bwd_prep_kernel(const __nv_bfloat16* __restrict__ dO,
                                                           const __nv_bfloat16* __restrict__ O,
                                                           const float* __restrict__ lse, float* __restrict__ ndelta,
                                                           float* __restrict__ nlse2, int H, int Sq, int Sq_pad,
                                                           long long do_sb, long long do_sh, long long do_ss,
                                                           long long o_sb, long long o_sh, long long o_ss) {
  follow_grid(dO, O, lse);
  constexpr int LPR = D / 8, RPB = 256 / LPR * PREP_U;    // lanes per row: 16 or 8; rows per block: 32 or 64
  static_assert(BT % RPB == 0, "a block stays inside a (batch, head)");
  const int per_bh = Sq_pad / RPB, rows = blockIdx.x / H, h = blockIdx.x - rows * H, b = rows / per_bh, bh = b * H + h;
  const int q0 = (rows - b * per_bh) * RPB + threadIdx.x / LPR, sub = threadIdx.x % LPR;
  const __nv_bfloat16* pd = dO + b * do_sb + h * do_sh + sub * 8;
  const __nv_bfloat16* po = O + b * o_sb + h * o_sh + sub * 8;
  uint4 ra[PREP_U], rc[PREP_U];
#pragma unroll
  for (int u = 0; u < PREP_U; ++u) {
    const int q = q0 + u * (256 / LPR);
    ra[u] = rc[u] = make_uint4(0, 0, 0, 0);
    if (q < Sq) {
      ra[u] = *reinterpret_cast<const uint4*>(pd + q * do_ss);
      rc[u] = *reinterpret_cast<const uint4*>(po + q * o_ss);
    }
  }
#pragma unroll
  for (int u = 0; u < PREP_U; ++u) {
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&ra[u]);
    const __nv_bfloat162* pc = reinterpret_cast<const __nv_bfloat162*>(&rc[u]);
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = __bfloat1622float2(pa[e]), y = __bfloat1622float2(pc[e]);
      acc += x.x * y.x + x.y * y.y;
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const int q = q0 + u * (256 / LPR);
    if (sub == 0) {
      const float l = q < Sq ? lse[(long long)bh * Sq + q] : -INFINITY;
      ndelta[(long long)bh * Sq_pad + q] = q < Sq ? -acc : 0.f;
      nlse2[(long long)bh * Sq_pad + q] = l == -INFINITY ? -INFINITY : -l * LOG2E;
    }
  }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}
// (B, H, S, D) bf16 view with D contiguous; element strides sb, sh, ss. Box = 64 x 128 rows x 1 x 1.
static int make_map4(CUtensorMap* map, const void* ptr, int B, int H, int S, int D, long long sb, long long sh,
                     long long ss) {
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return -1;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)S, (cuuint64_t)H, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)ss * 2, (cuuint64_t)(H > 1 ? sh : ss * S) * 2, (cuuint64_t)(B > 1 ? sb : sh * H) * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)BT, 1, 1};
  cuuint32_t es[4] = {1, 1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, es,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -(int)r - 100;
}

template <typename K>
static int set_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? 0 : -2;
}

// (batch, head) pairs whose two (rows x HD) bf16 operands fill about a quarter of the 126 MB L2.
static int l2_chunk(int nbh, long long rows, int hd) {
  const long long n = (32ll << 20) / (rows * hd * 4 > 0 ? rows * hd * 4 : 1);
  return (int)(n < 1 ? 1 : n > nbh ? nbh : n);
}

template <int HD>
static void combine(const FwdArgs& a, cudaStream_t stream) {
  const long long rows = (long long)a.B * a.H * a.Sq;
  launch_following(attn_fwd_combine_kernel<HD>, (unsigned)((rows + 3) / 4), 128, 0, stream, a);
}

// Blocks of a cluster for so many warps on a (batch, head): of four warps, of eight above 32.
static int dec_cluster(int warps) { return warps > 32 ? warps / 8 : warps / 4; }

// Blocks that load ahead hold 592 of four warps on the chip, clusters of more than two of them 512 (not every group of SMs divides into whole ones). us,
// one query, loading ahead and not: clusters of 64 pairs x 4001 keys x 128 26.9, 28.1, of 148 (592 blocks) 76, 61; ranges of 148 pairs x 4001 55, 60, of
// 300 (600 blocks) 137, 107.
static bool dec_ahead(int queries, int warps, long long blocks) { return queries == 1 && warps <= 32 && blocks <= (warps > 8 ? 512 : 592); }

// warps 0: key ranges joined by a second launch.
template <int HD, int NQ>
static int launch_decode(const DecodeArgs& a, int warps, cudaStream_t stream) {
  constexpr bool ONE = NQ == 1;
  const dim3 grid(a.f.nsplit, a.f.B * a.f.H);
  const bool ahead = dec_ahead(a.f.Sq, warps, (long long)grid.x * grid.y);
  if (warps == 0) {
    launch_following(ahead ? attn_decode_kernel<HD, NQ, 4, false, ONE> : attn_decode_kernel<HD, NQ, 4, false, false>, grid, 128, 0, stream, a);
    if (a.f.nsplit > 1) combine<HD>(a.f, stream);
    return cudaGetLastError() == cudaSuccess ? 0 : -3;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)a.f.nsplit;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(warps > 32 ? 256 : 128);
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const auto kernel = warps > 32 ? attn_decode_kernel<HD, NQ, 8, true, false>
                      : ahead    ? attn_decode_kernel<HD, NQ, 4, true, ONE> : attn_decode_kernel<HD, NQ, 4, true, false>;
  if (a.f.nsplit > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return -2;
  set_following(cfg);
  return cudaLaunchKernelEx(&cfg, kernel, a) == cudaSuccess ? 0 : -3;
}
template <int HD>
static int launch_decode(const DecodeArgs& a, int warps, cudaStream_t stream) {
  return a.f.Sq == 1 ? launch_decode<HD, 1>(a, warps, stream) : a.f.Sq == 2 ? launch_decode<HD, 2>(a, warps, stream)
                                                                            : launch_decode<HD, 4>(a, warps, stream);
}

template <int HD, UserMask MASK>
static int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdArgs& a,
                      cudaStream_t stream) {
  using L = FwdSmem<HD, MASK == MASK_KEYS>;
  static bool configured = false;
  if (!configured) {
    if (set_smem(attn_fwd_kernel<HD, MASK>, L::TOTAL)) return -2;
    configured = true;
  }
  const int nqt = (a.Sq + a.q_tiles * BT - 1) / (a.q_tiles * BT);
  const long long grid = (long long)nqt * a.H * a.B * a.nsplit;
  if (grid <= 0) return 0;
  launch_following(attn_fwd_kernel<HD, MASK>, (unsigned)grid, NTHREADS, L::TOTAL, stream, tq, tk, tv, a);
  if (a.nsplit > 1) combine<HD>(a, stream);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

template <int HD, UserMask MASK>
static int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                      const BwdArgs& a, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    if (set_smem(attn_bwd_dkdv_kernel<HD, MASK>, DkvSmem<HD>::TOTAL)) return -2;
    if (set_smem(attn_bwd_dq_kernel<HD, MASK>, DqSmem<HD>::TOTAL)) return -2;
    configured = true;
  }
  const long long bh = (long long)a.H * a.B;
  const int nkt = (a.Skv + BT - 1) / BT, nqt = (a.Sq + BT - 1) / BT;
  launch_following(attn_bwd_dkdv_kernel<HD, MASK>, (unsigned)(nkt * bh), NTHREADS, DkvSmem<HD>::TOTAL, stream, tq, tk, tv, tdo, a);
  launch_following(attn_bwd_dq_kernel<HD, MASK>, (unsigned)(nqt * bh), NTHREADS, DqSmem<HD>::TOTAL, stream, tq, tk, tv, tdo, a);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace nba

// Few queries and no user mask: the decode kernel (gridDim.y holds the (batch, head) pairs), which keeps the probabilities
// in fp32 (1.65e-3 from 64 bits, 2.1e-3 to 2.4e-3 with tiles). Times of both over 4 .. 1024 pairs and 64 .. 16384 keys: its
// FMAs grow with the queries and head_dim, where the tile kernel's time does not; it starts sooner (12 -> 8 us over 64
// keys), and a tile kernel of more CTAs than SMs takes a wave per 148 pairs.
// One and two queries: most lengths are faster (256 pairs x 1000 keys x 64: 26 and 32 us, 41 with tiles; 64 x 4096 x 128: 42
// and 44, 46 and 44 in key ranges, 65 whole), two of head_dim 128 over 128 to 256 pairs up to 3 us or a tenth slower.
// Three and four, head_dim 64: one tile of keys, or from 256 pairs on (128 x 1000: 28 and 25 with tiles, 256 x 1000: 38 and
// 41). Head_dim 128: 64 keys, or below 256 where the pairs are more than a wave (4 queries, 128 x 4096: 114 and 68).
static bool attn_decode(int B, int H, int Sq, int Skv, int D, bool mask) {
  const long long bh = (long long)B * H;
  if (mask || Sq > nba::DEC_MAX_Q || bh > 65535) return false;
  if (Sq <= 2) return true;
  return D == 64 ? Skv <= nba::BT || bh >= 256 : Skv <= 64 || (bh > 148 && Skv < 256);
}

// Query tiles that a CTA of the tile kernel owns. Two share the keys that it loads, and one's softmax runs beside the other's
// products; alone a tile is done sooner (its two math groups' exponentials no longer queue for one SM), so a grid that has an
// SM for every tile gives it one. us with two and with one: 2 x 8 heads x 1001 x 64, causal, 19.3 and 15.2, full 20.9 and 15.6;
// 64 x 256 x 128 11.0 and 9.3; 4 x 2048 x 64 under a mask of keys 48.9 and 35.1. A second wave costs more than that (16 x 1500 x
// 64, full: 28.7 and 38.4). Three causal tiles stay: the last is alone as it is (32 x 333 x 128 10.8 and 11.1).
static int attn_q_tiles(int B, int H, int Sq, int Skv, int causal, int nsplit) {
  const long long tiles = (Sq + nba::BT - 1) / nba::BT;
  if (tiles * B * H * nsplit > 148) return 2;
  return causal && tiles == 3 && Skv <= Sq ? 2 : 1;
}

// Key ranges that a forward pass is cut into (1: none).
// Decode kernel: ranges of at least 128 keys, for four blocks per SM; at head_dim 64 none below 512 keys, where a block walks
// them before a second launch would have started (64 pairs x 300 keys: 12.3 us whole, 15.4 in two ranges; 16.4 and 15.4 at
// head_dim 128).
// Otherwise a CTA owns up to 256 queries of one (batch, head), so a short query block against a long prefix gives one
// CTA per (batch, head), each walking all key tiles alone. The rule counts what the busiest SM walks: waves *
// (key tiles per CTA + 3), the 3 standing for a CTA's start and end, and 3 more for the launch that joins the
// ranges (a tile is 1.7 us at head_dim 128, the join 5): 500 keys 16.4 us whole and 17.4 in four ranges, 520 keys 18.4 and
// 15.4, 4096 keys of 64 pairs 65 and 44. With more than one block of 256 queries it stays as it is (2 x 8 heads x 1001
// queries, causal: 25.6 us, 27.6 in two ranges; few heads over long prefixes would gain, 8 heads x 512 queries x 8192 keys 129 -> 38).
extern "C" int nb_attn_fwd_splits(int B, int H, int Sq, int Skv, int D, int has_mask) {
  constexpr int SMS = 148;
  if (B <= 0 || H <= 0 || Sq <= 0 || Skv <= 0) return 1;
  if (attn_decode(B, H, Sq, Skv, D, has_mask != 0)) {
    if (D == 64 && Skv < 512) return 1;
    long long s = (4ll * SMS + (long long)B * H - 1) / ((long long)B * H);
    if (s > Skv / 128) s = Skv / 128;
    return (int)(s < 1 ? 1 : s > 64 ? 64 : s);
  }
  const long long ctas = (long long)B * H;
  const int n = (Skv + nba::BT - 1) / nba::BT;
  if (Sq > 2 * nba::BT || ctas >= SMS) return 1;
  int best = 1;
  long long best_cost = n + 3;
  for (int s = 2; s <= 32 && s <= n; ++s) {
    const long long cost = ((ctas * s + SMS - 1) / SMS) * ((n + s - 1) / s + 3) + 3;
    if (cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

// Warps that a (batch, head) of the decode kernel is given in a cluster of blocks, which needs no scratch and no second launch (0: key
// ranges as above). Timed for every number of warps and the ranges over 4 to 512 pairs, 128 to 8000 keys, one and two queries, both head_dims (826
// sizes, calls in a row): as many warps as leave no cluster waiting for its turn, of four warps with eight keys each. The lines:
//  - blocks of eight warps take few pairs, by 3 (one query) and 2 blocks an SM; a pair on 16 of them wants keys enough for the larger exchange.
//  - of four warps 512 blocks load ahead, up to 800 do not, and those of larger clusters pay under more keys only. Two queries: 600 blocks.
//  - ranges win where they fill the chip evenly and clusters do not (148 pairs x 4001 x 128 55 us, clusters 61), where clusters would leave it half
//    empty under long walks (two queries, 37 x 4001 x 128 26.2, 30.1), and under few keys (256 x 300 x 64 9.1, 9.9).
// us, ranges and clusters, one query: 4 pairs x 8000 keys x 128 21.6, 13.6; 16 x 1000 12.2, 7.9; 32 x 4001 23.9, 19.7; 64 x 512 11.4, 8.8.
extern "C" int nb_attn_decode_warps(int B, int H, int Sq, int Skv, int D, int has_mask) {
  if (B <= 0 || H <= 0 || Sq <= 0 || Sq > 2 || Skv < 128 || !attn_decode(B, H, Sq, Skv, D, has_mask != 0)) return 0;
  const long long bh = (long long)B * H;
  const bool one = Sq == 1, wide = D == 128;
  auto takes = [&](int w) {
    if (w == 128) return bh <= (one ? 16 : 8) && Skv >= (bh <= 4 ? 1500 : 3000);
    if (w == 64) return bh <= (one ? 48 : 32) && Skv >= (wide ? 300 : 700) && (one || !wide || Skv < 8000);
    const long long blocks = bh * w / 4;
    return w * 8 <= Skv && (one ? blocks <= 512 || (blocks <= 800 && Skv >= (w == 8 ? 128 : w == 16 ? 700 : 1000)) : blocks <= 600);
  };
  int w = 128;
  while (w >= 8 && !takes(w)) w /= 2;
  if (w < 8) return 0;
  if (one) {
    if (w <= 32 && 592 % bh == 0 && (Skv >= 1500 || w * bh > 4 * 512)) return 0;
    if (wide ? (Skv < 160 && bh > 8) || (Skv < 300 && bh > 256) : (Skv < 200 && bh > 4) || (Skv < 300 && bh > 16) || (Skv < 320 && bh > 24 && bh < 64)) return 0;
    if (!wide && bh > 148 && Skv < 512) return 0;
  } else {
    if (w == 32 && Skv >= (w * bh < 1300 ? 3000 : wide ? 4000 : 6000)) return 0;
    if (w == 16 && bh > 74 && Skv >= (wide ? 700 : 1500)) return 0;
    if (w == 8 && w * bh < 1900 && Skv >= 1000) return 0;
    if (wide ? Skv < 160 && bh > 24 : Skv < 160 || (Skv < 300 && bh > 16) || (Skv < 512 && bh > 24 && bh < 64)) return 0;
    if (bh >= 148 && Skv < (wide ? 300 : 512)) return 0;
  }
  return w;
}

// q, k, v: bf16 (B, H, S, D) views, D contiguous, strides in elements (multiples of 8, 16-byte
// aligned bases). o: bf16 with its own strides. lse: fp32 [B][H][Sq]. D in {64, 128}.
// mask: optional fp32 additive mask (null = none), element strides m_sb, m_sh, m_sq (0 = broadcast),
// key stride 1. nsplit = nb_attn_fwd_splits(...) or 1; above 1 part_o / part_lse are fp32 scratch of
// nsplit * B * H * Sq * D and nsplit * B * H * Sq elements (16-byte aligned). nsplit = -nb_attn_decode_warps(...) where that
// is not 0.
extern "C" int nb_attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int H, int Sq,
                           int Skv, int D, long long q_sb, long long q_sh, long long q_ss, long long k_sb,
                           long long k_sh, long long k_ss, long long v_sb, long long v_sh, long long v_ss,
                           long long o_sb, long long o_sh, long long o_ss, float scale, int causal, const float* mask,
                           long long m_sb, long long m_sh, long long m_sq, int nsplit, float* part_o,
                           float* part_lse, int* status, void* stream) {
  using namespace nba;
  if (D != 64 && D != 128) return -10;
  if (!(scale > 0.f)) return -13;
  if (B <= 0 || H <= 0 || Sq <= 0) return 0;
  const int warps = nsplit < 0 ? -nsplit : 0;
  if (nsplit < 0) {
    if ((warps != 8 && warps != 16 && warps != 32 && warps != 64 && warps != 128) || Skv <= 0 || !attn_decode(B, H, Sq, Skv, D, mask != nullptr))
      return -14;
    nsplit = dec_cluster(warps);
  } else if (nsplit < 1 || (nsplit > 1 && (part_o == nullptr || part_lse == nullptr || (reinterpret_cast<uintptr_t>(part_o) & 15)))) return -14;
  const long long strides[] = {q_sb, q_sh, q_ss, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss, o_ss, o_sh, o_sb};
  for (long long s : strides)
    if (s & 7) return -12;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(o)) & 15)
    return -11;
  FwdArgs a;
  a.B = B; a.H = H; a.Sq = Sq; a.Skv = Skv;
  a.scale_log2 = scale * LOG2E;
  a.causal = causal;
  a.O = reinterpret_cast<__nv_bfloat16*>(o);
  a.o_sb = o_sb; a.o_sh = o_sh; a.o_ss = o_ss;
  a.lse = lse;
  a.mask = MaskArg{mask, m_sb, m_sh, m_sq};
  a.status = status;
  a.vec32 = ((reinterpret_cast<uintptr_t>(o) & 31) | ((o_sb | o_sh | o_ss) & 15)) == 0;
  a.q_tiles = attn_q_tiles(B, H, Sq, Skv, causal, nsplit);
  a.bh_chunk = causal ? l2_chunk(B * H, Skv, D) * nsplit : 1;
  a.nsplit = nsplit; a.part_o = part_o; a.part_lse = part_lse;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (Skv > 0 && attn_decode(B, H, Sq, Skv, D, mask != nullptr)) {
    const DecodeArgs d{a, reinterpret_cast<const __nv_bfloat16*>(q), reinterpret_cast<const __nv_bfloat16*>(k),
                       reinterpret_cast<const __nv_bfloat16*>(v), q_sb, q_sh, q_ss, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss};
    return D == 128 ? launch_decode<128>(d, warps, s) : launch_decode<64>(d, warps, s);
  }
  CUtensorMap tq, tk, tv;
  int r;
  if ((r = make_map4(&tq, q, B, H, Sq, D, q_sb, q_sh, q_ss))) return r;
  if ((r = make_map4(&tk, k, B, H, Skv, D, k_sb, k_sh, k_ss))) return r;
  if ((r = make_map4(&tv, v, B, H, Skv, D, v_sb, v_sh, v_ss))) return r;
  if (mask == nullptr) return D == 128 ? launch_fwd<128, MASK_NONE>(tq, tk, tv, a, s) : launch_fwd<64, MASK_NONE>(tq, tk, tv, a, s);
  if (m_sq == 0) return D == 128 ? launch_fwd<128, MASK_KEYS>(tq, tk, tv, a, s) : launch_fwd<64, MASK_KEYS>(tq, tk, tv, a, s);
  return D == 128 ? launch_fwd<128, MASK_ROWS>(tq, tk, tv, a, s) : launch_fwd<64, MASK_ROWS>(tq, tk, tv, a, s);
}

// Backward. All tensors are (B, H, S, D) bf16 views with the head dim contiguous (element strides
// given per tensor), D in {64, 128}; lse fp32 [B][H][Sq] from the forward. `stats`: fp32 scratch of
// 2 * B * H * Sq_pad elements (Sq_pad = Sq rounded up to 128), filled here (delta, then lse2).
extern "C" int nb_attn_bwd(const void* dO, const void* q, const void* k, const void* v, const void* o, const float* lse,
                           void* dq, void* dk, void* dv, float* stats, int B, int H, int Sq, int Skv, int D,
                           long long q_sb, long long q_sh, long long q_ss, long long k_sb, long long k_sh, long long k_ss,
                           long long v_sb, long long v_sh, long long v_ss, long long do_sb, long long do_sh,
                           long long do_ss, long long o_sb, long long o_sh, long long o_ss, long long dq_sb,
                           long long dq_sh, long long dq_ss, long long dk_sb, long long dk_sh, long long dk_ss,
                           long long dv_sb, long long dv_sh, long long dv_ss, float scale, int causal, const float* mask,
                           long long m_sb, long long m_sh, long long m_sq, int* status, void* stream) {
  using namespace nba;
  if (D != 64 && D != 128) return -10;
  if (!(scale > 0.f)) return -13;
  if (B <= 0 || H <= 0 || Sq <= 0 || Skv <= 0) return 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  const long long st[] = {q_sb, q_sh, q_ss, k_sb, k_sh, k_ss, v_sb, v_sh, v_ss, do_sb, do_sh, do_ss,
                          o_sb, o_sh, o_ss, dq_sb, dq_sh, dq_ss, dk_sb, dk_sh, dk_ss, dv_sb, dv_sh, dv_ss};
  for (long long x : st)
    if (x & 7) return -12;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(dO) | reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) |
       reinterpret_cast<uintptr_t>(dv) | reinterpret_cast<uintptr_t>(stats) | reinterpret_cast<uintptr_t>(o)) & 15)
    return -11;
  const int Sq_pad = (Sq + BT - 1) / BT * BT;
  const long long rows = (long long)B * H * Sq_pad;
  float* ndelta = stats;
  float* nlse2 = stats + rows;
  const long long prep = rows / (256 / (D / 8) * PREP_U);
  if (prep > 0x7fffffffll) return -15;
#define PREP(HD) launch_following(attn_bwd_prep_kernel<HD>, (unsigned)prep, 256, 0, s,  \
      reinterpret_cast<const __nv_bfloat16*>(dO), reinterpret_cast<const __nv_bfloat16*>(o), lse, ndelta, nlse2, H, Sq, Sq_pad, \
      do_sb, do_sh, do_ss, o_sb, o_sh, o_ss)
  if (D == 128) PREP(128);
  else PREP(64);
#undef PREP
  CUtensorMap tq, tk, tv, tdo;
  int r;
  if ((r = make_map4(&tq, q, B, H, Sq, D, q_sb, q_sh, q_ss))) return r;
  if ((r = make_map4(&tdo, dO, B, H, Sq, D, do_sb, do_sh, do_ss))) return r;
  if ((r = make_map4(&tk, k, B, H, Skv, D, k_sb, k_sh, k_ss))) return r;
  if ((r = make_map4(&tv, v, B, H, Skv, D, v_sb, v_sh, v_ss))) return r;
  BwdArgs a;
  a.B = B; a.H = H; a.Sq = Sq; a.Skv = Skv; a.Sq_pad = Sq_pad;
  a.scale = scale; a.scale_log2 = scale * LOG2E;
  a.causal = causal;
  a.nlse2 = nlse2; a.ndelta = ndelta;
  a.dQ = reinterpret_cast<__nv_bfloat16*>(dq);
  a.dK = reinterpret_cast<__nv_bfloat16*>(dk); a.dV = reinterpret_cast<__nv_bfloat16*>(dv);
  a.dq_sb = dq_sb; a.dq_sh = dq_sh; a.dq_ss = dq_ss;
  a.dk_sb = dk_sb; a.dk_sh = dk_sh; a.dk_ss = dk_ss; a.dv_sb = dv_sb; a.dv_sh = dv_sh; a.dv_ss = dv_ss;
  a.mask = MaskArg{mask, m_sb, m_sh, m_sq};
  a.status = status;
  a.vec32 = (((reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 31) |
             ((dq_sb | dq_sh | dq_ss | dk_sb | dk_sh | dk_ss | dv_sb | dv_sh | dv_ss) & 15)) == 0;
  a.q_chunk = causal ? l2_chunk(B * H, Sq, D) : B * H;
  a.kv_chunk = causal ? l2_chunk(B * H, Skv, D) : 1;
  if (mask == nullptr) return D == 128 ? launch_bwd<128, MASK_NONE>(tq, tk, tv, tdo, a, s) : launch_bwd<64, MASK_NONE>(tq, tk, tv, tdo, a, s);
  if (m_sq == 0) return D == 128 ? launch_bwd<128, MASK_KEYS>(tq, tk, tv, tdo, a, s) : launch_bwd<64, MASK_KEYS>(tq, tk, tv, tdo, a, s);
  return D == 128 ? launch_bwd<128, MASK_ROWS>(tq, tk, tv, tdo, a, s) : launch_bwd<64, MASK_ROWS>(tq, tk, tv, tdo, a, s);
}

NB_DEBUG_DEFINE(attention)
