// The learned guide: a small MLP that seeds the trick search and orders the root lead.
//
//   input  217 = 52 cards x 4 owners (one-hot) + 5 strains + 4 leaders, padded to 256
//   hidden 256 GELU, 256 GELU (BF16 weights and activations, FP32 accumulate)
//   heads  14 NS-trick classes (softmax) + 52 lead-card scores (softmax over the leader's
//          cards), padded to 80 outputs
//
// Inference and the per-row half of a training step run in one kernel, mlp_rows: one CTA
// takes a tile of 128 examples through every layer, activations staying in shared memory
// and accumulators in tensor memory. Products are tcgen05 (5th-generation tensor core)
// instructions for sm_100a: operands in shared memory in the no-swizzle K-major core-matrix
// layout, one thread issues tcgen05.mma, tcgen05.commit signals an mbarrier, and the
// epilogue reads the accumulator back with tcgen05.ld (bias, GELU or its derivative fused).
// The weights are kept in that layout in global memory, in chunks of 64 of K, and stream
// through a ring of four shared-memory slots by bulk copies. The weight gradients, sums
// over the batch, are a second kernel split along the batch (gemm_dw), and dw_finish adds
// the parts and applies Adam. The guide only changes where searches start and which lead
// is tried first; the exact searches decide every answer.
#pragma once
#include <cuda_bf16.h>

#include "ddg_guide_rows.cuh"

namespace guide_nn {

typedef __nv_bfloat16 bf16;

enum : int {
  IN = 217,
  IN_PAD = 256,
  HID = 256,
  OUT_T = 14,   // NS tricks 0..13
  OUT_M = 52,   // lead card (suit*13 + rank)
  OUT = OUT_T + OUT_M,
  OUT_PAD = 80,  // N of the last layer (a multiple of 16)
  DO_LD = 128,   // row length of dO: K of the dH2 = dO . W3 product (a multiple of 64)
  KCHUNK = 64,
};

// Flat parameter layout (fp32): W1[256][256] b1[256] W2[256][256] b2[256] W3[80][256] b3[80].
constexpr int64_t OFF_W1 = 0, OFF_B1 = OFF_W1 + HID * IN_PAD, OFF_W2 = OFF_B1 + HID, OFF_B2 = OFF_W2 + HID * HID,
                  OFF_W3 = OFF_B2 + HID, OFF_B3 = OFF_W3 + OUT_PAD * HID, N_PARAMS = OFF_B3 + OUT_PAD;

// Weights in the tensor cores' layout (bf16, byte offsets): W1 and W2 as B of the forward
// products (4 chunks of 32 KB each), W3 (4 of 10 KB), and as B of the backward products W3
// transposed (K = 128, 2 chunks) and W2 transposed (4).
constexpr int CHUNK = 256 * KCHUNK * 2, CHUNK3 = OUT_PAD * KCHUNK * 2;
constexpr int PK_W1 = 0, PK_W2 = 4 * CHUNK, PK_W3 = 8 * CHUNK, PK_W3T = PK_W3 + 4 * CHUNK3, PK_W2T = PK_W3T + 2 * CHUNK,
              PK_BYTES = PK_W2T + 4 * CHUNK;
// Byte offset of element (row n, column k) of a K-major operand with `rows` rows: core
// matrices of 8 rows x 16 bytes, (k / 8) * rows / 8 + n / 8 in order.
__host__ __device__ constexpr int core_at(int n, int k, int rows) {
  return ((k >> 3) * (rows >> 3) + (n >> 3)) * 128 + (n & 7) * 16 + (k & 7) * 2;
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor (tcgen05): start address, leading (K) and stride (M/N)
// byte offsets, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)((lbo >> 4) & 0x3FFFu) << 16 |
         (uint64_t)((sbo >> 4) & 0x3FFFu) << 32 | (uint64_t)1 << 46;
}

// Instruction descriptor of kind::f16: D f32, A and B bf16, both K-major, M = 128, N.
__device__ __forceinline__ uint32_t instr_desc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TILE_M >> 4) << 24);
}

// Waits for the mbarrier phase with parity `parity`; false if it did not complete within
// the bound (the caller records an error and winds down).
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  for (int it = 0; it < (1 << 24); it++) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// ---- one tile of examples through all layers --------------------------------------------

struct MlpArgs {
  const uint64_t* hands;
  const int64_t* rows;  // training: example of each row (-1: none); inference: null, row r is example r
  int64_t n;            // rows with an example (inference), or the padded number of rows (training)
  int tiles;
  const unsigned char* packed;
  const float* master;  // for the biases
  int8_t* seed20;       // inference: NS seeds and root leads, n each (or null)
  int8_t* hint20;
  const uint8_t* tricks20;  // training: labels
  const int8_t* best20;
  int R;                                  // training: row length of the transposed outputs below
  bf16 *Xt, *H1t, *H2t, *dOt, *dZ2t, *dZ1t;  // [column][row]
  float *Z1t, *Z2t;
  float* acc;  // loss, hits, rows
  int* err;
};

__device__ __forceinline__ int card_index(int bit) { return (bit >> 4) * 13 + (bit & 15); }
__device__ __forceinline__ constexpr int card_bit(int idx) { return (idx / 13) * 16 + idx % 13; }

template <bool TRAIN>
constexpr int MLP_THREADS = TRAIN ? 512 : 1024;
constexpr int SM_A = 0, A_BYTES = TILE_M * HID * 2 + 1024;  // activations; training: logits in its upper half
constexpr int SM_LOGITS = TILE_M * HID;                     // 66 x 128 fp32
constexpr int SM_RING = A_BYTES, SM_BIAS = SM_RING + 4 * CHUNK, SM_BAR = SM_BIAS + (HID + HID + OUT_PAD) * 4;
constexpr int MLP_SMEM = SM_BAR + 11 * 8;
static_assert(SM_LOGITS + OUT * TILE_M * 4 <= A_BYTES && SM_RING % 128 == 0 && SM_BAR % 8 == 0, "shared-memory layout");

__device__ __forceinline__ int chunk_at(int c) {
  return c < 8 ? c * CHUNK : c < 12 ? PK_W3 + (c - 8) * CHUNK3 : PK_W3T + (c - 12) * CHUNK;
}
__device__ __forceinline__ int chunk_bytes(int c) { return c >= 8 && c < 12 ? CHUNK3 : CHUNK; }

__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mma(uint32_t d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(d), "l"(da), "l"(db),
      "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(a)) | (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(b)) << 16;
}

// The weight ring, run by one thread: chunk q of this CTA (counted over its tiles) goes to
// slot q & 3 for the (q >> 2)-th time.
struct Ring {
  uint32_t slots, full, empty;  // shared addresses: slot 0, the four barriers of each kind
  const unsigned char* packed;
  int total, per_tile, issued;
  __device__ __forceinline__ void load() {  // the next chunk into its (free) slot
    const int c = issued % per_tile, slot = issued & 3, bytes = chunk_bytes(c);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + slot * 8), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     slots + slot * CHUNK),
                 "l"(packed + chunk_at(c)), "r"(bytes), "r"(full + slot * 8)
                 : "memory");
    issued++;
  }
};

// One product of the tile: D (tensor memory, `d`) = A . W^T over `chunks` chunks from chunk
// q on, N columns; the slots it frees are filled again. Run by one thread; false when a
// bounded wait gave up.
__device__ __forceinline__ bool product(Ring& ring, int& q, uint32_t a, uint32_t d, int chunks, int n, uint32_t done) {
  const uint32_t idesc = instr_desc(n), lbo_a = (TILE_M / 8) * 128, lbo_b = (uint32_t)(n / 8) * 128;
  asm volatile("tcgen05.fence::after_thread_sync;");
  for (int c = 0; c < chunks; c++) {
    const int slot = (q + c) & 3;
    if (!mbar_wait(ring.full + slot * 8, (uint32_t)((q + c) >> 2) & 1)) return false;
    for (int j = 0; j < KCHUNK / 16; j++)
      mma(d, smem_desc(a + (c * (KCHUNK / 16) + j) * 2 * lbo_a, lbo_a, 128),
          smem_desc(ring.slots + slot * CHUNK + 2 * j * lbo_b, lbo_b, 128), idesc, c > 0 || j > 0);
    commit(ring.empty + slot * 8);
  }
  commit(done);
  for (int c = 0; c < chunks; c++, q++) {
    if (ring.issued >= ring.total) continue;
    if (!mbar_wait(ring.empty + (q & 3) * 8, (uint32_t)(q >> 2) & 1)) return false;
    ring.load();
  }
  return true;
}

// Features of rows [m0, m0 + 128) in A, by threads `who` of `of`: card c of owner s is column
// 4 c + s, then strain and leader; one 16-byte vector holds the owners of two cards.
__device__ __forceinline__ void tile_features(const MlpArgs& g, int64_t m0, unsigned char* sA, int who, int of) {
  const int row = who & (TILE_M - 1);
  const int64_t r = m0 + row;
  const int64_t e = g.rows ? g.rows[r] : (r < g.n ? r : -1);
  uint64_t h[4] = {0, 0, 0, 0};
  if (e >= 0)
    for (int s = 0; s < 4; s++) h[s] = g.hands[e / 20 * 4 + s];
  const int strain = (int)(e % 20) / 4, leader = ((int)(e % 4) + 1) & 3;
  for (int kg = who / TILE_M; kg < HID / 8; kg += of / TILE_M) {
    uint64_t v[2] = {0, 0};
    if (kg < 26) {
      for (int c = 0; c < 2; c++) {
        const int bit = card_bit(2 * kg + c);
        for (int s = 0; s < 4; s++) v[c] |= (h[s] >> bit & 1) * (0x3F80ull << (16 * s));
      }
    } else if (e >= 0 && kg < 28) {
      for (int k = 0; k < 8; k++) {
        const int col = kg * 8 + k;
        if (col == 208 + strain || col == 213 + leader) v[k >> 2] |= 0x3F80ull << (16 * (k & 3));
      }
    }
    *reinterpret_cast<ulonglong2*>(sA + (kg * (TILE_M / 8) + (row >> 3)) * 128 + (row & 7) * 16) = make_ulonglong2(v[0], v[1]);
  }
}

// What bounds it: inference, the GELUs (512 erff a row; the products take a tenth of the
// time): 32 warps an SM, 0.52 ms for the rows below against 0.55 with 16. Two CTAs an SM
// with a ring of their own each, 40 or 32 KB of it, were slower (0.90, 0.60 ms: the weights
// come too late). A training step's 32 tiles use 32 SMs and are bound by one tile's chain;
// 32 warps (64 registers, a few spilled) changed nothing there. Measured, against one kernel
// per layer with its activations in HBM and its weights loaded through registers, chunk by
// chunk: the 400,000 rows of 20,000 deals 0.52 against 14.2 ms; a step of 4,096 rows with its
// gradients copied out 0.27 against 1.76 ms (5 launches against 28; the three weight gradients
// 160 us each there, two CTAs walking the whole batch).
template <bool TRAIN>
__global__ void __launch_bounds__(MLP_THREADS<TRAIN>, 1) mlp_rows(MlpArgs g) {
  constexpr int THREADS = MLP_THREADS<TRAIN>, COLS = HID / (THREADS / TILE_M);  // a thread's columns
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned char* sA = sm + SM_A;
  float* bias = reinterpret_cast<float*>(sm + SM_BIAS);
  const uint32_t bars = smem_u32(sm + SM_BAR), done = bars + 64, last = bars + 72;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + SM_BAR + 80);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int b = 0; b < 10; b++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + b * 8));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  for (int k = tid; k < HID + HID + OUT_PAD; k += THREADS)
    bias[k] = g.master[k < HID ? OFF_B1 + k : k < 2 * HID ? OFF_B2 + k - HID : OFF_B3 + k - 2 * HID];
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tslot, a_addr = smem_u32(sA);
  const int per_tile = TRAIN ? 18 : 12;
  const int block = (int)blockIdx.x, grid = (int)gridDim.x, mine = block_tiles(g.tiles, block, grid);
  Ring ring = {smem_u32(sm + SM_RING), bars, bars + 32, g.packed, mine * per_tile, per_tile, 0};
  int q = 0;  // chunks used (thread 0)
  if (tid == 0)
    for (int c = 0; c < 4 && ring.issued < ring.total; c++) ring.load();
  const int quarter = warp & 3, group = warp >> 2;  // tensor-memory lanes 32 * quarter.., columns COLS * group..
  const int row = quarter * 32 + lane;
  const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
  uint32_t phase = 0;
  bool ok = true;
  if (mine) tile_features(g, first_row(0, block, grid), sA, tid, THREADS);
  for (int t = 0; t < mine && ok; t++) {
    const int64_t m0 = first_row(t, block, grid), at = m0 + row;  // the tile's rows, this thread's
    bool good = true;
    // A is written: visible to the tensor cores; the accumulators of before are read.
    auto run = [&](int col, int chunks, int n) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncthreads();
      if (tid == 0) good = product(ring, q, a_addr, tmem + (uint32_t)col, chunks, n, done);
    };
    auto wait = [&]() {  // until the product is done; false on every thread when a wait gave up
      const bool w = mbar_wait(done, phase);
      phase ^= 1;
      ok = __syncthreads_and(w && good);
      asm volatile("tcgen05.fence::after_thread_sync;");
      return ok;
    };
    // A hidden layer's epilogue: bias and GELU to A; training keeps both, transposed.
    auto hidden = [&](int col, const float* b, float* Zt, bf16* Ht) {
      for (int c0 = group * COLS; c0 < (group + 1) * COLS; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(tmem + lanes + (uint32_t)(col + c0), r);
        uint32_t pk[8];
#pragma unroll
        for (int k = 0; k < 16; k += 2) {
          const float z0 = __uint_as_float(r[k]) + b[c0 + k], z1 = __uint_as_float(r[k + 1]) + b[c0 + k + 1];
          pk[k / 2] = pack2(gelu(z0), gelu(z1));
          if (TRAIN) {
            Zt[(size_t)(c0 + k) * g.R + at] = z0;
            Zt[(size_t)(c0 + k + 1) * g.R + at] = z1;
            Ht[(size_t)(c0 + k) * g.R + at] = __ushort_as_bfloat16((unsigned short)pk[k / 2]);
            Ht[(size_t)(c0 + k + 1) * g.R + at] = __ushort_as_bfloat16((unsigned short)(pk[k / 2] >> 16));
          }
        }
        for (int v = 0; v < 2; v++)
          *reinterpret_cast<uint4*>(sA + core_at(row, c0 + 8 * v, TILE_M)) =
              make_uint4(pk[4 * v], pk[4 * v + 1], pk[4 * v + 2], pk[4 * v + 3]);
      }
    };
    run(0, 4, HID);
    if (TRAIN) {  // the features, transposed, while the first product runs
      for (int k = warp; k < HID; k += THREADS / 32)
        for (int rr = lane; rr < TILE_M; rr += 32)
          g.Xt[(size_t)k * g.R + m0 + rr] = *reinterpret_cast<const bf16*>(sA + core_at(rr, k, TILE_M));
    }
    if (!wait()) break;
    hidden(0, bias, g.Z1t, g.H1t);
    run(256, 4, HID);
    if (!wait()) break;
    hidden(256, bias + HID, g.Z2t, g.H2t);
    run(0, 4, OUT_PAD);
    if (!wait()) break;
    if (!TRAIN) {
      if (tid < TILE_M) {  // seeds and root leads: the best trick count, the leader's best-scored card
        const int64_t e = at;
        const float* b = bias + 2 * HID;
        const uint64_t own = e < g.n ? g.hands[e / 20 * 4 + (((int)(e % 4) + 1) & 3)] : 0;
        int arg = 0, best = -1;
        float bv = 0.f, bv2 = -1e30f;
#pragma unroll
        for (int c0 = 0; c0 < OUT_PAD; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(tmem + lanes + (uint32_t)c0, r);
#pragma unroll
          for (int k = 0; k < 16; k++) {
            const int c = c0 + k;
            if (c >= OUT) continue;
            const float v = __uint_as_float(r[k]) + b[c];
            if (c == 0) {
              bv = v;
            } else if (c < OUT_T) {
              if (v > bv) {
                bv = v;
                arg = c;
              }
            } else if ((own >> card_bit(c - OUT_T) & 1) && v > bv2) {
              bv2 = v;
              best = card_bit(c - OUT_T);
            }
          }
        }
        if (e < g.n) {
          if (g.seed20) g.seed20[e] = (int8_t)arg;
          if (g.hint20) g.hint20[e] = (int8_t)best;
        }
      } else if (t + 1 < mine) {  // meanwhile the other warps make the next tile's features
        tile_features(g, first_row(t + 1, block, grid), sA, tid - TILE_M, THREADS - TILE_M);
      }
    } else {
      if (tid < TILE_M) {
        // Softmax cross-entropy of both heads: dO = (p - y) / R to A (K = 128) and, transposed,
        // to memory; the row's loss and hits to the sums.
        float* l = reinterpret_cast<float*>(sm + SM_LOGITS) + row;  // column c at l[c * TILE_M]
#pragma unroll
        for (int c0 = 0; c0 < OUT_PAD; c0 += 16) {
          uint32_t r[16];
          tmem_ld16(tmem + lanes + (uint32_t)c0, r);
#pragma unroll
          for (int k = 0; k < 16; k++)
            if (c0 + k < OUT) l[(c0 + k) * TILE_M] = __uint_as_float(r[k]) + bias[2 * HID + c0 + k];
        }
        const int64_t e = g.rows[at];
        int ns = -1, y = -1, arg = 0;
        float mx = -1e30f, sum = 0.f, mx2 = -1e30f, sum2 = 0.f, loss = 0.f;
        const float inv = 1.0f / (float)g.R;
        uint64_t own = 0;
        if (e >= 0) {
          const int64_t deal = e / 20;
          const int sd = (int)(e % 20), decl = sd % 4, tr = g.tricks20[deal * 20 + sd];
          if (tr <= 13) ns = (decl & 1) == 0 ? tr : 13 - tr;
          own = g.hands[deal * 4 + ((decl + 1) & 3)];
          const int best = g.best20[deal * 20 + sd];
          if (ns >= 0 && best >= 0 && (own >> best & 1)) y = card_index(best);
        }
        if (ns >= 0) {
          for (int c = 0; c < OUT_T; c++) mx = fmaxf(mx, l[c * TILE_M]);
          for (int c = 0; c < OUT_T; c++) {
            sum += expf(l[c * TILE_M] - mx);
            if (l[c * TILE_M] > l[arg * TILE_M]) arg = c;
          }
          loss = -(l[ns * TILE_M] - mx - logf(sum));
        }
        if (y >= 0) {
          for (int c = 0; c < OUT_M; c++)
            if (own >> card_bit(c) & 1) mx2 = fmaxf(mx2, l[(OUT_T + c) * TILE_M]);
          for (int c = 0; c < OUT_M; c++)
            if (own >> card_bit(c) & 1) sum2 += expf(l[(OUT_T + c) * TILE_M] - mx2);
          loss += -(l[(OUT_T + y) * TILE_M] - mx2 - logf(sum2));
        }
        for (int c0 = 0; c0 < DO_LD; c0 += 8) {
          uint32_t pk[4];
          for (int k = 0; k < 8; k += 2) {
            float d[2] = {0.f, 0.f};
            for (int h = 0; h < 2; h++) {
              const int c = c0 + k + h;
              if (c < OUT_T) {
                if (ns >= 0) d[h] = (expf(l[c * TILE_M] - mx) / sum - (c == ns ? 1.f : 0.f)) * inv;
              } else if (c < OUT && y >= 0 && (own >> card_bit(c - OUT_T) & 1)) {
                d[h] = (expf(l[c * TILE_M] - mx2) / sum2 - (c - OUT_T == y ? 1.f : 0.f)) * inv;
              }
            }
            pk[k / 2] = pack2(d[0], d[1]);
            g.dOt[(size_t)(c0 + k) * g.R + at] = __ushort_as_bfloat16((unsigned short)pk[k / 2]);
            g.dOt[(size_t)(c0 + k + 1) * g.R + at] = __ushort_as_bfloat16((unsigned short)(pk[k / 2] >> 16));
          }
          *reinterpret_cast<uint4*>(sA + core_at(row, c0, TILE_M)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
        float s0 = loss * inv, s1 = ns >= 0 && arg == ns ? 1.f : 0.f, s2 = ns >= 0 ? 1.f : 0.f;
        for (int d = 16; d; d >>= 1) {
          s0 += __shfl_down_sync(0xFFFFFFFFu, s0, d);
          s1 += __shfl_down_sync(0xFFFFFFFFu, s1, d);
          s2 += __shfl_down_sync(0xFFFFFFFFu, s2, d);
        }
        if (lane == 0) {
          atomicAdd(g.acc + 0, s0);
          atomicAdd(g.acc + 1, s1);
          atomicAdd(g.acc + 2, s2);
        }
      }
      // dH2 = dO . W3, dH1 = dZ2 . W2, each times GELU' of the layer's pre-activation (which
      // this thread wrote).
      for (int layer = 0; layer < 2; layer++) {
        const int col = layer == 0 ? 256 : 0;
        run(col, layer == 0 ? 2 : 4, HID);
        if (!wait()) break;
        const float* Zt = layer == 0 ? g.Z2t : g.Z1t;
        bf16* dZt = layer == 0 ? g.dZ2t : g.dZ1t;
        for (int c0 = group * COLS; c0 < (group + 1) * COLS; c0 += 16) {
          uint32_t r[16], pk[8];
          tmem_ld16(tmem + lanes + (uint32_t)(col + c0), r);
#pragma unroll
          for (int k = 0; k < 16; k += 2) {
            const size_t o = (size_t)(c0 + k) * g.R + at;
            pk[k / 2] = pack2(__uint_as_float(r[k]) * gelu_grad(Zt[o]), __uint_as_float(r[k + 1]) * gelu_grad(Zt[o + g.R]));
            dZt[o] = __ushort_as_bfloat16((unsigned short)pk[k / 2]);
            dZt[o + g.R] = __ushort_as_bfloat16((unsigned short)(pk[k / 2] >> 16));
          }
          if (layer == 0)
            for (int v = 0; v < 2; v++)
              *reinterpret_cast<uint4*>(sA + core_at(row, c0 + 8 * v, TILE_M)) =
                  make_uint4(pk[4 * v], pk[4 * v + 1], pk[4 * v + 2], pk[4 * v + 3]);
        }
      }
      if (!ok) break;
      if (t + 1 < mine) {
        __syncthreads();
        tile_features(g, first_row(t + 1, block, grid), sA, tid, THREADS);
      }
    }
  }
  if (!ok && tid == 0) {
    // A wait gave up: the copies in flight land before their shared memory goes, the products
    // before their tensor memory does (bounded).
    atomicExch(g.err, 1);
    for (int c = q; c < ring.issued; c++) mbar_wait(ring.full + (c & 3) * 8, (uint32_t)(c >> 2) & 1);
    commit(last);
    mbar_wait(last, 0);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// ---- weight gradients --------------------------------------------------------------------

// dW = dY^T . X over the batch, split along it: CTA (x, y) makes rows 128 x' of one of the
// three gradients from batch rows [y * ks, (y + 1) * ks). Operands are the transposed
// outputs of mlp_rows (K = batch, contiguous). Part (y, x) is 128 x 256 fp32.
struct DwArgs {
  const bf16 *dZ1t, *Xt, *dZ2t, *H1t, *dOt, *H2t;
  int R, ks;
  float* part;
  int* err;
};
constexpr int DW_K = 128, DW_TILES = 5, DW_THREADS = 256;
constexpr int DW_SMEM = (TILE_M + HID) * DW_K * 2 + 16;

// What bounds it: the loads' latency (one 128-deep slice a CTA at 4,096 rows); unsplit, two
// CTAs walked 64 slices each, 160 us a product.
__global__ void __launch_bounds__(DW_THREADS, 2) gemm_dw(DwArgs g) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, x = blockIdx.x;
  const bf16* A = (x < 2 ? g.dZ1t + (size_t)x * TILE_M * g.R : x < 4 ? g.dZ2t + (size_t)(x - 2) * TILE_M * g.R : g.dOt);
  const bf16* B = x < 2 ? g.Xt : x < 4 ? g.H1t : g.H2t;
  unsigned char *sA = sm, *sB = sm + TILE_M * DW_K * 2;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + (TILE_M + HID) * DW_K * 2);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  const uint32_t bar_a = smem_u32(bar);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(256));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar_a));
    asm volatile("fence.mbarrier_init.release.cluster;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tslot, lbo_a = (TILE_M / 8) * 128, lbo_b = (HID / 8) * 128, idesc = instr_desc(HID);
  const int k_begin = (int)blockIdx.y * g.ks, k_end = k_begin + g.ks < g.R ? k_begin + g.ks : g.R;
  bool ok = true;
  uint32_t phase = 0;
  for (int k0 = k_begin; k0 < k_end && ok; k0 += DW_K) {
    for (int v = tid; v < (TILE_M + HID) * (DW_K / 8); v += DW_THREADS) {
      const int kg = v % (DW_K / 8), r = v / (DW_K / 8);  // 16 threads read 256 bytes of a row
      const bool in_a = r < TILE_M;
      const uint4 w = *reinterpret_cast<const uint4*>((in_a ? A + (size_t)r * g.R : B + (size_t)(r - TILE_M) * g.R) + k0 + kg * 8);
      *reinterpret_cast<uint4*>(in_a ? sA + core_at(r, kg * 8, TILE_M) : sB + core_at(r - TILE_M, kg * 8, HID)) = w;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      for (int j = 0; j < DW_K / 16; j++)
        mma(tmem, smem_desc(smem_u32(sA) + 2 * j * lbo_a, lbo_a, 128), smem_desc(smem_u32(sB) + 2 * j * lbo_b, lbo_b, 128),
            idesc, k0 > k_begin || j > 0);
      commit(bar_a);
    }
    ok = __syncthreads_and(mbar_wait(bar_a, phase));
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (!ok) {  // give the products in flight one more bounded wait before TMEM is freed
      mbar_wait(bar_a, phase);
      __syncthreads();
    }
    phase ^= 1;
  }
  if (!ok) {
    if (tid == 0) atomicExch(g.err, 1);
  } else {
    const int row = (warp & 3) * 32 + lane, half = (warp >> 2) * 128;
    float* out = g.part + ((size_t)blockIdx.y * DW_TILES + x) * (TILE_M * HID) + (size_t)row * HID;
    for (int c0 = half; c0 < half + 128; c0 += 16) {
      uint32_t r[16];
      tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, r);
      for (int k = 0; k < 16; k += 4) *reinterpret_cast<uint4*>(out + c0 + k) = make_uint4(r[k], r[k + 1], r[k + 2], r[k + 3]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256));
}

// A weight's bf16 copies in the tensor cores' layout.
__device__ __forceinline__ void pack_param(int64_t i, float v, unsigned char* packed) {
  const unsigned short x = __bfloat16_as_ushort(__float2bfloat16_rn(v));
  auto put = [&](int base, int n, int k, int rows) {
    *reinterpret_cast<unsigned short*>(packed + base + core_at(n, k, rows)) = x;
  };
  if (i < OFF_B1) {
    put(PK_W1, (int)(i / IN_PAD), (int)(i % IN_PAD), HID);
  } else if (i >= OFF_W2 && i < OFF_B2) {
    const int n = (int)((i - OFF_W2) / HID), k = (int)((i - OFF_W2) % HID);
    put(PK_W2, n, k, HID);
    put(PK_W2T, k, n, HID);
  } else if (i >= OFF_W3 && i < OFF_B3) {
    const int n = (int)((i - OFF_W3) / HID), k = (int)((i - OFF_W3) % HID);
    put(PK_W3, n, k, OUT_PAD);
    put(PK_W3T, k, n, HID);
  }
}
__global__ void pack_params(const float* master, unsigned char* packed) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N_PARAMS) pack_param(i, master[i], packed);
}

// The gradients from their parts (weights: the splits in order; biases: a warp sums a row of
// dY^T), and Adam on the fp32 master parameters when lr > 0, with the bf16 copies renewed.
struct FinishArgs {
  const float* part;
  int splits, R;
  const bf16 *dZ1t, *dZ2t, *dOt;
  float *grad, *master, *m, *v;
  unsigned char* packed;
  float lr, c1, c2;
};
__device__ __forceinline__ void finish_param(const FinishArgs& a, int64_t i, float gi) {
  a.grad[i] = gi;
  if (!(a.lr > 0)) return;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float m = b1 * a.m[i] + (1.f - b1) * gi, v = b2 * a.v[i] + (1.f - b2) * gi * gi;
  a.m[i] = m;
  a.v[i] = v;
  const float p = a.master[i] - a.lr * (m / a.c1) / (sqrtf(v / a.c2) + eps);
  a.master[i] = p;
  pack_param(i, p, a.packed);
}
constexpr int N_BIAS = HID + HID + OUT_PAD, N_WEIGHT = HID * IN_PAD + HID * HID + OUT_PAD * HID, FIN_THREADS = 256;
constexpr int FIN_BLOCKS_W = N_WEIGHT / FIN_THREADS, FIN_BLOCKS = FIN_BLOCKS_W + (N_BIAS + FIN_THREADS / 32 - 1) / (FIN_THREADS / 32);
static_assert(N_WEIGHT % FIN_THREADS == 0, "a block is all weights or all biases");
__global__ void dw_finish(FinishArgs a) {
  if (blockIdx.x < FIN_BLOCKS_W) {
    const int w = blockIdx.x * FIN_THREADS + threadIdx.x;  // 256 columns a row: rows 0..255 W1, ..511 W2, then W3
    const float* p = a.part + w;
    float s = 0.f;
#pragma unroll 8
    for (int k = 0; k < a.splits; k++) s += p[(size_t)k * DW_TILES * TILE_M * HID];
    const int r = w >> 8;
    finish_param(a, w + (r < HID ? 0 : r < 2 * HID ? OFF_W2 - (int64_t)HID * IN_PAD : OFF_W3 - (int64_t)2 * HID * HID), s);
    return;
  }
  const int b = (blockIdx.x - FIN_BLOCKS_W) * (FIN_THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= N_BIAS) return;
  const bf16* row = b < HID ? a.dZ1t + (size_t)b * a.R : b < 2 * HID ? a.dZ2t + (size_t)(b - HID) * a.R : a.dOt + (size_t)(b - 2 * HID) * a.R;
  float s = 0.f;
  for (int k = lane * 8; k < a.R; k += 256) {
    const uint4 x = *reinterpret_cast<const uint4*>(row + k);
    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
    for (int q = 0; q < 4; q++) s += __uint_as_float(w[q] << 16) + __uint_as_float(w[q] & 0xFFFF0000u);
  }
  for (int d = 16; d; d >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, d);
  if (lane == 0) finish_param(a, b < HID ? OFF_B1 + b : b < 2 * HID ? OFF_B2 + b - HID : OFF_B3 + b - 2 * HID, s);
}

}  // namespace guide_nn
