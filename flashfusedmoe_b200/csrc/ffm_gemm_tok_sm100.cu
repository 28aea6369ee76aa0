// The two projections of a decode-sized call: out[token, feature] = x[token, :] . W[feature, :] with a handful of tokens
// per expert, the shared expert as one more group of the same launch.
//
// Such a call streams the weights of the experts that were hit; everything else should cost nothing. The weights are the
// M operand (128 features per CTA), the tokens of one expert the N operand (up to 64), so a tile loads, computes and stores
// only the 4-, 16- and 8-token boxes that hold tokens. With the tokens on the M side (ffm_gemm_sm100.cu) every tile loads
// a 128-row box of mostly unused rows beside 256 rows of weights, and stores one.
// Measured, 48 tokens on 64 experts, top-6, K = 2048, H = 1408 (0.74 + 0.37 GB of weights): up + GLU 131 -> 121 us, down 75 ->
// 64 us with loads issued under `lane == 0`; with an elected thread the whole call went from 214 to 205 us. 128 tokens on 256
// experts, D = 7168, H = 2048: 2110 + 1070 us (7.0 and 6.9 TB/s, what a plain read of such tiles reaches) against 2365 + 1182.
// The up-projection can gather the token rows itself (TMA gather4, four rows per instruction), which saves the permute
// launch and costs about as much where experts have several rows (48 tokens on 64 experts and a shared one, whole call, replayed:
// 201 us with the permute, 197 without).
//
//   warp 0      TMA producer          warp 1   MMA issuer, TMEM owner
//   warps 2..9  epilogue: two groups of four warps (one per TMEM lane quarter) take the 32-token steps of a tile in turn
//
// Ring of 8 stages (16 KiB of weights + up to 8 KiB of tokens): 128 KiB of weights in flight per SM. Fewer stages were
// slower (8: 121 / 64 us, 6: 122 / 65, 4: 132 / 71, with loads issued under `lane == 0`); stages twice as deep (128 rows x 256 bytes in one box, four of them) take the same
// time within 1 %. As in the other GEMM: fp32 accumulators in TMEM, two of them, persistent CTAs,
// bounded waits, TMA stores.
//
// The accumulator has features on TMEM lanes and tokens on columns, so the epilogue transposes: tcgen05.ld.16x256b hands
// a warp 16 features x 8 tokens per four registers in the register layout of an 8x8 matrix fragment, and
// stmatrix.trans writes it token-major into a staged box of 32 tokens x 64 features (128-byte swizzle) that TMA stores.
// GLU: the gate and up rows of a weight tile are staged interleaved by 16 (one 5-D tensor map), so that lanes 0..15 of a
// quarter hold 16 gate features and lanes 16..31 the same up features: the activation stays inside a thread.
#include "ffm_gemm_common.cuh"
#include "ffm_internal.h"

namespace ffm {

namespace {

constexpr int BK = 64;  // K elements per stage row (128 bytes)
constexpr int UMMA_K = 16;
constexpr int NUM_ACC = 2;
constexpr int NMAX = 64;  // tokens per tile
constexpr int MAX_GROUPS = 256;
constexpr int THREADS = 320;
constexpr int EPI_GROUPS = 2;  // epilogue groups of four warps
constexpr int EPI_WARPS = 4 * EPI_GROUPS;
constexpr int STEP_TOKENS = 32;
constexpr int STORE_ROWS = 8;        // tokens per stored box
constexpr int BOX_BYTES = 32 * 128;  // 32 tokens x 64 features
constexpr int A_BYTES = 128 * 128;   // 128 weight rows x 64 K
constexpr int STAGE_BYTES = A_BYTES + NMAX * 128;
constexpr int STAGES = 8;
constexpr int RING_BYTES = STAGES * STAGE_BYTES;
constexpr int CTRL_BYTES = 4096;
constexpr int TMEM_COLS = NUM_ACC * NMAX;

enum { EPI_PLAIN = 0, EPI_GLU = 1 };  // down-projection, up-projection

template <int EPI>
struct Shape {
  static constexpr int FEATS = EPI == EPI_GLU ? 64 : 128;  // output features per tile
  static constexpr int STEP_BYTES = FEATS / 64 * BOX_BYTES;
  static constexpr int SMEM_BYTES = RING_BYTES + EPI_GROUPS * STEP_BYTES + CTRL_BYTES + 1024;  // + alignment slack
  static_assert(SMEM_BYTES <= 232448, "tile shape does not fit in shared memory");
};

// Index 1 of the pairs: the shared expert (rows 0 .. tokens - 1), present when feats[1] > 0.
struct TokParams {
  const int32_t* tile_start;  // [groups + 1] first 128-row tile of every group
  const int32_t* counts;      // [groups] rows of every group
  const int32_t* src;         // up: [rows] flat slot of a grouped row, or null: the rows lie grouped
  int groups;
  int top_k;
  int tokens;
  int k_blocks[2];   // 64-deep K blocks
  int feats[2];      // output features per group
  int swap_gate[2];  // up: the interleaved weight map holds up rows before gate rows
  int act[2];
  int32_t* status;
  long long wait_cycles;
};

struct Ctrl {
  unsigned long long full_bar[STAGES];
  unsigned long long empty_bar[STAGES];
  unsigned long long acc_full_bar[NUM_ACC];
  unsigned long long acc_empty_bar[NUM_ACC];
  unsigned long long drain_bar;  // after an abort: the MMAs in flight
  uint32_t tmem_base;
  int abort_flag;
  int filled;                 // stages the producer has filled in all
  int4 token[NMAX / 4];       // up: token rows of the producer's tile
  int base[MAX_GROUPS];       // first row of a group
  int count[MAX_GROUPS];      // rows of a group
  int items[MAX_GROUPS + 1];  // routed tiles before a group
};
static_assert(sizeof(Ctrl) <= CTRL_BYTES, "control block too large");

struct Tile {
  int group;
  int shared;  // 1: a tile of the shared expert
  int f_tile;
  int row0;    // first token row (grouped, or of the tokens)
  int tokens;  // valid tokens of this tile, 1..NMAX
};

// Tiles in launch order: the shared expert's, then by expert and feature tile, token tile fastest (the token tiles of an
// expert share its weights through L2). CTA c takes tile G - 1 - c first and then c + G, c + 2 G, ...: the shared expert's
// tiles, often the longest, go to the CTAs that have no tile in a partly filled last round.
struct Walker {
  const Ctrl* c;
  int groups, shared_tiles, shared_nt, tokens, cur, round, g, total;

  __device__ Walker(const Ctrl* ctrl, const TokParams& p, int feats_per_tile) {
    c = ctrl;
    groups = p.groups;
    tokens = p.tokens;
    shared_nt = token_tiles(tokens);
    shared_tiles = shared_nt * ((p.feats[1] + feats_per_tile - 1) / feats_per_tile);
    cur = gridDim.x - 1 - blockIdx.x;
    round = 0;
    g = 0;
    total = shared_tiles + (groups > 0 ? ctrl->items[groups] : 0);
  }
  __device__ static int token_tiles(int count) { return (count + NMAX - 1) / NMAX; }
  __device__ bool next(Tile& t) {
    if (cur >= total) return false;
    if (cur < shared_tiles) {
      const int first = (cur % shared_nt) * NMAX;
      t.group = 0;
      t.shared = 1;
      t.f_tile = cur / shared_nt;
      t.row0 = first;
      t.tokens = min(NMAX, tokens - first);
    } else {
      const int i = cur - shared_tiles;
      while (g < groups - 1 && i >= c->items[g + 1]) ++g;
      const int nt = token_tiles(c->count[g]);
      const int r = i - c->items[g];
      const int first = (r % nt) * NMAX;
      t.group = g;
      t.shared = 0;
      t.f_tile = r / nt;
      t.row0 = c->base[g] + first;
      t.tokens = min(NMAX, c->count[g] - first);
    }
    ++round;
    cur = round * gridDim.x + blockIdx.x;
    return true;
  }
};

// ---- PTX used only by this kernel --------------------------------------------------------------

// 16 lanes x 16 consecutive 32-bit columns in the 8x8-fragment layout: r[4 i + 0, 1] = lane / 4, columns 8 i +
// 2 (lane % 4) + 0, 1; r[4 i + 2, 3] = the same columns of lane / 4 + 8.
__device__ __forceinline__ void tmem_ld_16x256_x2(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

__device__ __forceinline__ void stmatrix_x4_trans(uint32_t addr, const uint32_t (&m)[4]) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(m[0]), "r"(m[1]),
               "r"(m[2]), "r"(m[3])
               : "memory");
}

// barrier of one epilogue group (128 threads); the second form returns whether every thread passed ok
__device__ __forceinline__ void group_sync(int id) { asm volatile("barrier.cta.sync %0, 128;" ::"r"(id) : "memory"); }
__device__ __forceinline__ bool group_all(int id, bool ok) {
  uint32_t r;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 q, %1, 0;\n"
      "barrier.cta.red.and.pred p, %2, 128, q;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(r)
      : "r"(ok ? 1u : 0u), "r"(id)
      : "memory");
  return r != 0;
}

// four rows y (any order) x 64 columns from x, stored as consecutive rows; the map's box is one row high
__device__ __forceinline__ void tma_gather4(uint32_t dst, const void* map, uint32_t bar, int x, const int4& y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(dst),
      "l"(map), "r"(bar), "r"(x), "r"(y.x), "r"(y.y), "r"(y.z), "r"(y.w)
      : "memory");
}

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const void* map, uint32_t bar, int c0, int c3, int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(0), "r"(c3), "r"(c4)
      : "memory");
}

// One 32-token step of the GLU epilogue for this warp's 16 features: gate and up accumulators are rounded to bf16 (as
// stored pre-activations would be), the activation is computed from the rounded values. `off` is the lane's offset in the
// box for token half 0 (stmatrix address); the other half lies 16 rows (2 KiB) further, under the same swizzle.
template <int ACT>
__device__ __forceinline__ void glu_step(uint32_t tcol, uint32_t box, uint32_t off, bool swap) {
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    uint32_t a[8], b[8], pa[4];
    tmem_ld_16x256_x2(tcol + half * 16, a);
    tmem_ld_16x256_x2(tcol + (16u << 16) + half * 16, b);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = unpack_bf16x2(pack_bf16x2(__uint_as_float(a[2 * i]), __uint_as_float(a[2 * i + 1])));
      const float2 y = unpack_bf16x2(pack_bf16x2(__uint_as_float(b[2 * i]), __uint_as_float(b[2 * i + 1])));
      const float2 g = swap ? y : x, u = swap ? x : y;
      pa[i] = pack_bf16x2(glu_fwd(ACT, g.x, u.x), glu_fwd(ACT, g.y, u.y));
    }
    stmatrix_x4_trans(box + off + half * 2048, pa);
  }
}

template <int EPI>
__global__ void __launch_bounds__(THREADS, 1)
ffm_gemm_tok_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmA1,
                    const __grid_constant__ CUtensorMap tmB1, const __grid_constant__ CUtensorMap tmC1,
                    const __grid_constant__ TokParams p) {
  using S = Shape<EPI>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
  uint8_t* smem = smem_raw + pad;
  const uint32_t smem_base = raw_addr + pad;
  const uint32_t stg_base = smem_base + RING_BYTES;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem + RING_BYTES + EPI_GROUPS * S::STEP_BYTES);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int f_tiles = (p.feats[0] + S::FEATS - 1) / S::FEATS;

  // ---- set-up ------------------------------------------------------------------------------
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&ctrl->full_bar[s]), 1);
      mbar_init(smem_u32(&ctrl->empty_bar[s]), 1);
    }
    for (int a = 0; a < NUM_ACC; ++a) {
      mbar_init(smem_u32(&ctrl->acc_full_bar[a]), 1);
      mbar_init(smem_u32(&ctrl->acc_empty_bar[a]), EPI_WARPS);
    }
    mbar_init(smem_u32(&ctrl->drain_bar), 1);
    ctrl->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
  }
  if (warp == 2) {
    // tiles before every group: eight consecutive groups per lane
    constexpr int PER = MAX_GROUPS / 32;
    int mine[PER];
    int sum = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int g = lane * PER + i;
      mine[i] = 0;
      if (g < p.groups) {
        const int cnt = __ldg(p.counts + g);
        ctrl->count[g] = cnt;
        ctrl->base[g] = __ldg(p.tile_start + g) * 128;
        mine[i] = Walker::token_tiles(cnt) * f_tiles;
      }
      sum += mine[i];
    }
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += t;
    }
    int run = incl - sum;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int g = lane * PER + i;
      if (g < p.groups) ctrl->items[g] = run;
      run += mine[i];
      if (g + 1 == p.groups) ctrl->items[p.groups] = run;
    }
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ctrl->tmem_base), TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  const uint32_t tmem_base = ctrl->tmem_base;
  volatile int* abort_flag = &ctrl->abort_flag;
  bool issuer = false;  // the thread that issues the MMAs
  Walker walker(ctrl, p, S::FEATS);
  Tile t;

  // ---- roles -------------------------------------------------------------------------------
  if (warp == 0) {
    // ================= TMA producer =================
    int stage = 0;
    uint32_t phase = 0;
    int filled = 0;
    bool ok = true;
    const bool producer = elect_one();
    const int producer_lane = __ffs(__ballot_sync(0xffffffffu, producer)) - 1;
    while (ok && walker.next(t)) {
      const int f0 = t.f_tile * S::FEATS;
      const CUtensorMap* mA = t.shared ? &tmA1 : &tmA;
      const CUtensorMap* mB = t.shared ? &tmB1 : &tmB;
      const int k_blocks = p.k_blocks[t.shared];
      // token rows staged: gathered in fours (the last four repeat the last token), or in boxes of 16
      const bool gather = EPI == EPI_GLU && p.src != nullptr && !t.shared;
      const int nb = gather ? (t.tokens + 3) & ~3 : (t.tokens + 15) & ~15;
      if (gather) {
        for (int i = lane; i < nb; i += 32) {
          reinterpret_cast<int*>(ctrl->token)[i] = __ldg(p.src + t.row0 + min(i, t.tokens - 1)) / p.top_k;
        }
        __syncwarp();
      }
      if (producer) {
        for (int kb = 0; kb < k_blocks; ++kb) {
          ok = mbar_wait_bounded(smem_u32(&ctrl->empty_bar[stage]), phase ^ 1u, abort_flag, p.status,
                                 FFM_STATUS_WAIT_PRODUCER, p.wait_cycles);
          if (!ok) break;
          const uint32_t full = smem_u32(&ctrl->full_bar[stage]);
          const uint32_t a_dst = smem_base + stage * STAGE_BYTES;
          const uint32_t b_dst = a_dst + A_BYTES;
          mbar_expect_tx(full, A_BYTES + nb * 128);
          const int k0 = kb * BK;
          if (EPI == EPI_GLU) {
            tma_load_5d(a_dst, mA, full, k0, f0 / 16, t.group);
          } else {
            tma_load_2d(a_dst, mA, full, k0, t.group * p.feats[0] + f0);
          }
          if (gather) {
            for (int r = 0; r < nb; r += 4) tma_gather4(b_dst + r * 128, mB, full, k0, ctrl->token[r >> 2]);
          } else {
            for (int r = 0; r < nb; r += 16) tma_load_2d(b_dst + r * 128, mB, full, k0, t.row0 + r);
          }
          ++filled;
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      // also: the token list is overwritten only after its last use
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, producer_lane) != 0;
    }
    if (producer) ctrl->filled = filled;
  } else if (warp == 1) {
    // ================= MMA issuer =================
    if (elect_one()) {
      issuer = true;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      while (ok && walker.next(t)) {
        const uint32_t idesc = make_idesc_bf16(128, (t.tokens + 15) & ~15, 0, 0);
        ok = mbar_wait_bounded(smem_u32(&ctrl->acc_empty_bar[acc]), acc_phase ^ 1u, abort_flag, p.status,
                               FFM_STATUS_WAIT_MMA, p.wait_cycles);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * NMAX;
        const int k_blocks = p.k_blocks[t.shared];
        for (int kb = 0; kb < k_blocks; ++kb) {
          ok = mbar_wait_bounded(smem_u32(&ctrl->full_bar[stage]), phase, abort_flag, p.status, FFM_STATUS_WAIT_MMA,
                                 p.wait_cycles);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_src = smem_base + stage * STAGE_BYTES;
          const uint32_t b_src = a_src + A_BYTES;
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {
            umma_bf16(d_tmem, make_smem_desc_sw128(a_src + kk * 32, 16, 1024),
                      make_smem_desc_sw128(b_src + kk * 32, 16, 1024), idesc, (kb > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(smem_u32(&ctrl->empty_bar[stage]));
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (!ok) break;
        umma_commit(smem_u32(&ctrl->acc_full_bar[acc]));
        if (++acc == NUM_ACC) {
          acc = 0;
          acc_phase ^= 1u;
        }
      }
    }
  } else {
    // ================= epilogue (warps 2..9) =================
    const int quarter = warp & 3;     // TMEM lanes [32 * quarter, 32 * quarter + 32)
    const int grp = (warp - 2) >> 2;  // takes the 32-token step grp of a tile
    const bool storer = ((warp - 2) & 3) == 0 && lane == 0;  // issues the group's bulk stores
    const int bar_id = 1 + grp;
    const uint32_t buf = stg_base + grp * S::STEP_BYTES;
    // the lane's row and 16-byte chunk when the warp writes four 8x8 blocks (matrix m = lane / 8): token
    // 8 (m / 2) + lane % 8, chunk m % 2 after the warp's first chunk
    const int m_row = ((lane >> 4) << 3) + (lane & 7);
    const int m_chunk = (lane >> 3) & 1;
    const int c0 = grp * STEP_TOKENS;
    int acc = 0;
    uint32_t acc_phase = 0;
    while (walker.next(t)) {
      const int f0 = t.f_tile * S::FEATS;
      const bool ok = mbar_wait_bounded(smem_u32(&ctrl->acc_full_bar[acc]), acc_phase, abort_flag, p.status,
                                        FFM_STATUS_WAIT_EPILOGUE, p.wait_cycles);
      // the staging buffer is free once the group's last store has read it; all four warps go on or none does
      if (storer) bulk_wait_read<0>();
      if (!group_all(bar_id, ok)) break;
      tc_fence_after();
      if (c0 < t.tokens) {
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * NMAX + c0;
        if (EPI == EPI_GLU) {
          const uint32_t o = box_offset(m_row, quarter * 2 + m_chunk);
          const bool swap = p.swap_gate[t.shared] != 0;
          switch (p.act[t.shared]) {
            case FFM_ACT_SWIGLU: glu_step<FFM_ACT_SWIGLU>(taddr, buf, o, swap); break;
            case FFM_ACT_GEGLU_TANH: glu_step<FFM_ACT_GEGLU_TANH>(taddr, buf, o, swap); break;
            case FFM_ACT_RELU2: glu_step<FFM_ACT_RELU2>(taddr, buf, o, swap); break;
            default: glu_step<FFM_ACT_GEGLU_ERF>(taddr, buf, o, swap); break;
          }
        } else {
          uint32_t v[4][8];  // 2 x token half + feature half
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            tmem_ld_16x256_x2(taddr + (static_cast<uint32_t>(16 * (h & 1)) << 16) + 16 * (h >> 1), v[h]);
          }
          tmem_ld_wait();
          const uint32_t box = buf + (quarter >> 1) * BOX_BYTES;
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            uint32_t m[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              m[i] = pack_bf16x2(__uint_as_float(v[h][2 * i]), __uint_as_float(v[h][2 * i + 1]));
            }
            const int ch = (quarter & 1) * 4 + 2 * (h & 1) + m_chunk;
            stmatrix_x4_trans(box + box_offset(m_row, ch) + (h >> 1) * 2048, m);
          }
        }
        fence_proxy_async();
        group_sync(bar_id);
        if (storer) {
          const int rows = min(STEP_TOKENS, t.tokens - c0);
          const CUtensorMap* mC = t.shared ? &tmC1 : &tmC;
          for (int r = 0; r < rows; r += STORE_ROWS) {
            tma_store_3d(mC, buf + r * 128, f0, t.row0 + c0 + r, 0);
            if (EPI == EPI_PLAIN && f0 + 64 < p.feats[t.shared]) {
              tma_store_3d(mC, buf + BOX_BYTES + r * 128, f0 + 64, t.row0 + c0 + r, 0);
            }
          }
          bulk_commit();
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->acc_empty_bar[acc]));
      if (++acc == NUM_ACC) {
        acc = 0;
        acc_phase ^= 1u;
      }
    }
    if (storer) bulk_wait0();  // its bulk stores have landed before the CTA's shared memory goes away
  }

  // ---- common exit: every role reaches this point, also after an abort ----------------------
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    // loads and MMAs that nobody waited for must not land in shared memory or TMEM that the CTA has given back
    if (threadIdx.x == 0) {
      for (int f = max(ctrl->filled - STAGES, 0); f < ctrl->filled; ++f) {
        mbar_drain(smem_u32(&ctrl->full_bar[f % STAGES]), (f / STAGES) & 1);
      }
    } else if (issuer) {
      umma_commit(smem_u32(&ctrl->drain_bar));
      mbar_drain(smem_u32(&ctrl->drain_bar), 0);
    }
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---- host side ---------------------------------------------------------------------------------

// 3-D bf16 output map over [rows, cols] (row-major), 128-byte swizzle, box {64, STORE_ROWS, 1}.
int make_store_map(CUtensorMap* map, const void* base, long long rows, long long cols) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return FFM_ERR_NO_DRIVER;
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0 || (cols * 2) % 16 != 0) return FFM_ERR_UNSUPPORTED;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), 1};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols) * 2, static_cast<cuuint64_t>(cols) * rows * 2};
  cuuint32_t box[3] = {64, STORE_ROWS, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FFM_OK : FFM_ERR_LAUNCH;
}

// 5-D map {K, 16 rows, gate / up, H / 16, groups}: a box {64, 16, 2, 4, 1} is a 128-row weight tile with gate and up rows
// interleaved by 16. `lo` is the matrix at the lower address, `gap` the bytes to the other.
int make_glu_weight_map(CUtensorMap* map, const void* lo, long long gap, int K, int H, int groups, long long group_bytes) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return FFM_ERR_NO_DRIVER;
  const long long row = static_cast<long long>(K) * 2;
  if ((reinterpret_cast<uintptr_t>(lo) & 15u) != 0) return FFM_ERR_UNSUPPORTED;
  cuuint64_t dims[5] = {static_cast<cuuint64_t>(K), 16, 2, static_cast<cuuint64_t>(H / 16),
                        static_cast<cuuint64_t>(groups)};
  cuuint64_t strides[4] = {static_cast<cuuint64_t>(row), static_cast<cuuint64_t>(gap), static_cast<cuuint64_t>(row * 16),
                           static_cast<cuuint64_t>(group_bytes)};
  cuuint32_t box[5] = {64, 16, 2, 4, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(lo), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? FFM_OK : FFM_ERR_LAUNCH;
}

template <int EPI>
int launch_tok(const CUtensorMap (&m)[6], const TokParams& p, long long rows, cudaStream_t stream) {
  using S = Shape<EPI>;
  static PerDevice ready;
  auto kernel = ffm_gemm_tok_kernel<EPI>;
  const bool ok = ready.get([&] {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM_BYTES) == cudaSuccess) return 1;
    cudaGetLastError();
    return 0;
  }) > 0;
  if (!ok) return FFM_ERR_LAUNCH;
  // no more CTAs than there can be tiles: every group may end in a partly filled token tile, and every routed row may be
  // alone in its group
  long long tiles = rows / NMAX + p.groups;
  if (tiles > static_cast<long long>(p.tokens) * p.top_k) tiles = static_cast<long long>(p.tokens) * p.top_k;
  long long ctas = tiles * ((p.feats[0] + S::FEATS - 1) / S::FEATS) +
                   (p.tokens + NMAX - 1) / NMAX * ((p.feats[1] + S::FEATS - 1) / S::FEATS);
  if (ctas > num_sms()) ctas = num_sms();
  kernel<<<static_cast<unsigned>(ctas), THREADS, S::SMEM_BYTES, stream>>>(m[0], m[1], m[2], m[3], m[4], m[5], p);
  return cudaGetLastError() == cudaSuccess ? FFM_OK : FFM_ERR_LAUNCH;
}

// the maps of an absent part are never used, but the kernel prefetches their descriptors
void fill_missing(CUtensorMap (&m)[6], bool routed, bool shared) {
  for (int i = 0; i < 3; ++i) {
    if (!routed) m[i] = m[i + 3];
    if (!shared) m[i + 3] = m[i];
  }
}

// weight map, output map and parameters of one GLU (routed or shared) of the up-projection
int up_side(CUtensorMap* tmA, CUtensorMap* tmC, TokParams* p, int i, const void* w_gate, const void* w_up, int groups,
            long long group_bytes, int D, int H, int activation, void* act, long long rows) {
  const uint8_t* g = static_cast<const uint8_t*>(w_gate);
  const uint8_t* u = static_cast<const uint8_t*>(w_up);
  const bool up_low = reinterpret_cast<uintptr_t>(u) < reinterpret_cast<uintptr_t>(g);
  const long long gap = static_cast<long long>(up_low ? reinterpret_cast<uintptr_t>(g) - reinterpret_cast<uintptr_t>(u)
                                                      : reinterpret_cast<uintptr_t>(u) - reinterpret_cast<uintptr_t>(g));
  // a tensor map's strides are multiples of 16 bytes below 2^40
  if (H % 64 != 0 || gap == 0 || gap % 16 != 0 || gap >= (1LL << 40)) return FFM_ERR_UNSUPPORTED;
  if (activation < 0 || activation > 3) return FFM_ERR_BAD_ARG;
  p->feats[i] = H;
  p->swap_gate[i] = up_low ? 1 : 0;
  p->act[i] = activation;
  const int rc = make_glu_weight_map(tmA, up_low ? u : g, gap, D, H, groups, group_bytes);
  return rc != FFM_OK ? rc : make_store_map(tmC, act, rows, H);
}

}  // namespace

}  // namespace ffm

using namespace ffm;

// groups == 0: the shared expert alone
static bool bad_decode(int64_t N, int D, int H, int Hs, int top_k, int groups, const int32_t* tile_start,
                       const int32_t* counts, int64_t rows, const int32_t* status) {
  if (!status || N < 1 || N > (1LL << 30) || D <= 0 || Hs < 0 || top_k < 1) return true;
  if (groups < 0 || groups > MAX_GROUPS || rows < 0 || rows > (1LL << 30)) return true;
  if (groups == 0) return Hs == 0;
  return !tile_start || !counts || H <= 0 || rows < 1;
}

extern "C" int ffm_decode_up(const void* x, const int32_t* src, const void* hidden, int64_t N, int D, int top_k, int groups,
                             const int32_t* tile_start, const int32_t* counts, int64_t rows, const void* w_up, int H,
                             int activation, void* act, const void* sw_gate, const void* sw_up, int Hs,
                             int shared_activation, void* s_act, int32_t* status, ffm_stream_t stream) {
  if (bad_decode(N, D, H, Hs, top_k, groups, tile_start, counts, rows, status)) return FFM_ERR_BAD_ARG;
  if (groups > 0 && (!x || !w_up || !act)) return FFM_ERR_BAD_ARG;
  if (Hs > 0 && (!hidden || !sw_gate || !sw_up || !s_act)) return FFM_ERR_BAD_ARG;
  if (D % 64 != 0) return FFM_ERR_UNSUPPORTED;
  TokParams p = {};
  CUtensorMap m[6];
  int rc;
  if (groups > 0) {
    const long long half = static_cast<long long>(H) * D * 2;
    if ((rc = up_side(&m[0], &m[2], &p, 0, w_up, static_cast<const uint8_t*>(w_up) + half, groups, 2 * half, D, H,
                      activation, act, rows)) != FFM_OK) return rc;
    if ((rc = make_map_2d(&m[1], x, src != nullptr ? N : rows, D, 64, src != nullptr ? 1 : 16)) != FFM_OK) return rc;
  }
  if (Hs > 0) {
    if ((rc = up_side(&m[3], &m[5], &p, 1, sw_gate, sw_up, 1, static_cast<long long>(Hs) * D * 2, D, Hs, shared_activation,
                      s_act, N)) != FFM_OK) return rc;
    if ((rc = make_map_2d(&m[4], hidden, N, D, 64, 16)) != FFM_OK) return rc;
  }
  fill_missing(m, groups > 0, Hs > 0);
  p.tile_start = tile_start;
  p.counts = counts;
  p.src = src;
  p.groups = groups;
  p.top_k = top_k;
  p.tokens = static_cast<int>(N);
  p.k_blocks[0] = p.k_blocks[1] = D / BK;
  p.status = status;
  p.wait_cycles = gemm_wait_cycles();
  return launch_tok<EPI_GLU>(m, p, rows, static_cast<cudaStream_t>(stream));
}

extern "C" int ffm_decode_down(const void* act, int64_t rows, int H, int groups, const int32_t* tile_start,
                               const int32_t* counts, int top_k, const void* w_down, int D, void* Y, const void* s_act,
                               int64_t N, int Hs, const void* sw_down, void* s_out, int32_t* status, ffm_stream_t stream) {
  if (bad_decode(N, D, H, Hs, top_k, groups, tile_start, counts, rows, status)) return FFM_ERR_BAD_ARG;
  if (groups > 0 && (!act || !w_down || !Y)) return FFM_ERR_BAD_ARG;
  if (Hs > 0 && (!s_act || !sw_down || !s_out)) return FFM_ERR_BAD_ARG;
  if ((groups > 0 && H % 64 != 0) || Hs % 64 != 0 || D % 32 != 0) return FFM_ERR_UNSUPPORTED;
  if (static_cast<long long>(groups) * D > 0x7fffffffLL) return FFM_ERR_UNSUPPORTED;
  TokParams p = {};
  CUtensorMap m[6];
  int rc;
  if (groups > 0) {
    if ((rc = make_map_2d(&m[0], w_down, static_cast<long long>(groups) * D, H, 64, 128)) != FFM_OK) return rc;
    if ((rc = make_map_2d(&m[1], act, rows, H, 64, 16)) != FFM_OK) return rc;
    if ((rc = make_store_map(&m[2], Y, rows, D)) != FFM_OK) return rc;
    p.k_blocks[0] = H / BK;
    p.feats[0] = D;
  }
  if (Hs > 0) {
    if ((rc = make_map_2d(&m[3], sw_down, D, Hs, 64, 128)) != FFM_OK) return rc;
    if ((rc = make_map_2d(&m[4], s_act, N, Hs, 64, 16)) != FFM_OK) return rc;
    if ((rc = make_store_map(&m[5], s_out, N, D)) != FFM_OK) return rc;
    p.k_blocks[1] = Hs / BK;
    p.feats[1] = D;
  }
  fill_missing(m, groups > 0, Hs > 0);
  p.tile_start = tile_start;
  p.counts = counts;
  p.groups = groups;
  p.top_k = top_k;
  p.tokens = static_cast<int>(N);
  p.status = status;
  p.wait_cycles = gemm_wait_cycles();
  return launch_tok<EPI_PLAIN>(m, p, rows, static_cast<cudaStream_t>(stream));
}
