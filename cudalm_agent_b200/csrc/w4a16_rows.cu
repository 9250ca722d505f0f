// Many activation rows (a prompt: more than 64) on the fifth-generation tensor cores.
//
// One CTA per SM works on units of 128 weight rows x NT activation rows of one projection
// (NT = 256, 128 or 64).  The weight rows are the M dimension of the MMA (A, in tensor
// memory), the activation rows its N dimension (B, in shared memory).  Per quantisation
// group of 128 k:
//
//   * 128 "dequantising" threads, one per weight row, turn the row's 64 packed bytes into
//     exact bf16 integers and write them to tensor memory (tcgen05.st).  Two sets of 128
//     take alternate groups;
//   * an issuing thread runs the group's eight K=16 MMAs into a fresh fp32 accumulator
//     slot (two issuers with a slot each at NT = 256);
//   * 256 "fold" threads read the slot back and add scale * sum to the unit's running
//     sums in registers, NT / 2 per thread, two to an instruction (fma.rn.f32x2).
//
// The group's scale multiplies its fp32 sum, as in the kernel for up to 64 rows: folding
// it into the bf16 operand would round it away (an fp16 scale times a 4-bit integer has 14
// significant bits).  Products are exact and sums are fp32.
//
// Work runs along three rings: packed weights (shared memory, two groups per stage),
// activations (shared memory, one group per stage) and A buffers / accumulator slots
// (tensor memory).
//
// What bounds it: not DRAM (a projection is read once into L2) and not yet the tensor pipe
// (a third busy): a chain of hand-overs per group.  An unsatisfied wait polls, and polling
// slows every other role (with a tight loop in place of tc_wait's reads of the timer 6144 x
// 1024 and 2048 rows took 40 us instead of 29); so each role waits once per group on all it
// needs, and one barrier per group tells everybody that its MMAs are done.  2048 rows of a
// layer with hidden size 1024 (four calls): 2018 us as passes of 64 rows, 180 with direct
// stores and three commits per group, 128 now.
//
// Every wait is bounded; a wait that runs out raises a CTA-wide abort flag, the kernel
// stores ERR_TIMEOUT in the status word, frees its tensor memory and returns.
#include <cuda.h>

#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "tcgen05.cuh"

namespace cb200 {
namespace {

enum : int { kRowsPlain = 0, kRowsPair = 1, kRowsResidual = 2 };

// A launch's parameters reach each CTA through a cold constant cache, so the numbers that
// every role needs before it can start lie together in front of the tensor maps.
struct RowsInfo {
  const std::uint16_t* S;
  const std::uint16_t* S2;   // kRowsPair: scales of the second matrix
  const std::uint16_t* res;  // kRowsResidual: residual [M][N]; may be y
  std::uint16_t* y;
  int N, K, M;
  int mode;
  int direct_store;  // outputs (or the residual) are not what the TMA unit takes
  int tok_tiles;     // unit = weight tile * tok_tiles + activation tile
  int unit_begin;    // first unit of this projection in the launch
  int unit_end;
  int cost_begin;  // groups before this projection
};
struct alignas(64) RowsMaps {
  CUtensorMap tmap;   // weights as uint32 [N][K/8], box 128 rows (a pair: 64) x 32 words
  CUtensorMap tmap2;  // kRowsPair: the second (up) matrix
  CUtensorMap xmap;   // activations as bf16 [K/64][M][64], box kBoxes x NT rows x 64 values
  CUtensorMap ymap;   // outputs as bf16 [M][N], box 32 rows x 32 values (a pair: 16)
  CUtensorMap rmap;   // kRowsResidual: the residual, box as ymap
};
struct RowsParams {
  int n_desc;
  int total_units;
  int total_cost;
  int* status;
  RowsInfo d[CUDALM_B200_MAX_INLINE_LINEARS];
  RowsMaps maps[CUDALM_B200_MAX_INLINE_LINEARS];
};

// Register shares (of the 640 x 96 the CTA is launched with; 256 fold, 256 dequantising
// and 128 other threads): 256 x 176 + 256 x 48 + 128 x 32 = 61440 where a fold thread keeps
// 128 sums, 256 x 136 + 256 x 72 + 128 x 64 = 61440 otherwise.
template <int NT>
struct RowsCfg {
  static constexpr int kSub = NT == 256 ? 2 : 1;         // MMAs along N per K=16 step (N <= 128 each)
  static constexpr int kSlot = NT / kSub;                // columns of an accumulator slot
  static constexpr int kAcc = NT / 2;                    // running sums per fold thread
  static constexpr int kLd = 32;                         // columns read back at a time
  static constexpr int kD = NT == 256 ? 3 : (NT == 128 ? 2 : 4);  // accumulator slots
  // Barriers for a freed slot.  NT = 256: the three slots go round over both halves, so one
  // half can hold all three; four barriers keep it from lapping one.
  static constexpr int kDB = NT == 256 ? 4 : kD;
  static constexpr int kA = NT == 256 ? 2 : 4;           // A buffers of 64 columns
  static constexpr int kW = NT == 256 ? 2 : (NT == 128 ? 4 : 6);   // weight stages (two groups, 16 KB)
  // An activation stage holds kBoxes blocks of 64 k (two per group), fetched by one copy
  // instruction: issuing one costs the copy thread several hundred cycles.
  static constexpr int kBoxes = NT == 256 ? 1 : (NT == 128 ? 2 : 4);
  static constexpr int kB = NT == 256 ? 5 : (NT == 128 ? 4 : 3);
  // Barriers for a finished group: more than any ring that waits for them reaches back.
  static constexpr int kR = NT == 256 ? 4 : 8;
  static constexpr int kBoxBytes = NT * 128;             // NT rows x 64 values
  static constexpr int kBBytes = kBoxes * kBoxBytes;
  static constexpr int kRegFold = NT == 256 ? 176 : 136;
  static constexpr int kRegDequant = NT == 256 ? 48 : 72;
  static constexpr int kRegOther = NT == 256 ? 32 : 64;
  static_assert(kD * kSlot + kA * 64 <= 512, "tensor memory");
  static_assert(kW % 2 == 0 && kA <= kR && kB * kBoxes / 2 < kR, "rings");
};
constexpr int kRowsWBytes = kTcRowsPerTile * 128;
constexpr int kRowsHeaderBytes = 1024;
constexpr int kRowsChunk = 32;                                       // activation rows per output box
constexpr int kRowsOutBytes = kRowsChunk * 32 * 2;                   // two of them per fold warp
template <int NT>
constexpr int rows_smem_bytes() {
  return 1024 + kRowsHeaderBytes + RowsCfg<NT>::kW * kRowsWBytes + RowsCfg<NT>::kB * RowsCfg<NT>::kBBytes +
         16 * kRowsOutBytes;
}

// Warp roles: 0..3 and 4..7 dequantise alternate weight stages, 8..11 and 12..15 fold (each
// half of the activation rows), 16 copies weights, 18 activations, 17 and 19 issue MMAs.
constexpr int kRowsThreads = 640;
constexpr int kRowsFoldWarp0 = 8;
constexpr int kRowsWeightWarp = 16;
constexpr int kRowsIssueWarp = 17;  // second issuer: + 2
constexpr int kRowsActWarp = 18;

struct RowsSmem {
  std::uint64_t w_full[6], w_empty[6];
  std::uint64_t b_full[5];
  std::uint64_t a_full[4];
  // a group's MMAs have completed: its sums are in their slot, its A buffer and activations
  // are free ([half of the activation rows at NT = 256][group modulo kR])
  std::uint64_t done[2][8];
  std::uint64_t d_free[2][4];
  std::uint64_t res_full[8][2];  // [fold warp][output buffer]: residual values have arrived
  std::uint32_t tmem_base;
  int abort_flag;
};
static_assert(sizeof(RowsSmem) <= kRowsHeaderBytes, "barrier block too large");

// A position in a ring of n stages and the parity of the phase it is in.
struct Ring {
  int i = 0;
  std::uint32_t phase = 0;
  __device__ __forceinline__ void next(int n) {
    if (++i == n) {
      i = 0;
      phase ^= 1u;
    }
  }
};

// Waits of one warp on several barriers at once: every lane with `need` waits on its own
// (a satisfied wait costs a warp on the order of two hundred cycles in this kernel, so they
// are not made one after the other).  All lanes return the same value.
__device__ __forceinline__ bool wait_lanes(bool need, std::uint64_t* bar, std::uint32_t parity,
                                           volatile int* abort_flag) {
  const bool ok = !need || tc_wait(bar, parity, abort_flag);
  const bool all = __all_sync(0xffffffffu, ok);
  __syncwarp();
  return all;
}

// acc += {s, s} * {d0, d1}; volatile, so that it stays behind the wait for the tensor-memory
// load that d0 and d1 come from.
__device__ __forceinline__ void fma_f32x2(unsigned long long& acc, std::uint32_t d0, std::uint32_t d1,
                                          unsigned long long s2) {
  asm volatile("{\n\t.reg .b64 p;\n\tmov.b64 p, {%1, %2};\n\tfma.rn.f32x2 %0, p, %3, %0;\n\t}"
               : "+l"(acc)
               : "r"(d0), "r"(d1), "l"(s2));
}
__device__ __forceinline__ float lo_f(unsigned long long v) {
  return __uint_as_float(static_cast<std::uint32_t>(v));
}
__device__ __forceinline__ float hi_f(unsigned long long v) {
  return __uint_as_float(static_cast<std::uint32_t>(v >> 32));
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, std::uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, std::uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
// bf16(silu(gate)) of a bf16 value, the bits of silu_bits(): the quotient comes from an
// approximate reciprocal and one Newton correction of its residual (Markstein's method)
// without a branch.  Every bf16 argument was compared.  A denominator too large for its
// reciprocal is scaled down; where the residual is not a number (an infinite gate or
// denominator) the product stands.  A branch to the correctly rounded division, as rarely as
// it was taken, cost 13 us of 69 (3584 x 1024, 2048 rows): its eight copies in the loop below.
__device__ __forceinline__ std::uint16_t silu_bits_fast(std::uint16_t gate_bits) {
  const float g = bf16_bits_to_float(gate_bits);
  const float scale = g < -64.f ? 0x1p-64f : 1.f;
  const float d = (1.0f + expf(-g)) * scale;
  float rc;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc) : "f"(d));
  const float q = g * rc;
  const float r = fmaf(-q, d, g);
  return float_to_bf16_bits((r == r ? fmaf(r, rc, q) : q) * scale);
}

// The weight and activation tile of consecutive units of one projection.
struct UnitTiles {
  int j, t;
  __device__ __forceinline__ void start(const RowsInfo& L, int u) {
    j = (u - L.unit_begin) / L.tok_tiles;
    t = (u - L.unit_begin) - j * L.tok_tiles;
  }
  __device__ __forceinline__ void next(const RowsInfo& L) {
    if (++t == L.tok_tiles) {
      t = 0;
      ++j;
    }
  }
};

template <int NT, bool EXTRA>
__global__ void __launch_bounds__(kRowsThreads, 1) w4a16_rows_kernel(const __grid_constant__ RowsParams p) {
  using C = RowsCfg<NT>;
  extern __shared__ __align__(1024) std::uint8_t smem_raw[];
  // the swizzled TMA destinations need 1024-byte alignment; the launch adds the slack
  std::uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  RowsSmem* sm = reinterpret_cast<RowsSmem*>(smem);
  std::uint8_t* wst = smem + kRowsHeaderBytes;
  std::uint8_t* bst = wst + C::kW * kRowsWBytes;
  std::uint8_t* outsm = bst + C::kB * C::kBBytes;
  volatile int* abort_flag = &sm->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int i = 0; i < C::kW; ++i) {
      mbar_init(&sm->w_full[i], 1);
      mbar_init(&sm->w_empty[i], 4);  // the warps of the stage's dequantising set
    }
    for (int i = 0; i < C::kB; ++i) mbar_init(&sm->b_full[i], 1);
    for (int i = 0; i < C::kA; ++i) mbar_init(&sm->a_full[i], 4);
    for (int h = 0; h < C::kSub; ++h) {
      for (int i = 0; i < C::kR; ++i) mbar_init(&sm->done[h][i], 1);
      for (int i = 0; i < C::kDB; ++i) mbar_init(&sm->d_free[h][i], C::kSub == 2 ? 4 : 8);
    }
    if (EXTRA)
      for (int i = 0; i < 16; ++i) mbar_init(&sm->res_full[i >> 1][i & 1], 1);
    sm->abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(&sm->tmem_base, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const std::uint32_t tmem_d = sm->tmem_base;
  const std::uint32_t tmem_a = tmem_d + C::kD * C::kSlot;

  // This CTA's contiguous range of units: an equal share of the groups.
  // (One projection, as almost always: 32-bit arithmetic; 64-bit divisions by every thread
  // took a microsecond.)
  int u_lo, u_hi;
  if (p.n_desc == 1 && p.total_units < (1 << 22)) {
    const unsigned units = static_cast<unsigned>(p.total_units);
    u_lo = static_cast<int>(blockIdx.x * units / gridDim.x);
    u_hi = static_cast<int>((blockIdx.x + 1) * units / gridDim.x);
  } else {
    auto unit_at = [&](long long cost) -> int {
      if (cost >= p.total_cost) return p.total_units;
      int d = p.n_desc - 1;
      while (d > 0 && p.d[d].cost_begin > cost) --d;
      const int per = p.d[d].K >> 7;
      return p.d[d].unit_begin + static_cast<int>((cost - p.d[d].cost_begin + per - 1) / per);
    };
    u_lo = unit_at(static_cast<long long>(blockIdx.x) * p.total_cost / gridDim.x);
    u_hi = unit_at(static_cast<long long>(blockIdx.x + 1) * p.total_cost / gridDim.x);
  }
  int di = 0;  // projection of the current unit
  UnitTiles tile = {0, 0};
  int tile_di = -1;
  auto seek = [&](int u) {
    while (u >= p.d[di].unit_end) ++di;
    if (di != tile_di) {
      tile_di = di;
      tile.start(p.d[di], u);
    } else {
      tile.next(p.d[di]);
    }
  };

  // Programmatic dependent launch: only the weight copies (weights are nobody's output)
  // may run before the preceding kernel has completed.
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (warp != kRowsWeightWarp) asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp >= kRowsWeightWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kRegOther) : "memory");
    if (warp == kRowsWeightWarp) {
      if (lane == 0) {
        // ---------------- packed weights ----------------
        Ring w;
        bool first_round = true, ok = true;
        for (int u = u_lo; u < u_hi && ok && !*abort_flag; ++u) {
          seek(u);
          const RowsInfo& L = p.d[di];
          const bool pair = EXTRA && L.mode == kRowsPair;
          const int j = tile.j;
          const int stages = ((L.K >> 7) + 1) >> 1;
          for (int c = 0; c < stages; ++c) {
            if (!first_round && !tc_wait(&sm->w_empty[w.i], w.phase ^ 1u, abort_flag)) {
              ok = false;
              break;
            }
            std::uint8_t* st = wst + w.i * kRowsWBytes;
            mbar_arrive_expect_tx(&sm->w_full[w.i], kRowsWBytes);
            for (int m = 0; m < (pair ? 2 : 1); ++m)
              tma_load_2d(st + m * (kRowsWBytes / 2), m ? &p.maps[di].tmap2 : &p.maps[di].tmap, c * 32, j * (pair ? 64 : 128),
                          &sm->w_full[w.i]);
            w.next(C::kW);
            if (w.i == 0) first_round = false;
          }
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
      }
    } else if (warp == kRowsActWarp) {
      // ---------------- activations ----------------
      Ring b;
      int n_stage = 0;  // stages so far
      // last group (in the CTA's count) of the stages in the ring, to know when one is free
      std::uint32_t last[C::kB];
      std::uint32_t git = 0;
      bool ok = true;
      for (int u = u_lo; u < u_hi && ok && !*abort_flag; ++u) {
        seek(u);
        const RowsInfo& L = p.d[di];
        const int t = tile.t;
        const int blocks = L.K >> 6;
        for (int q = 0; q < blocks; q += C::kBoxes, ++n_stage) {
          // the last group whose activations were here is done with (by both issuers at
          // NT = 256, where a stage is half a group)
          std::uint32_t past = 0;
#pragma unroll
          for (int i = 0; i < C::kB; ++i)
            if (i == b.i) past = last[i];
          ok = wait_lanes(n_stage >= C::kB && lane < C::kSub, &sm->done[lane & (C::kSub - 1)][past % C::kR],
                          (past / C::kR) & 1u, abort_flag);
          if (!ok) break;
          const int end = q + C::kBoxes < blocks ? q + C::kBoxes : blocks;
#pragma unroll
          for (int i = 0; i < C::kB; ++i)
            if (i == b.i) last[i] = git + ((end - 1) >> 1);
          if (lane == 0) {
            // rows past M and blocks past K arrive as zeros
            mbar_arrive_expect_tx(&sm->b_full[b.i], C::kBBytes);
            tma_load_3d(bst + b.i * C::kBBytes, &p.maps[di].xmap, 0, t * NT, q, &sm->b_full[b.i]);
          }
          b.next(C::kB);
        }
        git += blocks >> 1;
      }
    } else {
      // ---------------- MMA issue ----------------
      // NT = 256: one issuer per half of the activation rows; otherwise they take
      // alternate groups, so that one's waits and commits run beside the other's MMAs.
      const std::uint32_t who = static_cast<std::uint32_t>(warp - kRowsIssueWarp) >> 1;
      const int h = C::kSub == 2 ? static_cast<int>(who) : 0;
      const std::uint32_t desc_hi = static_cast<std::uint32_t>(tc_b_desc(0) >> 32);
      const std::uint32_t desc_lo0 = static_cast<std::uint32_t>(tc_b_desc(0));
      const std::uint32_t b0 = smem_u32(bst) + static_cast<std::uint32_t>(h) * 128u * 128u;
      constexpr std::uint32_t kIdesc = tc_idesc(C::kSlot);
      Ring b;
      std::uint32_t git = 0;
      int slot = h;  // NT = 256: slots go round over both halves, 2 git + h modulo 3
      bool ok = true;
      for (int u = u_lo; u < u_hi && ok && !*abort_flag; ++u) {
        seek(u);
        const int G = p.d[di].K >> 7;
        for (int g = 0; g < G; ++g, ++git) {
          // the stage or stages of the group, and where in them its two blocks of 64 k are
          const Ring b_lo = b;
          if (C::kBoxes == 1) b.next(C::kB);
          const Ring b_hi = b;
          const std::uint32_t block = C::kBoxes == 4 ? 2u * (g & 1) : 0u;
          if (C::kBoxes <= 2 || (g & 1) || g == G - 1) b.next(C::kB);
          if (C::kSub == 1 && (git & 1u) != who) continue;
          // Lane 0: the slot's previous sums have been read.  NT = 256: they were the other
          // half's, three slot uses ago, i.e. of group git - 1 (h = 1) or git - 2 (h = 0);
          // otherwise those of kD groups ago.  Lanes 1, 2: both halves of the group's
          // activations have landed.  Lane 3: the A buffer holds the group.
          const std::uint32_t back = C::kSub == 2 ? (h == 1 ? 1u : 2u) : static_cast<std::uint32_t>(C::kD);
          const std::uint32_t prev = git - back;
          std::uint64_t* bar = &sm->d_free[C::kSub == 2 ? 1 - h : 0][prev % C::kDB];
          std::uint32_t parity = (prev / C::kDB) & 1u;
          if (lane == 1) bar = &sm->b_full[b_lo.i], parity = b_lo.phase;
          if (lane == 2) bar = &sm->b_full[b_hi.i], parity = b_hi.phase;
          if (lane == 3) bar = &sm->a_full[git % C::kA], parity = (git / C::kA) & 1u;
          ok = wait_lanes(lane < 4 && (lane > 0 || git >= back), bar, parity, abort_flag);
          if (!ok) break;
          if (lane == 0) {
            tc_fence_after();
            const std::uint32_t lo = (b0 + b_lo.i * C::kBBytes + block * C::kBoxBytes) >> 4;
            const std::uint32_t hi =
                C::kBoxes == 1 ? (b0 + b_hi.i * C::kBBytes) >> 4 : lo + (C::kBoxBytes >> 4);
            const int s = C::kSub == 2 ? slot : static_cast<int>(git % C::kD);
            tc_mma_group(tmem_d + s * C::kSlot, tmem_a + (git % C::kA) * 64, desc_lo0 | lo, desc_hi, hi - lo, kIdesc);
            tc_commit(&sm->done[h][git % C::kR]);
          }
          __syncwarp();
          slot += 2;
          if (slot >= C::kD) slot -= C::kD;
        }
      }
    }
  } else if (warp < kRowsFoldWarp0) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kRegDequant) : "memory");
    // ---------------- dequantise: the A operand ----------------
    const int set = warp >> 2;  // takes the weight stages of this parity (kW is even)
    const int lrow = (warp & 3) * 32 + lane;
    const std::uint32_t a_base = tmem_a + (static_cast<std::uint32_t>((warp & 3) * 32) << 16);
    // groups handed over at a time: both of a stage where a group is short (NT = 64)
    constexpr int kStep = NT == 64 ? 2 : 1;
    std::uint32_t git = 0;
    Ring w;
    bool alive = true;
    for (int u = u_lo; u < u_hi && alive; ++u) {
      seek(u);
      const int G = p.d[di].K >> 7;
      // a pair's rows alternate gate, up (64 rows of either matrix)
      const bool pair = EXTRA && p.d[di].mode == kRowsPair;
      const int srow = pair ? (lrow & 1) * 64 + (lrow >> 1) : lrow;
      for (int g = 0; g < G && alive; g += 2) {
        const int n = G - g < 2 ? 1 : 2;
        if ((w.i & 1) == set) {
          const std::uint8_t* rowp = wst + w.i * kRowsWBytes + srow * 128;
          for (int i0 = 0; i0 < n; i0 += kStep) {
            // lane 0: the stage has landed; the others: the groups that were in the A
            // buffers are done with
            const int m = n - i0 < kStep ? n - i0 : kStep;
            const int which = (lane - 1) / C::kSub;  // group of this step the lane asks about
            const std::uint32_t past = git + i0 + which - C::kA;
            const bool asks = lane >= 1 && which < m && git + i0 + which >= static_cast<std::uint32_t>(C::kA);
            alive = wait_lanes(lane == 0 || asks,
                               lane == 0 ? &sm->w_full[w.i] : &sm->done[(lane - 1) & (C::kSub - 1)][past % C::kR],
                               lane == 0 ? w.phase : (past / C::kR) & 1u, abort_flag);
            if (!alive) break;
            tc_fence_after();
            for (int i = i0; i < i0 + m; ++i) {
              const std::uint32_t a_addr = a_base + ((git + i) % C::kA) * 64;
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                std::uint32_t regs[16];
                const uint4 v = lds128(rowp + (((4 * i + q) ^ (srow & 7)) << 4));
                dequant_word_natural(v.x, regs);
                dequant_word_natural(v.y, regs + 4);
                dequant_word_natural(v.z, regs + 8);
                dequant_word_natural(v.w, regs + 12);
                tmem_st16(a_addr + 16 * q, regs);
              }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane < m) mbar_arrive(&sm->a_full[(git + i0 + lane) % C::kA]);
          }
          if (!alive) break;
          if (lane == 0) mbar_arrive(&sm->w_empty[w.i]);
        }
        git += n;
        w.next(C::kW);
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kRegFold) : "memory");
    // ---------------- fold: acc += scale * sum ----------------
    const int f = (warp - kRowsFoldWarp0) >> 2;  // half of the activation rows
    const int h = C::kSub == 2 ? f : 0;
    const int lrow = (warp & 3) * 32 + lane;
    const std::uint32_t d_base = tmem_d + (static_cast<std::uint32_t>((warp & 3) * 32) << 16) +
                                 (C::kSub == 2 ? 0u : static_cast<std::uint32_t>(f) * C::kAcc);
    const int fw = warp - kRowsFoldWarp0;
    std::uint8_t* outs = outsm + fw * 2 * kRowsOutBytes;  // this warp's two output buffers
    constexpr int kChunks = C::kAcc / kRowsChunk;
    static_assert(kChunks == 1 || kChunks % 2 == 0, "output buffers");
    std::uint32_t git = 0;
    std::uint32_t res_phase = 0;  // bit i: phase of res_full[fw][i]
    int slot = h;
    bool alive = true;
    for (int u = u_lo; u < u_hi && alive; ++u) {
      seek(u);
      const RowsInfo& L = p.d[di];
      const int N = L.N, G = L.K >> 7;
      const int j = tile.j, t = tile.t;
      const bool pair = EXTRA && NT < 256 && L.mode == kRowsPair;
      const bool residual = EXTRA && L.mode == kRowsResidual;
      const bool tma_residual = residual && !L.direct_store;
      // first weight row of this warp, and this lane's (a pair: lanes alternate gate, up)
      const int row0 = pair ? j * 64 + (warp & 3) * 16 : j * 128 + (warp & 3) * 32;
      const int row = row0 + (pair ? lane >> 1 : lane);
      const int tok0 = t * NT + f * C::kAcc;
      const bool row_ok = row < N;
      const std::uint16_t* srow = ((pair && (lrow & 1)) ? L.S2 : L.S) + static_cast<std::size_t>(row_ok ? row : 0) * G;
      // the buffers take turns, across units too (at NT = 64 a unit has one box only)
      auto buffer = [&](int c) { return kChunks == 1 ? (u - u_lo) & 1 : c & 1; };
      auto fetch_residual = [&](int c) {
        const int b = buffer(c);
        mbar_arrive_expect_tx(&sm->res_full[fw][b], kRowsOutBytes);
        tma_load_2d(outs + b * kRowsOutBytes, &p.maps[di].rmap, row0, tok0 + c * kRowsChunk, &sm->res_full[fw][b]);
      };
      if (tma_residual && lane == 0) {
        // into the output buffers, once the previous unit's stores have read them
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        for (int c = 0; c < (kChunks < 2 ? kChunks : 2); ++c) fetch_residual(c);
      }
      unsigned long long acc[C::kAcc / 2];
#pragma unroll
      for (int n = 0; n < C::kAcc / 2; ++n) acc[n] = 0ull;
      // the scale of the next group is fetched while this one's sums are awaited
      std::uint16_t sc_bits = __ldg(srow);
      for (int g = 0; g < G; ++g, ++git) {
        const std::uint32_t sc = __float_as_uint(__half2float(__ushort_as_half(sc_bits)));
        const unsigned long long s2 = (static_cast<unsigned long long>(sc) << 32) | sc;
        if (g + 1 < G) sc_bits = __ldg(srow + g + 1);
        const bool ok = tc_wait(&sm->done[h][git % C::kR], (git / C::kR) & 1u, abort_flag);
        alive = __all_sync(0xffffffffu, ok);
        if (!alive) break;
        tc_fence_after();
        const std::uint32_t d_addr = d_base + (C::kSub == 2 ? slot : static_cast<int>(git % C::kD)) * C::kSlot;
#pragma unroll
        for (int c = 0; c < C::kAcc / C::kLd; ++c) {
          std::uint32_t d[C::kLd];
          tmem_ld_cols<C::kLd>(d_addr + c * C::kLd, d);
          if (c == C::kAcc / C::kLd - 1) {
            // the sums are in registers: hand the slot back before the arithmetic
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm->d_free[h][git % C::kDB]);
          }
#pragma unroll
          for (int i = 0; i < C::kLd / 2; ++i)
            fma_f32x2(acc[c * (C::kLd / 2) + i], d[2 * i], d[2 * i + 1], s2);
        }
        slot += 2;
        if (slot >= C::kD) slot -= C::kD;
      }
      if (!alive) break;
      // ---- outputs, 32 activation rows at a time through the warp's own box [activation
      // row][weight row] in shared memory, which a TMA store (or the lanes, where the TMA
      // unit does not take the addresses) copies out.  Boxes of all four warps together
      // make longer rows, but their two barriers per box cost more than the stores. ----
#pragma unroll
      for (int c = 0; c < kChunks; ++c) {
        const int b = buffer(c);
        std::uint8_t* box = outs + b * kRowsOutBytes;
        if (tma_residual) {
          const bool ok = tc_wait(&sm->res_full[fw][b], (res_phase >> b) & 1u, abort_flag);
          res_phase ^= 1u << b;
          alive = __all_sync(0xffffffffu, ok);
          if (!alive) break;
        } else {
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
          __syncwarp();
        }
        if (pair) {
          // An even lane holds the gate and its odd neighbour the up output of one row: they
          // exchange one of every two values, and each finishes one activation row.  The
          // box first takes {gate, up} words and is then rewritten from the front, eight
          // words a lane at a time (unrolled over all of them the code misses the
          // instruction cache).
          std::uint32_t* words = reinterpret_cast<std::uint32_t*>(box) + lane;
#pragma unroll
          for (int n = 0; n < kRowsChunk; n += 2) {
            const unsigned long long v = acc[(c * kRowsChunk + n) / 2];
            const std::uint32_t mine = pack_bf16x2(lo_f(v), hi_f(v));
            const std::uint32_t other = __shfl_xor_sync(0xffffffffu, mine, 1);
            words[n * 16] = (lane & 1) ? __byte_perm(mine, other, 0x3276) : __byte_perm(mine, other, 0x5410);
          }
          std::uint8_t* slot16 = box + (lane & 1) * 32 + (lane >> 1) * 2;
#pragma unroll 1
          for (int i = 0; i < kRowsChunk / 2; i += 8) {
            std::uint32_t w[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) w[k] = words[(i + k) * 32];
            __syncwarp();  // the words behind these outputs have been read by every lane
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              // CUDALM's rounding order: bf16 after each projection, after silu, after the product
              const float silu = bf16_bits_to_float(silu_bits_fast(static_cast<std::uint16_t>(w[k])));
              *reinterpret_cast<std::uint16_t*>(slot16 + (i + k) * 64) =
                  float_to_bf16_bits(silu * bf16_bits_to_float(static_cast<std::uint16_t>(w[k] >> 16)));
            }
            __syncwarp();
          }
        } else {
          std::uint8_t* slot16 = box + lane * 2;
#pragma unroll
          for (int n = 0; n < kRowsChunk; n += 2) {
            const unsigned long long v = acc[(c * kRowsChunk + n) / 2];
            const std::uint32_t two = pack_bf16x2(lo_f(v), hi_f(v));
            std::uint16_t* s0 = reinterpret_cast<std::uint16_t*>(slot16 + n * 64);
            std::uint16_t* s1 = reinterpret_cast<std::uint16_t*>(slot16 + (n + 1) * 64);
            if (tma_residual) {
              *s0 = add_bits(*s0, static_cast<std::uint16_t>(two));
              *s1 = add_bits(*s1, static_cast<std::uint16_t>(two >> 16));
            } else {
              *s0 = static_cast<std::uint16_t>(two);
              *s1 = static_cast<std::uint16_t>(two >> 16);
            }
          }
        }
        const int tok = tok0 + c * kRowsChunk;
        if (!L.direct_store) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            if (tok < L.M && row0 < N)
              asm volatile(
                  "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                      &p.maps[di].ymap),
                  "r"(row0), "r"(tok), "r"(smem_u32(box))
                  : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            if (tma_residual && c + 2 < kChunks) {
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
              fetch_residual(c + 2);
            }
          }
        } else if (row_ok) {
          // each lane copies out the values it has written
          const int step = pair ? 2 : 1, n0 = pair ? lane & 1 : 0;
          for (int n = n0; n < kRowsChunk && tok + n < L.M; n += step) {
            std::uint16_t v = *reinterpret_cast<const std::uint16_t*>(
                pair ? box + n * 32 + (lane >> 1) * 2 : box + n * 64 + lane * 2);
            const std::size_t at = static_cast<std::size_t>(tok + n) * N + row;
            if (residual) v = add_bits(L.res[at], v);
            L.y[at] = v;
          }
        }
      }
    }
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }

  __syncthreads();
  if (*abort_flag && tid == 0) atomicExch(p.status, CUDALM_B200_ERR_TIMEOUT);
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_d, 512);
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
template <int NT, bool EXTRA>
int rows_launch(const RowsParams& p, cudaStream_t stream) {
  auto kern = w4a16_rows_kernel<NT, EXTRA>;
  constexpr int smem = rows_smem_bytes<NT>();
  static_assert(smem <= kMaxSmemBytes, "shared memory");
  static std::mutex mu;
  static std::vector<int> done;
  int dev = 0;
  CB200_CUDA_TRY(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lk(mu);
    bool seen = false;
    for (int d : done) seen |= (d == dev);
    if (!seen) {
      CB200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      done.push_back(dev);
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.total_units < num_sms() ? p.total_units : num_sms()));
  cfg.blockDim = dim3(kRowsThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, p);
  if (le != cudaSuccess) {
    g_last_cuda_error = static_cast<int>(le);
    (void)cudaGetLastError();
    return CUDALM_B200_ERR_CUDA;
  }
  return check_launch();
}

template <int NT>
int rows_launch_any(const RowsParams& p, bool extra, cudaStream_t stream) {
  return extra ? rows_launch<NT, true>(p, stream) : rows_launch<NT, false>(p, stream);
}

}  // namespace

// True when the many-row kernel takes this projection: the TMA unit needs 16-byte aligned
// bases for the weights and activations (their row pitches are multiples of 64 bytes).
bool rows_eligible(const cudalm_b200_linear& l) {
  if (l.M < 1 || l.K <= 0 || (l.K % 128) != 0 || l.N < 1) return false;
  return aligned_to(l.weight, 16) && aligned_to(l.x, 16);
}

// Up to CUDALM_B200_MAX_INLINE_LINEARS projections in one launch.  A single one may carry
// an MLP epilogue: weight2/scales2 non-null -> y = silu(W x) * (W2 x), residual non-null ->
// y = residual + W x.
int run_rows(const cudalm_b200_linear* ls, int count, const std::uint8_t* weight2, const std::uint16_t* scales2,
             const std::uint16_t* residual, cudaStream_t stream) {
  if (count < 1 || count > CUDALM_B200_MAX_INLINE_LINEARS) return CUDALM_B200_ERR_BAD_SHAPE;
  const bool pair = weight2 != nullptr;
  if (pair && (!aligned_to(weight2, 16) || !scales2)) return CUDALM_B200_ERR_UNSUPPORTED;
  for (int i = 0; i < count; ++i)
    if (!rows_eligible(ls[i])) return CUDALM_B200_ERR_UNSUPPORTED;
  const int tile_rows = pair ? 64 : 128;
  // The tile that finishes first: units of the most loaded SM times a unit's cycles, which
  // are its groups' and a fixed part (filling the pipeline, outputs).  Measured on 1024 x
  // 3584 and 6144 x 1024 with 2048 rows, 256 / 128 / 64: 29.3 / 19.8 / 34.4 and 29.4 / 34.9 /
  // 54.2 us.  A pair's silu lengthens the fixed part; with 128 sums a thread it has no
  // registers (3584 x 1024, 2048 rows: 140 us against 55).
  static constexpr int kTiles[3] = {256, 128, 64};
  static constexpr int kPerGroup[3] = {1560, 1075, 965};
  static constexpr int kPerUnit[3] = {6000, 2400, 1600};
  static constexpr int kPerPair[3] = {0, 6300, 2800};
  int nt = 0;
  long long best = 0;
  for (int k = pair ? 1 : 0; k < 3; ++k) {
    long long cycles = 0, units = 0, groups = 0, longest = 0;
    for (int i = 0; i < count; ++i) {
      const long long n = static_cast<long long>((ls[i].N + tile_rows - 1) / tile_rows) *
                          ((ls[i].M + kTiles[k] - 1) / kTiles[k]);
      const long long unit = static_cast<long long>(ls[i].K >> 7) * kPerGroup[k] + (pair ? kPerPair : kPerUnit)[k];
      units += n;
      groups += n * (ls[i].K >> 7);
      cycles += n * unit;
      if (unit > longest) longest = unit;
    }
    if (units > 0x3fffffff || groups > 0x3fffffff) return CUDALM_B200_ERR_TOO_LARGE;
    const long long time = count == 1 ? (units + num_sms() - 1) / num_sms() * longest : cycles / num_sms() + longest;
    if (nt == 0 || time < best) {
      best = time;
      nt = kTiles[k];
    }
  }
  RowsParams p;
  std::memset(&p, 0, sizeof(p));
  int units = 0, cost = 0;
  for (int i = 0; i < count; ++i) {
    const cudalm_b200_linear& l = ls[i];
    RowsInfo& d = p.d[i];
    RowsMaps& maps = p.maps[i];
    if (int rc = tc_encode(l.weight, l.K / 8, l.N, 32, tile_rows, 0, &maps.tmap)) return rc;
    if (pair)
      if (int rc = tc_encode(weight2, l.K / 8, l.N, 32, tile_rows, 0, &maps.tmap2)) return rc;
    if (int rc = tc_encode_blocks(l.x, l.K, l.M, nt, nt == 256 ? 1 : (nt == 128 ? 2 : 4), &maps.xmap)) return rc;
    d.S = l.scales;
    d.S2 = scales2;
    d.res = residual;
    d.y = l.y;
    d.N = l.N;
    d.K = l.K;
    d.M = l.M;
    d.mode = pair ? kRowsPair : (residual ? kRowsResidual : kRowsPlain);
    d.direct_store = (l.N % 8 != 0 || !aligned_to(l.y, 16) || (residual && !aligned_to(residual, 16))) ? 1 : 0;
    if (!d.direct_store) {
      if (int rc = tc_encode(l.y, l.N, l.M, tile_rows / 4, kRowsChunk, 2, &maps.ymap)) return rc;
      if (residual)
        if (int rc = tc_encode(residual, l.N, l.M, tile_rows / 4, kRowsChunk, 2, &maps.rmap)) return rc;
    }
    d.tok_tiles = (l.M + nt - 1) / nt;
    d.unit_begin = units;
    d.cost_begin = cost;
    const int n = (l.N + tile_rows - 1) / tile_rows * d.tok_tiles;
    units += n;
    cost += n * (l.K >> 7);
    d.unit_end = units;
  }
  p.n_desc = count;
  p.total_units = units;
  p.total_cost = cost;
  p.status = device_status_word();
  if (!p.status) return CUDALM_B200_ERR_CUDA;
  const bool extra = pair || residual;
  if (nt == 256) return rows_launch_any<256>(p, extra, stream);
  if (nt == 128) return rows_launch_any<128>(p, extra, stream);
  return rows_launch_any<64>(p, extra, stream);
}

}  // namespace cb200
