// The Lightning Attention-2 block kernel: warp-specialised and software-pipelined. Mathematics, operands, shared-memory slab layout
// and state conventions are described in la_kernels.cuh. Four roles work on different 128-token blocks at the same time and hand
// tiles to each other through mbarriers:
//
//   warp 0      TMA producer   loads A, Bm, C tiles of block i+1, i+2 into two shared-memory stages
//   warp 1      MMA issuer     X_i = A State_i, D_i = C^T (w Bm), PC_i = P_i C, S_{i+1} = A Bm^T, in this order (one thread)
//   warps 2-3   scaling        half of: Bm_i rows *= w_state (for D_i)
//   warps 4-7   mask group     S_i (TMEM) -> decay mask -> P_i (bf16, back into TMEM over S)
//   warps 8-15  state/output   the other half; D_i -> StateT = lambda^128 StateT + D_i (fp32 registers)
//                              -> bf16 copy for X_{i+1}; O_i = PC_i + w_out X_i -> swizzled shared-memory tile -> TMA store
//
// P never touches shared memory: it is written to TMEM with tcgen05.st and consumed by tcgen05.mma as the
// A operand, which frees the 32 KB that double-buffering A needs. Every wait is bounded and checks a
// CTA-wide abort flag, so a protocol error ends with an error status instead of a hang.
//
// Key widths of 129 to 256 (NKS = 3, 4; WIDE) run the same roles on 64-wide dv slices, with two differences. What does not fit twice
// into 227 KB has one stage: A always (200 KB at NKS = 3), at NKS = 4 Bm too; A is reloaded as soon as X_i has read it. And the
// fp32 state is held un-transposed: a warp can only read the TMEM lanes of its own quadrant, and the accumulator C^T (w Bm) has dv
// on its lanes, so with a 64-wide slice half of the state warps would reach nothing and the others need 96 to 128 registers per
// thread for their share. (w Bm)^T C has dk on its lanes, two M = 128 tiles of 64 columns, one per half of the state group: 64
// registers per thread, and the copy X reads is then a [dk][64] slab used as an MN-major operand, like C itself. What bounds a
// block is the chain X_i -> reload of A -> S_{i+1} -> mask -> P C. b2 h12 n2048 d=e=192: 59.6 us per launch with the phases of a
// block one after another behind CTA-wide barriers (the kernel these widths had before), now 31.8 (state-only pass 25.0 -> 17.7).
#pragma once
#include "la_kernels.cuh"

namespace lab200 {

// Four warpgroups: loads, MMAs and half of the Bm scaling, mask, and two of the state/output group. The launch gives every thread
// 128 registers; the fp32 state and the tiles beside it need more, the issuing threads far less, so the warpgroups split what
// the launch was given. At 128 for all, the loops spilled 124-144 bytes per thread, and what spills goes through the shared-memory
// pipe that bounds the kernel: b4 h32 n2048 d=e=128 forward 53.4 -> 51.4 us (at n32768 runs under the power cap differ by as much).
// What still spills in the block loop: 60 bytes at dk > 192, 4 to 8 at dk <= 64 and on 64-wide slices of dk <= 128.
constexpr int LAP_THREADS = 512;
constexpr int LAP_REGS[3] = {56, 120, 168};
static_assert(LAP_REGS[0] + LAP_REGS[1] + 2 * LAP_REGS[2] <= 512, "the split must not ask for more than the launch gave");
constexpr int LAP_MASK_THREADS = 128, LAP_STATE_THREADS = 256;
constexpr int LAP_SCALE_THREADS = 64;  // warps 2 and 3


// barrier slots (each has one instance per stage, indexed by block modulo the stage count)
enum : int { LAP_FULL_AB = 0, LAP_FULL_C, LAP_S_READY, LAP_P_READY, LAP_PC_DONE, LAP_D_DONE, LAP_O_FREE, LAP_D_FREE,
             LAP_STATE_READY, LAP_O_STAGED, LAP_BM_SCALED, LAP_A_FREE, LAP_NUM_BARS };

// Shared-memory stages, in 16 KB slabs (host and device agree through these).
__host__ __device__ constexpr bool lap_wide(int nks) { return nks > 2; }
__host__ __device__ constexpr int lap_a_slabs(int nks, int nvs) { return lap_wide(nks) ? nks : 2 * (nks > nvs ? nks : nvs); }  // all stages of A, full block loop
// Two stages in the full block loop. The state-only pass has nothing else in shared memory and takes three of (Bm, C), as far as they
// fit: a stage goes through load, scaling and D before its reload, and two of them left HBM idle between (b1 h32 n131072
// d=e=128: 339 -> 311 us per pass, 6.9 TB/s; b2 h16 n4096: 22.6 -> 20.6).
__host__ __device__ constexpr int lap_stages(int mode, int nks) { return (mode == 0 || nks == 4) ? 2 : 3; }
__host__ __device__ constexpr int lap_b_stages(int nks, int mode) { return (nks == 4 && mode == 0) ? 1 : lap_stages(mode, nks); }
__host__ __device__ constexpr int lap_c_slabs(int nks) { return lap_wide(nks) ? 1 : 2; }  // per stage: the M = 128 side of D for dk <= 128 reads two
__host__ __device__ constexpr int lap_smem_bytes(int nks, int nvs, int mode) {
  int b = (lap_b_stages(nks, mode) * nks + lap_stages(mode, nks) * lap_c_slabs(nks)) * LA_SLAB_BYTES;
  if (mode == 0) b += lap_a_slabs(nks, nvs) * LA_SLAB_BYTES + nks * nvs * 64 * 128;
  return b + lap_stages(mode, nks) * LAP_NUM_BARS * 8 + 16 + 512 + 1024;  // barriers, flags, decay table, alignment slack
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// TMA store of one [128 rows][64 columns] slab, shared -> global; rows/columns outside the tensor are dropped.
__device__ __forceinline__ void tma_store_3d(const void* tmap, uint32_t src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(tmap)), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Bounded, abortable wait. Returns false if the budget ran out here or another role gave up.
__device__ __forceinline__ bool lap_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, long long budget) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > budget) {
      *abort_flag = 1;
      return false;
    }
  }
  return true;
}

// NP 16-byte chunks of one 128-byte tile row times the row's factor, in place: positions rot, rot + 1, ... modulo 8. rot grows with the
// row, so that the same step of eight neighbouring rows covers all banks. EXACT: by w in fp32, one rounding per element; else packed, by
// w rounded to the 16-bit type.
template <int FMT, bool EXACT, int NP>
__device__ __forceinline__ void lap_scale(uint32_t row, int rot, float w) {
  uint32_t u[NP][4];
  const uint32_t w2 = pack2<FMT>(w, w);
#pragma unroll
  for (int c = 0; c < NP; ++c) ld_shared_v4(row + (((rot + c) & 7) << 4), u[c][0], u[c][1], u[c][2], u[c][3]);
#pragma unroll
  for (int c = 0; c < NP; ++c) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if constexpr (EXACT) {
        const float2 f = unpack2<FMT>(u[c][j]);
        u[c][j] = pack2<FMT>(f.x * w, f.y * w);
      } else {
        u[c][j] = mul2<FMT>(u[c][j], w2);
      }
    }
    st_shared_v4(row + (((rot + c) & 7) << 4), u[c][0], u[c][1], u[c][2], u[c][3]);
  }
}

template <int NKS, int NVS, int MODE, int FMT>
__global__ void __launch_bounds__(LAP_THREADS, 1)
la_pipe_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmO, const LaParams p) {
  constexpr bool WIDE = lap_wide(NKS);
  static_assert(NKS <= 4 && NVS <= 2 && (!WIDE || NVS == 1), "tile sizes");
  constexpr int SLAB = LA_SLAB_BYTES;
  constexpr int DV = 64 * NVS;
  constexpr int DKP = 64 * NKS;
  constexpr int SC = WIDE ? DV : DKP / 2;  // state columns per thread
  constexpr int OC = DV / 2;
  constexpr int NAS = WIDE ? 0 : (NKS > NVS ? NKS : NVS);  // slabs from one A stage to the next (0: there is one)
  constexpr int NBS = lap_b_stages(NKS, MODE) > 1 ? NKS : 0;
  constexpr int NST = lap_stages(MODE, NKS);
  // Warps 2 and 3 take half of the Bm scaling in the narrow block loop. In the state-only pass the state group has the time. The wide
  // widths (fp32 multiply, 48-64 KB) were measured at dk = 256 only, where Bm has one stage, and are slower with it there (4 x 16 x
  // 4096 x 256 forward 244 -> 268 us); 129 to 192, with two stages of Bm, follow that rule unmeasured.
  constexpr bool HELP = MODE == 0 && !WIDE;
  constexpr int NCS = lap_c_slabs(NKS);
  constexpr uint32_t T_S = 0, T_OI = 128, T_OX = 128 + DV, T_D = 128 + 2 * DV;
  static_assert(T_D + (WIDE ? 2 * DV : DKP) <= 512, "TMEM budget");
  constexpr uint32_t IDESC_S = umma_idesc(FMT, 128, 128, 0, 0);
  constexpr uint32_t IDESC_X = umma_idesc(FMT, 128, DV, 0, 0);
  constexpr uint32_t IDESC_PC = umma_idesc(FMT, 128, DV, 0, 1);
  constexpr uint32_t IDESC_ST = umma_idesc(FMT, 128, WIDE ? DV : DKP, 1, 1);

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t sA = base;                                         // MODE 0 only: 2 stages x NAS slabs, wide: 1 x NKS
  const uint32_t sB = sA + (MODE == 0 ? lap_a_slabs(NKS, NVS) * SLAB : 0);  // lap_b_stages x NKS slabs: 2 (NKS = 4: 1), state-only 3 (NKS = 4: 2)
  const uint32_t sC = sB + lap_b_stages(NKS, MODE) * NKS * SLAB;    // NST stages x NCS slabs: 2, state-only 3 (NKS = 4: 2)
  // 16-bit state: NKS x [DV rows][128 B] (rows dv, columns dk); wide: [DKP rows][128 B] (rows dk, columns dv) (MODE 0). The second
  // M = 128 tile of D at NKS = 3 reads one slab behind its Bm stage: that is the other stage or C, and only reaches accumulator
  // rows that nobody reads.
  const uint32_t sS = sC + NST * NCS * SLAB;
  // Output tiles are staged in the C stage of their own block (free once P C is done) and leave by TMA store.
  const uint32_t sBar = sS + (MODE == 0 ? NKS * DV * 128 : 0);      // NST x LAP_NUM_BARS mbarriers
  const uint32_t sMisc = sBar + NST * LAP_NUM_BARS * 8;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_raw + (sMisc - raw));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_raw + (sMisc + 4 - raw));
  volatile int* fail_code = reinterpret_cast<volatile int*>(smem_raw + (sMisc + 8 - raw));
  volatile float* decay_tab = reinterpret_cast<volatile float*>(smem_raw + (sMisc + 16 - raw));
  auto bar = [&](int which, int inst) -> uint32_t { return sBar + (which * NST + inst) * 8; };
  auto stage_of = [](int i) { return NST == 2 ? (i & 1) : i % NST; };                       // stage and barrier instance of block i
  auto parity_of = [](int i) -> uint32_t { return (NST == 2 ? (i >> 1) : i / NST) & 1; };  // and the barriers' phase
  // accumulator of D: the state-only pass alternates between two, so that D of a block does not wait for the readers of the last
  auto t_d = [](int i) -> uint32_t { return MODE == 0 ? T_D : T_D - ((i & 1) ? 256u : 0u); };

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int slice = blockIdx.x;
  const int chunk = p.chunk0 + blockIdx.y;
  const int bh = blockIdx.z;
  const int dv_off = slice * DV;
  const int blk_begin = chunk * p.blocks_per_chunk;
  const int blk_end = min(p.nblocks, blk_begin + p.blocks_per_chunk);
  const int nb = blk_end - blk_begin;
  const int reverse = p.reverse;
  // third tensor-map coordinate of this (batch, head) pair
  const int zc = p.layout ? (bh / p.h) * p.n * p.h + (bh % p.h) : bh;
  const int nk16 = p.dk >> 4;
  const long long budget = p.wait_budget;
  const bool have_state_in = (p.state_in != nullptr);
  // The state group waits for the kernel in front before it touches chunk states or outputs. A bounded wait on anything that follows
  // from there must not start earlier: its budget is for this CTA's own work, and the kernel in front may run for any time (one
  // narrow pair of 60 million tokens in one chunk: longer than the budget). So every role passes the same point before its first
  // such wait; what needs only loads and S of block 0 stays in front of it.
  const bool behind_previous = MODE == 0 || have_state_in;

  const float s = p.slopes ? p.slopes[bh % p.h] : 0.f;
  const float s2 = -s * 1.4426950408889634f;

  pdl_let_next_start();
  la_status_begin(p.status);
  if (tid == 0) {
    for (int i = 0; i < LAP_NUM_BARS; ++i) {
      const uint32_t count = (i == LAP_P_READY) ? LAP_MASK_THREADS
                           : (i == LAP_O_FREE || i == LAP_D_FREE || i == LAP_STATE_READY || i == LAP_O_STAGED) ? LAP_STATE_THREADS
                           : (i == LAP_BM_SCALED) ? LAP_STATE_THREADS + (HELP ? LAP_SCALE_THREADS : 0) : 1u;
      for (int j = 0; j < NST; ++j) mbar_init(bar(i, j), count);
    }
    *abort_flag = 0;
    *fail_code = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
    if (MODE == 0) tma_prefetch_desc(&tmO);
  }
  if (tid < LA_BLOCK) decay_tab[tid] = ex2f(s2 * static_cast<float>(tid));
  if (warp == 0) {
    tmem_alloc(sMisc, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *tmem_slot;

#define LAP_FAIL(code) { if (*fail_code == 0) *fail_code = (code); }
#define LAP_TRACE(slot, it) if (p.trace != nullptr && bh == 0 && blockIdx.x == 0 && blockIdx.y == 0 && (it) < p.trace_blocks) \
    p.trace[(it) * LA_TRACE_SLOTS + (slot)] = clock64();

  if (warp < 4) {
    regs_set<128, LAP_REGS[0]>();
    if (warp == 0) {
      // =========================================== TMA producer ===========================================
      // Also issues the TMA stores of the output tiles: a tile is staged in the C stage of its block (P C, the last MMA of a
      // block, has read C by then), and that stage is reloaded (for block it+2) only after the store has read it.
      if (issuer_lane(lane)) {
        auto blk_of = [&](int i) { return reverse ? (blk_end - 1 - i) : (blk_begin + i); };
        auto store_tile = [&](int i) -> bool {  // output tile of block i: wait until it is staged, then store it
          const int sst = i & 1;
          if (!lap_wait(bar(LAP_O_STAGED, sst), (i >> 1) & 1, abort_flag, budget)) return false;
#pragma unroll
          for (int vs = 0; vs < NVS; ++vs)
            tma_store_3d(&tmO, sC + (sst * NCS + vs) * SLAB, dv_off + vs * 64, blk_of(i) * LA_BLOCK, zc);
          tma_store_commit();
          return true;
        };
        bool alive = true;
        for (int it = 0; it < nb && alive; ++it) {
          const int blk = blk_of(it);
          const int st = stage_of(it);
          const uint32_t prev_par = parity_of(it) ^ 1;  // phase of the previous use of this stage (block it - NST)
          // A and Bm of block it: their stages are free once every MMA of block it-2 has run (P C is the last one issued; in
          // state-only mode D). They are what S of block it waits for, so they go first and wait for nothing else.
          // Where there is one stage, A is free after X of block it-1 and Bm after D of block it-1.
          const uint32_t last_par = parity_of(it - 1);
          auto load_b = [&]() {
#pragma unroll
            for (int ks = 0; ks < NKS; ++ks)
              tma_load_3d(sB + (st * NBS + ks) * SLAB, &tmB, ks * 64, blk * LA_BLOCK, zc, bar(LAP_FULL_AB, st));
          };
          if (behind_previous && it == (NAS == 0 ? 1 : NST)) pdl_wait_for_previous();
          if (NBS != 0 && it >= NST) {
            if (!lap_wait(bar(MODE == 0 ? LAP_PC_DONE : LAP_D_DONE, st), prev_par, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
          }
          mbar_arrive_expect_tx(bar(LAP_FULL_AB, st), (MODE == 0 ? 2 * NKS : NKS) * SLAB);
          if (NBS != 0) load_b();
          if (MODE == 0) {
            if (NAS == 0 && it >= 1 && !lap_wait(bar(LAP_A_FREE, st ^ 1), last_par, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
#pragma unroll
            for (int ks = 0; ks < NKS; ++ks)
              tma_load_3d(sA + (st * NAS + ks) * SLAB, &tmA, ks * 64, blk * LA_BLOCK, zc, bar(LAP_FULL_AB, st));
          }
          if (NBS == 0) {
            if (it >= 1 && !lap_wait(bar(LAP_D_DONE, st ^ 1), last_par, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
            load_b();
          }
          // C of block it: in the full block loop its stage holds the staged output tile of block it-2, which is stored first;
          // C is not needed before D of block it, a whole block later than A and Bm.
          if (MODE == 0 && it >= 2) {
            if (!store_tile(it - 2)) { LAP_FAIL(LA_ERR_WAIT_MMA2) alive = false; break; }
            tma_store_wait_read();
          }
          // Only the slabs of this CTA's dv slice are loaded. D = C^T (w Bm) is an M = 128 MMA and reads both slabs of the stage; with
          // a 64-wide slice the second one holds stale bytes, which only reach accumulator rows >= 64 that nobody reads.
          mbar_arrive_expect_tx(bar(LAP_FULL_C, st), NVS * SLAB);
#pragma unroll
          for (int vs = 0; vs < NVS; ++vs)
            tma_load_3d(sC + (st * NCS + vs) * SLAB, &tmC, dv_off + vs * 64, blk * LA_BLOCK, zc, bar(LAP_FULL_C, st));
        }
        if (MODE == 0 && alive && *abort_flag == 0) {
          pdl_wait_for_previous();  // fewer blocks than stages: not passed yet
          for (int i = max(nb - 2, 0); i < nb; ++i) {
            if (!store_tile(i)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
          }
        }
        if (MODE == 0) tma_store_wait_all();
      }
    } else if (warp == 1) {
      // ============================================ MMA issuer ============================================
      // Issue order per block: X_i, D_i, PC_i, S_{i+1}. X_i and D_i need nothing from the mask group, so they run while
      // it turns S_i into P_i; D_i this early also means the next state is ready long before X_{i+1} asks for it.
      // S_{i+1} overwrites the TMEM columns P_i lives in, so it follows PC_i (the tensor pipe executes in issue order).
      // D and P C commit to their own barriers: the state update starts after D_i, the output tile leaves TMEM after
      // PC_i while S_{i+1}, X_{i+1} and D_{i+1} run.
      if (issuer_lane(lane)) {
        auto issue_S = [&](int i) -> bool {
          const int ist = i & 1;
          if (!lap_wait(bar(LAP_FULL_AB, ist), (i >> 1) & 1, abort_flag, budget)) return false;
          tc_fence_after_sync();
          const uint32_t a0 = sA + ist * NAS * SLAB, b0 = sB + ist * NBS * SLAB;
          for (int kq = 0; kq < nk16; ++kq) {  // S = A Bm^T
            const uint32_t off = (kq >> 2) * SLAB + (kq & 3) * 32;
            umma_f16(tmem + T_S, smem_desc_sw128(a0 + off, 16), smem_desc_sw128(b0 + off, 16), IDESC_S, kq > 0);
          }
          umma_commit(bar(LAP_S_READY, ist));
          return true;
        };
        bool alive = true;
        if (MODE == 0 && nb > 0) {
          alive = issue_S(0);
          if (!alive) LAP_FAIL(LA_ERR_WAIT_INPUT)
        }
        if (behind_previous) pdl_wait_for_previous();
        for (int it = 0; it < nb && alive; ++it) {
          const int st = stage_of(it);
          const uint32_t par = parity_of(it);
          const int pst = stage_of(it - 1);               // instance used by block it-1
          const uint32_t ppar = parity_of(it - 1);        // and its phase
          const uint32_t sAs = sA + st * NAS * SLAB, sBs = sB + st * NBS * SLAB, sCs = sC + st * NCS * SLAB;
          const bool have_state = have_state_in || (it > 0);
          LAP_TRACE(0, it)
          if (MODE == 0) {
            if (have_state) {
              if (!lap_wait(bar(LAP_STATE_READY, st), par, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
              if (it > 0 && !lap_wait(bar(LAP_O_FREE, pst), ppar, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
              tc_fence_after_sync();
              for (int kq = 0; kq < nk16; ++kq) {  // X = A State
                const uint32_t offA = (kq >> 2) * SLAB + (kq & 3) * 32;
                if constexpr (WIDE) {
                  umma_f16(tmem + T_OX, smem_desc_sw128(sAs + offA, 16), smem_desc_sw128(sS + kq * 2048, SLAB), IDESC_PC, kq > 0);
                } else {
                  const uint32_t offS = (kq >> 2) * (DV * 128) + (kq & 3) * 32;
                  umma_f16(tmem + T_OX, smem_desc_sw128(sAs + offA, 16), smem_desc_sw128(sS + offS, 16), IDESC_X, kq > 0);
                }
              }
            }
            if (WIDE) umma_commit(bar(LAP_A_FREE, st));  // S and X of this block are done with A
            LAP_TRACE(1, it)
          }
          if (MODE != 0 && !lap_wait(bar(LAP_FULL_AB, st), par, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_INPUT) break; }
          if (!lap_wait(bar(LAP_FULL_C, st), par, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_INPUT) break; }
          if (!lap_wait(bar(LAP_BM_SCALED, st), par, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
          if (MODE == 0) {
            if (it > 0 && !lap_wait(bar(LAP_D_FREE, pst), ppar, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
          } else if (it > 1 && !lap_wait(bar(LAP_D_FREE, stage_of(it - 2)), parity_of(it - 2), abort_flag, budget)) {
            LAP_FAIL(LA_ERR_WAIT_MMA2) break;
          }
          tc_fence_after_sync();
          if constexpr (WIDE) {
#pragma unroll
            for (int kk = 0; kk < 16; ++kk)  // local State = (w_state Bm)^T C, dk rows 0-127 and 128-255
              umma_f16(tmem + t_d(it) + (kk >> 3) * DV, smem_desc_sw128(sBs + (kk >> 3) * 2 * SLAB + (kk & 7) * 2048, SLAB),
                       smem_desc_sw128(sCs + (kk & 7) * 2048, SLAB), IDESC_ST, (kk & 7) > 0);
          } else {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)  // local StateT = C^T (w_state Bm)
              umma_f16(tmem + t_d(it), smem_desc_sw128(sCs + kk * 2048, SLAB), smem_desc_sw128(sBs + kk * 2048, SLAB), IDESC_ST, kk > 0);
          }
          umma_commit(bar(LAP_D_DONE, st));  // also: X_it is done with the bf16 state copy
          LAP_TRACE(3, it)
          if (MODE == 0) {
            if (!lap_wait(bar(LAP_P_READY, st), par, abort_flag, budget)) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
            LAP_TRACE(2, it)
            tc_fence_after_sync();
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)  // O_intra = P C, P read from TMEM
              umma_f16_ts(tmem + T_OI, tmem + T_S + kk * 8, smem_desc_sw128(sCs + kk * 2048, SLAB), IDESC_PC, kk > 0);
            umma_commit(bar(LAP_PC_DONE, st));  // O_intra and O_inter are complete; nothing reads A, Bm, C of this block any more
            if (it + 1 < nb) {
              if (!issue_S(it + 1)) { LAP_FAIL(LA_ERR_WAIT_INPUT) break; }
            }
          }
        }
      }
    } else if (HELP) {
      // ============================================ scaling ===============================================
      // The state group is the busiest role: state update, output tile, then the scaling that the next D waits for (clock stamps of
      // b4 h32 n2048 d=e=128: 3,600 of a block's 4,750 cycles; 4,350 with this). These two warps take half of every row of Bm (positions
      // rot + 4 .. rot + 7 of each slab) as soon as S is done with it, two rows per thread. Forward 51.4 -> 49.7 us.
      const int r0 = (warp - 2) * 32 + lane;
      const int tail = p.n - (p.nblocks - 1) * LA_BLOCK;
      const bool tail_fix = !reverse && tail < LA_BLOCK && blk_end == p.nblocks;  // see the state group
      const float wa = ex2f(s2 * static_cast<float>(reverse ? r0 : LA_BLOCK - r0));
      const float wb = ex2f(s2 * static_cast<float>(reverse ? r0 + 64 : LA_BLOCK - 64 - r0));
      for (int j = 0; j < nb; ++j) {
        const int st = stage_of(j);
        bool ok = lap_wait(bar(LAP_S_READY, st), parity_of(j), abort_flag, budget);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { LAP_FAIL(LA_ERR_WAIT_MMA1) break; }
        if (s != 0.f) {
          float w0 = wa, w1 = wb;
          if (tail_fix && j == nb - 1) {
            w0 = r0 < tail ? ex2f(s2 * static_cast<float>(tail - r0)) : 0.f;
            w1 = r0 + 64 < tail ? ex2f(s2 * static_cast<float>(tail - r0 - 64)) : 0.f;
          }
          const uint32_t row = sB + st * NBS * SLAB + r0 * 128;
#pragma unroll 1
          for (int ks = 0; ks < NKS; ++ks) {
            lap_scale<FMT, false, 4>(row + ks * SLAB, r0 + 4, w0);
            lap_scale<FMT, false, 4>(row + ks * SLAB + 64 * 128, r0 + 4, w1);
          }
          fence_proxy_async_smem();
        }
        mbar_arrive(bar(LAP_BM_SCALED, st));
        if (j == 0) pdl_wait_for_previous();
      }
    }
  } else if (warp < 8) {
    regs_set<128, LAP_REGS[1]>();
    // ============================================ mask group ============================================
    // One warp per TMEM lane quadrant, four 32-column tiles each, in column order. P tile t goes back into TMEM at
    // columns [16 t, 16 t + 16), i.e. over S columns of S tile t/2 <= t, which the warp has already pulled into
    // registers by then.
    if (MODE == 0) {
      const int q = warp & 3;
      const int r = q * 32 + lane;
      const uint32_t lanebase = static_cast<uint32_t>(q * 32) << 16;
      const bool tracer = lane == 0 && q == (reverse ? 0 : 3);  // the quadrant with the most unmasked tiles
      float g[32];  // per-column part of the decay inside a live tile: lambda^i (reverse) or lambda^(31-i) (forward)
#pragma unroll
      for (int i = 0; i < 32; ++i) g[i] = ex2f(s2 * static_cast<float>(reverse ? i : 31 - i));
      // Diagonal tile: lambda^(lane-i) = g[i] * lambda^(lane-31) (forward), lambda^(i-lane) = g[i] * lambda^(-lane) (reverse).
      // The row factor is >= 1 here, at most lambda^-31; for decay rates where that could leave the fp32 range the
      // per-element table is used instead (CTA-uniform choice).
      const bool diag_rank1 = s * 31.f < 60.f;
      const float rowd = diag_rank1 ? ex2f(s2 * static_cast<float>(reverse ? -lane : lane - 31)) : 0.f;
      for (int it = 0; it < nb; ++it) {
        const int st = it & 1;
        const uint32_t par = (it >> 1) & 1;
        bool ok = lap_wait(bar(LAP_S_READY, st), par, abort_flag, budget);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { LAP_FAIL(LA_ERR_WAIT_MMA1) break; }
        if (tracer) { LAP_TRACE(4, it) }
        tc_fence_after_sync();
        // kind of tile t for this quadrant: 0 dead (all masked), 1 live (nothing masked), 2 diagonal; warp-uniform
        auto tile_kind = [&](int t) { return (t == q) ? 2 : ((reverse ? (t > q) : (t < q)) ? 1 : 0); };
#pragma unroll 1
        for (int t = 0; t < 4; ++t) {
          const int c0 = t * 32;
          const int kind = tile_kind(t);
          uint32_t v[1][32];
          if (kind) {
            tmem_ld32(tmem + lanebase + T_S + c0, v[0]);
            tmem_wait_ld();
          }
          uint32_t pk[16];
          if (kind == 1) {
            // lambda^|r-c| = (per-row part, one table look-up) x (per-column part g[i]); both factors are <= 1
            const float rowf = decay_tab[reverse ? (c0 - r) : (r - c0 - 31)];
#pragma unroll
            for (int i = 0; i < 32; i += 2)
              pk[i >> 1] = pack2<FMT>(__uint_as_float(v[0][i]) * (rowf * g[i]), __uint_as_float(v[0][i + 1]) * (rowf * g[i + 1]));
          } else if (kind == 2 && diag_rank1) {
            float rd = rowd;
            asm volatile("" : "+f"(rd));  // keeps the 32 products rd * g[i] from being hoisted out of the block loop into registers
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const int d0 = reverse ? (i - lane) : (lane - i);
              const int d1 = reverse ? (d0 + 1) : (d0 - 1);
              const float f0 = (d0 >= 0) ? __uint_as_float(v[0][i]) * (rd * g[i]) : 0.f;
              const float f1 = (d1 >= 0) ? __uint_as_float(v[0][i + 1]) * (rd * g[i + 1]) : 0.f;
              pk[i >> 1] = pack2<FMT>(f0, f1);
            }
          } else if (kind == 2) {
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const int d0 = reverse ? (i - lane) : (lane - i);
              const int d1 = reverse ? (d0 + 1) : (d0 - 1);
              const float m0 = decay_tab[max(d0, 0)], m1 = decay_tab[max(d1, 0)];
              const float f0 = (d0 >= 0) ? __uint_as_float(v[0][i]) * m0 : 0.f;
              const float f1 = (d1 >= 0) ? __uint_as_float(v[0][i + 1]) * m1 : 0.f;
              pk[i >> 1] = pack2<FMT>(f0, f1);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[i] = 0u;
          }
          tmem_st16(tmem + lanebase + T_S + t * 16, pk);
        }
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(bar(LAP_P_READY, st));
        if (tracer) { LAP_TRACE(5, it) }
        if (it == 0) pdl_wait_for_previous();
      }
    }
  } else {
    // ========================================= state / output group =====================================
    regs_set<128, LAP_REGS[2]>();
    const int w8 = warp - 8;
    const int q = warp & 3, hf = w8 >> 2;
    const int r = q * 32 + lane;
    const uint32_t lanebase = static_cast<uint32_t>(q * 32) << 16;
    const float w_out = reverse ? ex2f(s2 * static_cast<float>(LA_BLOCK - r)) : ex2f(s2 * static_cast<float>(r));
    const float decay_blk = ex2f(s2 * static_cast<float>(LA_BLOCK));
    const float w_state = reverse ? ex2f(s2 * static_cast<float>(r)) : ex2f(s2 * static_cast<float>(LA_BLOCK - r));
    // A forward-time sweep that ends in a ragged block (n not a multiple of 128): the state leaving that block is decayed
    // to token n, not to the end of the 128-token tile, so that state_out chains exactly (rows >= tail are zero padding).
    const int tail = p.n - (p.nblocks - 1) * LA_BLOCK;
    const bool tail_fix = !reverse && tail < LA_BLOCK && blk_end == p.nblocks;
    const float w_tail = (tail_fix && r < tail) ? ex2f(s2 * static_cast<float>(tail - r)) : 0.f;
    const float decay_tail = ex2f(s2 * static_cast<float>(tail));
    // this thread's part of the state: row r (dv), columns hf SC + i (dk); wide: row hf 128 + r (dk), columns i (dv)
    const int st_row = WIDE ? hf * 128 + r : r;
    const bool st_warp = WIDE ? (hf * 128 + q * 32 < DKP) : (q * 32 < DV);  // the accumulator lanes of this warp hold state rows
    const bool st_row_valid = WIDE ? (st_row < p.dk) : ((r < DV) && (dv_off + r < p.dv));
    const bool store_thread = (w8 == 0 && lane == 0);

    // The tensors of the call are complete before its first kernel starts; the states are written by the kernels in front of this one.
    // Output tiles and scaled copies follow this in program order.
    if (behind_previous) pdl_wait_for_previous();
    float stt[SC];
#pragma unroll
    for (int i = 0; i < SC; ++i) stt[i] = 0.f;
    if (have_state_in && st_row_valid) {
      const float* src = p.state_in + (static_cast<size_t>(bh) * p.state_slots + chunk) * p.dv * p.dk;
      const bool swapped = MODE == 0 && p.in_swapped;
      const int ld = swapped ? p.dv : p.dk, cols = WIDE ? p.dv - dv_off : p.dk - hf * SC;
      if (WIDE != swapped) {  // this thread's part is a column of the stored matrix: neighbouring lanes read neighbouring elements
        src += WIDE ? static_cast<size_t>(dv_off) * ld + st_row : static_cast<size_t>(hf * SC) * ld + dv_off + r;
#pragma unroll
        for (int i = 0; i < SC; ++i)
          if (i < cols) stt[i] = src[static_cast<size_t>(i) * ld];
      } else {
        src += WIDE ? static_cast<size_t>(st_row) * ld + dv_off : static_cast<size_t>(dv_off + r) * ld + hf * SC;
#pragma unroll
        for (int i = 0; i < SC; i += 4) {
          if (i < cols) {
            const float4 v4 = *reinterpret_cast<const float4*>(src + i);
            stt[i] = v4.x; stt[i + 1] = v4.y; stt[i + 2] = v4.z; stt[i + 3] = v4.w;
          }
        }
      }
    }
    auto store_state_smem = [&]() {
      if (WIDE ? st_warp : (r < DV)) {
#pragma unroll
        for (int i = 0; i < SC; i += 8) {
          const int col = WIDE ? i : hf * SC + i;
          const uint32_t addr = sS + (col >> 6) * (DV * 128) + st_row * 128 + ((((col & 63) >> 3) ^ (r & 7)) << 4);
          st_shared_v4(addr, pack2<FMT>(stt[i], stt[i + 1]), pack2<FMT>(stt[i + 2], stt[i + 3]),
                       pack2<FMT>(stt[i + 4], stt[i + 5]), pack2<FMT>(stt[i + 6], stt[i + 7]));
        }
      }
    };
    if (MODE == 0) {
      if (have_state_in) {
        store_state_smem();
        fence_proxy_async_smem();
      }
      mbar_arrive(bar(LAP_STATE_READY, 0));  // state entering block 0
    }

    // Bm rows of block j *= w_state(r), in place, for D_j: this thread's share of the row, or of the half that warps 2 and 3 leave.
    auto scale_bm = [&](int j) -> bool {
      const int st = stage_of(j);
      // S_j must be done with the unscaled tile (state-only mode: the tile must have landed)
      bool ok = lap_wait(bar(MODE == 0 ? LAP_S_READY : LAP_FULL_AB, st), parity_of(j), abort_flag, budget);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return false;
      if (s != 0.f) {
        const float w = (tail_fix && j == nb - 1) ? w_tail : w_state;
        const uint32_t row = sB + st * NBS * SLAB + r * 128;
        if constexpr (NKS == 2) {
          lap_scale<FMT, false, HELP ? 4 : 8>(row + hf * SLAB, r, w);
        } else {
#pragma unroll 1
          for (int ks = 0; ks < NKS; ++ks) lap_scale<FMT, WIDE, HELP ? 2 : 4>(row + ks * SLAB, hf * (HELP ? 2 : 4) + r, w);
        }
        fence_proxy_async_smem();
      }
      mbar_arrive(bar(LAP_BM_SCALED, st));
      if (store_thread) { LAP_TRACE(6, j) }
      return true;
    };
    // Order of work per block it: state update (after D_it), output tile (after PC_it), Bm scaling for block it+1
    // (after S_{it+1}) - the order in which the MMA warp completes them.
    bool live = true;
    if (nb > 0) {
      live = scale_bm(0);
      if (!live) LAP_FAIL(LA_ERR_WAIT_MMA1)
    }
    for (int it = 0; it < nb && live; ++it) {
      const int st = stage_of(it);
      const uint32_t par = parity_of(it);
      const bool has_next = (it + 1 < nb);
      const bool have_state = have_state_in || (it > 0);
      // state-only mode: the next block's Bm tile is scaled while D of this block runs
      if (MODE != 0 && has_next && !scale_bm(it + 1)) { LAP_FAIL(LA_ERR_WAIT_MMA1) break; }
      {
        bool ok = lap_wait(bar(LAP_D_DONE, st), par, abort_flag, budget);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
      }
      if (store_thread) { LAP_TRACE(8, it) }
      tc_fence_after_sync();
      // ---- state recurrence --------------------------------------------------------------------------
      if (st_warp) {
#pragma unroll
        for (int cc = 0; cc < SC; cc += 32) {
          uint32_t dl[32];
          tmem_ld32(tmem + lanebase + t_d(it) + hf * SC + cc, dl);
          tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i)
            stt[cc + i] = fmaf((tail_fix && it == nb - 1) ? decay_tail : decay_blk, stt[cc + i], __uint_as_float(dl[i]));
        }
      }
      tc_fence_before_sync();
      mbar_arrive(bar(LAP_D_FREE, st));
      if (MODE == 0 && has_next) {
        // X_it was issued before D_it, so it is done with the old bf16 copy of the state
        store_state_smem();
        fence_proxy_async_smem();
        mbar_arrive(bar(LAP_STATE_READY, st ^ 1));  // state entering block it+1
      }
      if (store_thread) { LAP_TRACE(9, it) }
      if (MODE == 0) {
        // ---- output tile: TMEM -> registers -> swizzled shared-memory slabs -> TMA store. Runs while S_{it+1},
        //      X_{it+1} and D_{it+1} are in the tensor pipe. --------------------------------------------------------------
        bool ok = lap_wait(bar(LAP_PC_DONE, st), par, abort_flag, budget);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) { LAP_FAIL(LA_ERR_WAIT_MMA2) break; }
        if (store_thread) { LAP_TRACE(7, it) }
        tc_fence_after_sync();
        const uint32_t sOs = sC + st * NCS * SLAB;  // P C and D of this block are done with this C stage
#pragma unroll
        for (int cc = 0; cc < OC; cc += 16) {
          uint32_t a[16], b[16];
          tmem_ld16(tmem + lanebase + T_OI + hf * OC + cc, a);
          if (have_state) tmem_ld16(tmem + lanebase + T_OX + hf * OC + cc, b);
          tmem_wait_ld();
          if (cc + 16 >= OC) {  // last read of this block's accumulators
            tc_fence_before_sync();
            mbar_arrive(bar(LAP_O_FREE, st));
            if (store_thread) { LAP_TRACE(10, it) }
          }
#pragma unroll
          for (int g = 0; g < 2; ++g) {
            uint32_t o4[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float x0 = __uint_as_float(a[g * 8 + 2 * j]), x1 = __uint_as_float(a[g * 8 + 2 * j + 1]);
              if (have_state) {
                x0 = fmaf(w_out, __uint_as_float(b[g * 8 + 2 * j]), x0);
                x1 = fmaf(w_out, __uint_as_float(b[g * 8 + 2 * j + 1]), x1);
              }
              o4[j] = pack2<FMT>(x0, x1);
            }
            const int col = hf * OC + cc + g * 8;  // column inside this CTA's dv slice
            st_shared_v4(sOs + (col >> 6) * SLAB + r * 128 + ((((col & 63) >> 3) ^ (r & 7)) << 4), o4[0], o4[1], o4[2], o4[3]);
          }
        }
        fence_proxy_async_smem();
        mbar_arrive(bar(LAP_O_STAGED, st));  // the producer warp stores the tile
        if (store_thread) { LAP_TRACE(11, it) }
      }
      if (MODE == 0 && has_next && !scale_bm(it + 1)) { LAP_FAIL(LA_ERR_WAIT_MMA1) break; }
    }
    if (MODE != 0) pdl_wait_for_previous();  // the kernel in front may still be reading the states of the product before
    if (*abort_flag == 0 && p.state_out != nullptr && st_row_valid) {
      float* dst = p.state_out + (static_cast<size_t>(bh) * p.state_slots + chunk) * p.dv * p.dk;
      if constexpr (WIDE) {
        dst += static_cast<size_t>(dv_off) * p.dk + st_row;
#pragma unroll
        for (int i = 0; i < SC; ++i)
          if (dv_off + i < p.dv) dst[static_cast<size_t>(i) * p.dk] = stt[i];
      } else {
        dst += static_cast<size_t>(dv_off + r) * p.dk + hf * SC;
#pragma unroll
        for (int i = 0; i < SC; i += 4) {
          if (hf * SC + i < p.dk) *reinterpret_cast<float4*>(dst + i) = make_float4(stt[i], stt[i + 1], stt[i + 2], stt[i + 3]);
        }
      }
    }
  }
#undef LAP_TRACE
#undef LAP_FAIL

  tc_fence_before_sync();
  __syncthreads();
  if (tid == 0 && *abort_flag) la_status_report(p.status, *fail_code ? *fail_code : LA_ERR_WAIT_MMA2);
  if (warp == 0) {
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace lab200
