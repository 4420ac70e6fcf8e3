// Lightning Attention-2 device kernels for sm_100a.
//
// One generic kernel covers the forward pass and all three gradients. For row-major inputs
// A (n x dk, "query-like"), Bm (n x dk, "key-like"), C (n x dv, "value-like") of one (batch, head)
// pair and decay rate s (lambda = exp(-s)) it computes, in forward time order,
//
//     out_t = sum_{j <= t} lambda^(t-j) (A_t . Bm_j) C_j                    (reverse = 0)
//
// or, in reverse time order,
//
//     out_t = sum_{j >= t} lambda^(j-t) (A_t . Bm_j) C_j                    (reverse = 1)
//
// The reference computes the same quantities with three Triton kernels
// (lightning_attn/ops/triton/lightning_attn2.py:8-85 forward, :88-183 in-block gradients,
// :186-395 cross-block gradients). With (A,Bm,C) = (q,k,v) forward time gives o; (do,v,k) forward
// time gives dq; (v,do,q) reverse time gives dk; (k,q,do) reverse time gives dv.
//
// The sequence is cut into blocks of 128 tokens. Per block (r, c = row indices inside the block):
//     S      = A Bm^T                                   tcgen05.mma, fp32 in TMEM
//     P      = S (.) M,  M[r,c] = lambda^|r-c| on the causal side, 0 elsewhere   (CUDA cores, back into TMEM)
//     O      = P C + diag(w_out) A State                two tcgen05.mma chains, combined in the epilogue
//     StateT = lambda^128 StateT + C^T (diag(w_state) Bm)   tcgen05.mma + fp32 registers
// with w_out(r) = lambda^r, w_state(r) = lambda^(128-r) in forward time and the two swapped in
// reverse time (lightning_attn2.py:47-48, :352-358, :392-395). StateT (dv x dk, the transposed
// d x e "KV" state of the reference) lives in fp32 registers for the whole block loop; a rounded
// copy in shared memory feeds the tensor cores.
//
// Shared-memory tiles are [128 tokens][64 features] slabs with the 128-byte swizzle, exactly as TMA
// writes them; the same slab serves as a K-major operand (contraction over features) and as an
// MN-major operand (contraction over tokens), so no transposes are ever materialised.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "ptx_sm100.cuh"

namespace lab200 {

constexpr int LA_BLOCK = 128;        // tokens per block
constexpr int LA_SLAB_BYTES = 16384; // 128 rows x 128 bytes
constexpr int LA_TRACE_SLOTS = 16;    // clock stamps per block in the optional trace buffer

enum LaError : int {
  LA_OK = 0,
  LA_ERR_WAIT_INPUT = 101,  // TMA bytes never arrived
  LA_ERR_WAIT_MMA1 = 102,   // first MMA group never completed
  LA_ERR_WAIT_MMA2 = 103,   // second MMA group never completed
};

// Where a CTA whose bounded wait ran out reports it: `word`, the status word in front of the call's workspace, and `host`,
// the device's word in pinned host memory that lab200_last_status() reads (nullptr: none). `reset` is set for the first block
// kernel of a call, whose CTA (0, 0, 0) then clears the word: no memset launch in front of every call and no 4-byte copy
// behind it (together ~10 us of stream time per call: 1.5 + 3.3 us of work and the switches to the copy engine and back).
// The clearing store cannot overtake a report: block (0, 0, 0) is dispatched first and stores within microseconds of
// starting, while a report follows a wait of ~1 s.
struct LaStatus {
  int* word;
  int* host;
  int reset;
};
__device__ __forceinline__ void la_status_begin(const LaStatus& s) {
  if (s.reset && (threadIdx.x | blockIdx.x | blockIdx.y | blockIdx.z) == 0) *const_cast<volatile int*>(s.word) = 0;
}
__device__ __forceinline__ void la_status_report(const LaStatus& s, int code) {
  atomicExch(s.word, code);
  if (s.host) {
    *const_cast<volatile int*>(s.host) = code;
    __threadfence_system();
  }
}

struct LaParams {
  const float* slopes;     // [h] decay rates, or nullptr for no decay
  const float* state_in;   // [bh][state_slots][dv][dk] fp32, or nullptr for a zero initial state
  float* state_out;        // same indexing, or nullptr
  int in_swapped;          // the matrices of state_in are stored [dk][dv]: they come from the product with Bm and C exchanged (block loop)
  LaStatus status;         // where a failure is reported
  int n, h, dk, dv;
  int nblocks;             // ceil(n / 128)
  int blocks_per_chunk;
  int chunk0;              // chunk handled by blockIdx.y == 0
  int state_slots;         // chunk slots per (batch, head) in state_in / state_out
  int reverse;
  int layout;              // 0: tensors are (b, h, n, dim) contiguous; 1: (b, n, h, dim) contiguous:
                           // the tensor maps then index their third dimension by batch * n * h + head, see make_tmap
  long long wait_budget;   // clock cycles after which a barrier wait gives up
  long long* trace;        // optional: CTA (0,0,0) records clock64() stamps here, LA_TRACE_SLOTS per block
  int trace_blocks;        // capacity of `trace` in blocks
};

template <int FMT>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (FMT == 1) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}
// packed multiply of two 16-bit pairs (rounds once per element, in the 16-bit format)
template <int FMT>
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
  if constexpr (FMT == 1) {
    __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a), *reinterpret_cast<__nv_bfloat162*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
  } else {
    __half2 r = __hmul2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
  }
}
template <int FMT>
__device__ __forceinline__ float2 unpack2(uint32_t u) {
  if constexpr (FMT == 1) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
  } else {
    return __half22float2(*reinterpret_cast<__half2*>(&u));
  }
}

// Exclusive decayed scan over the per-chunk local states, in place:
//   forward time:  prefix[c] = run;  run = lambda^(tokens in chunk c) * run + local[c]   for c = 0..nchunks-1
//   reverse time:  the same for c = nchunks-1..0.
// `init` seeds `run` (state arriving from outside the sequence), `total` receives the final run.
// The reference's unfinished "parallel" variant does the same with one program per head
// (lightning_attn2_parallel.py:198-249, :650-701); here every state element is an independent thread.
// When `skip_last` is set the local state of the last chunk in scan order was not computed and is ignored.
// The chain over chunks is a multiply-add per step, so what bounds the kernel is the latency of its loads: a thread owns four
// neighbouring elements (one 16-byte access per chunk) and has the local states of eight chunks in flight before it starts
// the chain. With one element and one dependent load per step, 4 chunks of 32 pairs of 128 x 128 took 19 us, now 6.
constexpr int LA_SCAN_AHEAD = 8;
__global__ void __launch_bounds__(256)
la_scan_kernel(float4* __restrict__ states, const float4* __restrict__ init, float4* __restrict__ total,
               const float* __restrict__ slopes, int h, int nchunks, int elems4, int nblocks, int blocks_per_chunk, int n,
               int reverse, int skip_last, long long total4) {
  pdl_let_next_start();
  pdl_wait_for_previous();
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= total4) return;
  const int bh = static_cast<int>(idx / elems4);
  const int e = static_cast<int>(idx - static_cast<long long>(bh) * elems4);
  const float s = slopes ? slopes[bh % h] : 0.f;
  float4 run = init ? init[idx] : make_float4(0.f, 0.f, 0.f, 0.f);
  // tokens of a full chunk, and of the chunk that holds the end of the sequence. Forward time: that chunk may end in a ragged
  // block, and its local state is decayed to token n (see the block kernels).
  const int full = blocks_per_chunk * LA_BLOCK, edge_begin = (nchunks - 1) * blocks_per_chunk;
  const int edge = reverse ? (nblocks - edge_begin) * LA_BLOCK : n - edge_begin * LA_BLOCK;
  const float lam_full = __expf(-s * static_cast<float>(full)), lam_edge = __expf(-s * static_cast<float>(edge));
  float4* base = states + static_cast<size_t>(bh) * nchunks * elems4 + e;
  for (int k0 = 0; k0 < nchunks; k0 += LA_SCAN_AHEAD) {
    float4 loc[LA_SCAN_AHEAD];
#pragma unroll
    for (int j = 0; j < LA_SCAN_AHEAD; ++j) {
      const int k = k0 + j, c = reverse ? (nchunks - 1 - k) : k;
      loc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < nchunks && !(skip_last && k == nchunks - 1)) loc[j] = base[static_cast<size_t>(c) * elems4];
    }
#pragma unroll
    for (int j = 0; j < LA_SCAN_AHEAD; ++j) {
      const int k = k0 + j, c = reverse ? (nchunks - 1 - k) : k;
      if (k < nchunks) {
        base[static_cast<size_t>(c) * elems4] = run;
        const float lam = (c == nchunks - 1) ? lam_edge : lam_full;
        run = make_float4(fmaf(lam, run.x, loc[j].x), fmaf(lam, run.y, loc[j].y), fmaf(lam, run.z, loc[j].z), fmaf(lam, run.w, loc[j].w));
      }
    }
  }
  if (total) total[idx] = run;
}

// Adds a state that arrives from outside the sequence to per-chunk prefix states that were computed from a zero
// initial state: prefix[c] += lambda^(tokens between the sequence edge and chunk c) * init. Lets a caller compute the
// local states first, learn the incoming state later (sequence parallelism) and still run the chunk pass only once.
__global__ void la_rebase_kernel(float* __restrict__ states, const float* __restrict__ init,
                                 const float* __restrict__ slopes, int h, int nchunks, int elems, int nblocks,
                                 int blocks_per_chunk, int reverse, long long total_elems) {
  const long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= total_elems) return;
  const int bh = static_cast<int>(idx / elems);
  const int e = static_cast<int>(idx - static_cast<long long>(bh) * elems);
  const float s = slopes ? slopes[bh % h] : 0.f;
  const float v = init[idx];
  for (int c = 0; c < nchunks; ++c) {
    const int before = reverse ? (nblocks - min(nblocks, (c + 1) * blocks_per_chunk)) : c * blocks_per_chunk;
    states[(static_cast<size_t>(bh) * nchunks + c) * elems + e] += __expf(-s * static_cast<float>(before * LA_BLOCK)) * v;
  }
}

// State entering this rank's sequence shard from the all-gathered local shard states (sequence parallelism):
//   forward time:  out = sum_{r < rank} lambda^((rank-1-r) L) gathered[r]
//   reverse time:  out = sum_{r > rank} lambda^((r-rank-1) L) gathered[r]
// gathered is (R, bh, X, Y) fp32, L the tokens per shard. `out` (bh, X, Y) and/or `out_t` (bh, Y, X, the same state
// for the product with Bm and C exchanged) may be null. Grid (ceil(Y/32), ceil(X/32), bh), block (32, 8).
__global__ void la_combine_kernel(const float* __restrict__ gathered, const float* __restrict__ slopes,
                                  float* __restrict__ out, float* __restrict__ out_t, int R, int rank, int bh_total, int h,
                                  int X, int Y, float shard_tokens, int reverse) {
  __shared__ float tile[32][33];
  const int bh = blockIdx.z;
  const int x0 = blockIdx.y * 32, y0 = blockIdx.x * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const float s = slopes ? slopes[bh % h] : 0.f;
  const int r_begin = reverse ? rank + 1 : 0, r_end = reverse ? R : rank;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  const int y = y0 + tx;
  for (int r = r_begin; r < r_end; ++r) {
    const int expo = reverse ? (r - rank - 1) : (rank - 1 - r);
    const float w = expf(-s * shard_tokens * static_cast<float>(expo));
    const float* src = gathered + (static_cast<size_t>(r) * bh_total + bh) * X * Y;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int x = x0 + ty + 8 * k;
      if (x < X && y < Y) acc[k] = fmaf(w, src[static_cast<size_t>(x) * Y + y], acc[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int x = x0 + ty + 8 * k;
    if (out && x < X && y < Y) out[(static_cast<size_t>(bh) * X + x) * Y + y] = acc[k];
    tile[ty + 8 * k][tx] = acc[k];
  }
  if (out_t) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int yy = y0 + ty + 8 * k, xx = x0 + tx;  // out_t[yy][xx] = state[xx][yy]
      if (yy < Y && xx < X) out_t[(static_cast<size_t>(bh) * Y + yy) * X + xx] = tile[tx][ty + 8 * k];
    }
  }
}

// In-place transpose of `count` square D x D fp32 matrices stored back to back (the per-chunk states of a product,
// turned into those of the product with Bm and C exchanged). Grid (count, tile pairs i <= j), block (32, 8).
__global__ void la_transpose_square_kernel(float* __restrict__ m, int D) {
  __shared__ float ta[32][33], tb[32][33];
  const int nt = (D + 31) / 32;
  int pair = blockIdx.y, ti = 0;
  for (; ti < nt && pair >= nt - ti; ++ti) pair -= nt - ti;  // row ti of the upper triangle of tile pairs
  if (ti >= nt) return;
  const int tj = ti + pair;
  float* base = m + static_cast<size_t>(blockIdx.x) * D * D;
  const int tx = threadIdx.x, ty = threadIdx.y;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = ty + 8 * k;
    const int ai = ti * 32 + r, aj = tj * 32 + tx;  // tile (ti, tj)
    const int bi = tj * 32 + r, bj = ti * 32 + tx;  // tile (tj, ti)
    ta[r][tx] = (ai < D && aj < D) ? base[static_cast<size_t>(ai) * D + aj] : 0.f;
    tb[r][tx] = (bi < D && bj < D) ? base[static_cast<size_t>(bi) * D + bj] : 0.f;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = ty + 8 * k;
    const int ai = ti * 32 + r, aj = tj * 32 + tx;
    const int bi = tj * 32 + r, bj = ti * 32 + tx;
    if (ai < D && aj < D) base[static_cast<size_t>(ai) * D + aj] = tb[tx][r];
    if (ti != tj && bi < D && bj < D) base[static_cast<size_t>(bi) * D + bj] = ta[tx][r];
  }
}

// One decode step of the recurrence for every (batch, head) pair (inference; no counterpart in the reference):
//   o = q (S + k^T v),   S <- lambda (S + k^T v),
// S being the (dv, dk) fp32 state entering the token (what the block kernels hand out as state_out). HBM-bound on the state,
// 8 bytes per element. Every state element is read once and written back once, so both go in 256-bit accesses marked
// evict-first: 256 sequences x 32 heads x 128 x 128 take 156 us = 6.9 TB/s, 162 without the mark, 194 with 16-byte accesses.
// CTAs are small and rows per warp few, because a CTA's loads, reduction and stores do not overlap each other: 256 threads with
// the same rows per warp take 164 us, 64 x 64 states 111 against 80 us (16-byte accesses, 8 rows per warp, 256 threads: 157).
constexpr int LA_DECODE_THREADS = 128;
constexpr int LA_DECODE_R = 4;  // row accesses in flight per lane

template <int W> struct LaStateVec { float f[4 * W]; };
__device__ __forceinline__ void la_state_ld(LaStateVec<2>& v, const float* p) {
  asm volatile("ld.global.L1::no_allocate.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v.f[0]), "=f"(v.f[1]), "=f"(v.f[2]), "=f"(v.f[3]), "=f"(v.f[4]), "=f"(v.f[5]), "=f"(v.f[6]), "=f"(v.f[7])
               : "l"(p));
}
__device__ __forceinline__ void la_state_st(float* p, const LaStateVec<2>& v) {
  asm volatile("st.global.L1::no_allocate.L2::evict_first.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v.f[0]), "f"(v.f[1]),
               "f"(v.f[2]), "f"(v.f[3]), "f"(v.f[4]), "f"(v.f[5]), "f"(v.f[6]), "f"(v.f[7]) : "memory");
}
__device__ __forceinline__ void la_state_ld(LaStateVec<1>& v, const float* p) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v.f[0] = t.x; v.f[1] = t.y; v.f[2] = t.z; v.f[3] = t.w;
}
__device__ __forceinline__ void la_state_st(float* p, const LaStateVec<1>& v) {
  *reinterpret_cast<float4*>(p) = make_float4(v.f[0], v.f[1], v.f[2], v.f[3]);
}

template <int FMT>
__device__ __forceinline__ uint16_t to_16bit(float x) {
  if constexpr (FMT == 1) {
    const __nv_bfloat16 b = __float2bfloat16_rn(x);
    return *reinterpret_cast<const uint16_t*>(&b);
  } else {
    const __half hh = __float2half_rn(x);
    return *reinterpret_cast<const uint16_t*>(&hh);
  }
}
template <int FMT>
__device__ __forceinline__ float from_16bit(uint16_t x) {
  if constexpr (FMT == 1) return __uint_as_float(static_cast<uint32_t>(x) << 16);
  else return __half2float(__ushort_as_half(x));
}

// Grid (ceil(dv / rows per CTA), bh). LPR lanes share a state row, each with 4 W neighbouring elements per access; a warp owns 32 / LPR * R rows, R accesses in flight.
template <int FMT, int W, int LPR, int R>
__global__ void __launch_bounds__(LA_DECODE_THREADS)
la_decode_kernel(const uint16_t* __restrict__ q, const uint16_t* __restrict__ k, const uint16_t* __restrict__ v,
                 const float* __restrict__ slopes, float* __restrict__ state, uint16_t* __restrict__ o, int h, int dk,
                 int dv) {
  constexpr int EPL = 4 * W, RPW = 32 / LPR;
  static_assert(R <= LPR, "lane j of a row's group writes the j-th result");
  const int bh = blockIdx.y;
  const int lane = threadIdx.x & 31, sub = lane % LPR;
  const int row0 = (blockIdx.x * (LA_DECODE_THREADS / 32) + (threadIdx.x >> 5)) * (RPW * R) + lane / LPR;  // rows row0 + j RPW
  float ve[R], acc[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    ve[j] = (row0 + j * RPW < dv) ? from_16bit<FMT>(v[static_cast<size_t>(bh) * dv + row0 + j * RPW]) : 0.f;
    acc[j] = 0.f;
  }
  const float lam = slopes ? __expf(-slopes[bh % h]) : 1.f;
  const uint16_t* qp = q + static_cast<size_t>(bh) * dk;
  const uint16_t* kp = k + static_cast<size_t>(bh) * dk;
  float* sp = state + (static_cast<size_t>(bh) * dv + row0) * dk;
  for (int c = sub * EPL; c < dk; c += LPR * EPL) {
    LaStateVec<W> st[R];
#pragma unroll
    for (int j = 0; j < R; ++j)
      if (row0 + j * RPW < dv) la_state_ld(st[j], sp + static_cast<size_t>(j * RPW) * dk + c);
    float kf[EPL], qf[EPL];
#pragma unroll
    for (int i = 0; i < EPL; i += 4) {
      const uint2 qq = *reinterpret_cast<const uint2*>(qp + c + i), kk = *reinterpret_cast<const uint2*>(kp + c + i);
      kf[i] = from_16bit<FMT>(kk.x & 0xffffu); kf[i + 1] = from_16bit<FMT>(kk.x >> 16);
      kf[i + 2] = from_16bit<FMT>(kk.y & 0xffffu); kf[i + 3] = from_16bit<FMT>(kk.y >> 16);
      qf[i] = from_16bit<FMT>(qq.x & 0xffffu); qf[i + 1] = from_16bit<FMT>(qq.x >> 16);
      qf[i + 2] = from_16bit<FMT>(qq.y & 0xffffu); qf[i + 3] = from_16bit<FMT>(qq.y >> 16);
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (row0 + j * RPW < dv) {
#pragma unroll
        for (int i = 0; i < EPL; ++i) {
          const float nw = fmaf(kf[i], ve[j], st[j].f[i]);
          acc[j] = fmaf(qf[i], nw, acc[j]);
          st[j].f[i] = lam * nw;
        }
        la_state_st(sp + static_cast<size_t>(j * RPW) * dk + c, st[j]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < R; ++j) {
#pragma unroll
    for (int off = LPR / 2; off > 0; off >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], off);
  }
  float mine = acc[0];
#pragma unroll
  for (int j = 1; j < R; ++j) mine = (sub == j) ? acc[j] : mine;
  if (sub < R && row0 + sub * RPW < dv) o[static_cast<size_t>(bh) * dv + row0 + sub * RPW] = to_16bit<FMT>(mine);
}

}  // namespace lab200
