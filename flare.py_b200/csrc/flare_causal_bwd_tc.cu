// Backward of causal FLARE on the tensor cores (bf16, M <= 128, D in {32, 64}): every 128-token chunk is one unit of
// work for one CTA, and the only thing that passes between the chunks of a (b, h) is the suffix state
// (R [M][D], r [M], mu [M]) of flare_causal_bwd.cu, handed from chunk to chunk through global memory.
//
// With E = e^{S - mu}, l = a l0 + cumsum_t E, A = softmax_M(S), G = A / l, X = v g^T (g = dy), Rin = w R, rin = w r
// (w = e^{mu - nu}, nu the mu of the chunk that produced the state), a chunk is
//
//   S = q k^T, S^T, X                                  [three products on the tiles as loaded]
//   C = (a acc0) g^T + E triu(X),  c = C / l            delta_t = sum_m A_mt c_mt
//   W^T = E^T G (token rows),      Gg = G g             Rout = Rin + Gg,  rout = rin - sum_t G c
//   de = Rin v^T + G triu(X)^T                          dS = E (de + rin - revcumsum(G c)) + A (c - delta)
//   dv = E^T Rin + tril(W)^T g,    dk = scale dS^T q,   dq += scale dS k
//
// Schedule.  512 threads (thread (r, w): tensor-memory lane r, columns 32 w ... 32 w + 31: the latent or the token r of
// every 128 x 128 tile); warp 0 issues the loads and products between two phases of its own row work, since every phase
// waits for the products of the one before it anyway and a 17th warp would cost a quarter of the registers (it spilled
// 400 bytes a thread at the 96 that leaves).  One CTA per SM, persistent, taking units from a counter in the order
// "last chunk of every (b, h), then the one before it, ...".  A unit's predecessor has therefore always been taken
// before it by a running CTA, so the wait for its state ends (and is bounded all the same).  The wait sits in the
// middle of a chunk: everything up to c and Gg is independent of it, and a chunk publishes its own state as soon as it
// has read its predecessor's.  Before this kernel one CTA per (b, h) walked its chunks alone in fp32 FMA loops.
//
// Operands.  Every 128 x 128 operand is written where the next product reads it: rows of E, G, dS packed in tensor
// memory (A operand, contraction over the tokens) and as 64-token column blocks in shared memory (MN-major operand,
// contraction over the latents); X once, masked to t >= n, serves as the MN-major operand of C and the K-major operand
// of de.  All of them, and a acc0, Rin and W, are carried as two bf16 terms (value and remainder; remainder times
// remainder is dropped), about 16 bits where the fp32 kernel has 24: a chunk's own contractions are off by 4e-6 to 1e-5,
// there by 1e-7 to 6e-7.  That is far below what both start from, chunk records with 16-bit weights: dq32 is 1.8e-4 to
// 7.1e-4 off in both, the same to three or four digits (N from 200 to 8192, M = 64 and 128, D = 32 and 64, with wide heads
// too), and dq, dk, dv after their rounding to bf16 (1.67e-3) as well.  With one term of E, G in W and Gg, a acc0 and Rin
// they were 2.23e-3, 2.08e-3, 1.74e-3 off (B = 1, H = 8, N = 512, M = 128, D = 64) instead of 1.72e-3, 1.71e-3, 1.68e-3.
// Shared memory has room for one pair of remainders at a time: first those of E and G, for W; then X, which waits in
// tensor memory until W is complete; then dS.  The second term of E^T Rin comes last, over E.
//
// Tensor memory (512 columns):   0 S | E, G packed | G remainder over E | dS, dS remainder
//                              128 S^T | W^T | W packed in place
//                              256 X | C | de | dk
//                              384 E remainder | dq of the unit      448 a acc0 remainder | Gg | dv
//
// Range: E, l and G are relative to the chunk's final maximum, as in the forward walk, with the same bounds (64
// octaves of climb, 50 between the latents' maxima and the first token's column maximum).  A (b, h) with a chunk
// outside them is flagged and redone as a whole by the fp32 kernel behind this one, from the same two-term prefixes.
// That kernel walks a head alone: one flagged head at the shape below makes the step 20.5 ms (20.05 when it took them all).
//
// B = 4, H = 16, N = 8192, D = 64, M = 128: 546 us for 4096 chunks (the fp32 kernel: 19.1 ms), about 20 us a chunk, of which
// the products are a small part: six waits for products a chunk and no second chunk on the SM to fill them.
#include "common.cuh"
#include "launch.h"
#include "tc_common.cuh"
#include "tma_host.h"

namespace flare {

using namespace tc;

namespace {

constexpr int kRowT = 512;
constexpr int kHalf = 128 * 128;                   // bytes of a 64-column block of a 128-row 16-bit tile

struct CausalBwdTcArgs {
  int B, H, N, M;
  int chunks;
  float scale, scale_log2;
  int q_batched;
  const __nv_bfloat16* pacc;                       // prefix of every chunk as the scan left it, in two terms
  const __nv_bfloat16* plo;
  const float2* pml;
  float4* dq_part;                                 // [chunks][B*H][D/4][128]: four columns of a latent's dq, not yet scaled
  float4* carry;                                   // [B*H][D/4][128]: R of the chunk handed on
  float2* carry_ml;                                // [B*H][2][128]: (r, mu), alternating by chunk
  int* sync;                                       // [0] chunk counter, [1 + c * B*H + bh] "the state of chunk c is out"
  int* redo;                                       // [B*H]
  int* status;
};

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void wait_ld16(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :: "memory");
}
// a pair of values as two bf16 terms: hi, and what hi left over
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(a, b);
  lo = pack_bf16(a - __uint_as_float(hi << 16), b - __uint_as_float(hi & 0xffff0000u));
}
// sum over the 32 lanes of 16 values held by every lane: lane i returns the sum of value i & 15
__device__ __forceinline__ float lane_sums16(float (&v)[16], int lane) {
#pragma unroll
  for (int s = 8; s >= 1; s >>= 1) {
    const bool up = lane & s;
#pragma unroll
    for (int i = 0; i < s; ++i) {
      const float keep = up ? v[i + s] : v[i], give = up ? v[i] : v[i + s];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, s);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

// One 128 x 128 tile row piece (32 columns) of this thread masked to the columns that are not before row r, as two bf16
// terms.  The column block lies before, on or behind the row block for a whole warp, so only the diagonal one masks.
__device__ __forceinline__ void split_upper(const uint32_t (&v)[32], int w, int rb, int lane, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
  if (w > rb) {
#pragma unroll
    for (int j = 0; j < 16; ++j) split2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]), hi[j], lo[j]);
  } else if (w < rb) {
#pragma unroll
    for (int j = 0; j < 16; ++j) hi[j] = lo[j] = 0u;
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      split2(2 * j >= lane ? __uint_as_float(v[2 * j]) : 0.f, 2 * j + 1 >= lane ? __uint_as_float(v[2 * j + 1]) : 0.f, hi[j], lo[j]);
  }
}
// 32 columns (packed pairs) of row r into a 16-bit tile of two 64-column blocks
__device__ __forceinline__ void put_row(uint8_t* tile, int r, int w, const uint32_t (&p)[16]) {
  uint8_t* t = tile + (w >> 1) * kHalf;
#pragma unroll
  for (int q = 0; q < 4; ++q)
    *reinterpret_cast<uint4*>(t + swz_off<128>(r, 4 * (w & 1) + q)) = make_uint4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
}
__device__ __forceinline__ float rcp(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* src, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(map), "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

template <int D>
__global__ void __launch_bounds__(kRowT, 1)
k_causal_bwd_tc(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmG,
                const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV, CausalBwdTcArgs a) {
  constexpr int ROWB = 2 * D, CPR = ROWB / 16;     // bytes and 16-byte pieces of a token row
  constexpr int kTile = 128 * ROWB;
  constexpr int DQ = D / 4;                        // columns of a 128 x D tile a thread owns
  constexpr int NP = CPR / 4;                      // 16-byte pieces of a 16-bit token row it owns
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;
  uint8_t* sK = sQ + kTile;
  uint8_t* sV = sK + kTile;
  uint8_t* sg = sV + kTile;                        // dy rows
  uint8_t* sAR = sg + kTile;                       // a acc0 as bf16 [latent][D], then Rin
  uint8_t* sE = sAR + kTile;
  uint8_t* sG = sE + 2 * kHalf;                    // G; at the end dv and dk on their way out
  uint8_t* sXh = sG + 2 * kHalf;                   // X, then dS
  uint8_t* sXl = sXh + 2 * kHalf;                  // their remainders
  float2* sPart = reinterpret_cast<float2*>(sXl + 2 * kHalf);   // [4][128] (maximum, sum) of a token over a quarter of the latents
  float* sMuP = reinterpret_cast<float*>(sPart + 512);          // [4][128] maximum of a latent over a quarter of the tokens
  float* sRow = sMuP + 512;                        // [4][128] sum of E over a quarter of the tokens
  float* sGc = sRow + 512;                         // [4][128] sum of G c over a quarter of the tokens
  float* sDel = sGc + 512;                         // [4][128] sum of A c over a quarter of the latents
  float* sWt = sDel + 512;                         // [128] w_t: A_mt = E_mt u_m w_t
  float* sDelta = sWt + 128;                       // [128] delta_t
  uint64_t* bars = reinterpret_cast<uint64_t*>(sDelta + 128);
  uint64_t* bar_ld = bars;                         // Q, K, V, g landed
  uint64_t* bar_s = bars + 1;                      // S, S^T, X complete
  uint64_t* bar_c = bars + 2;                      // C complete
  uint64_t* bar_w = bars + 3;                      // W^T complete
  uint64_t* bar_de = bars + 4;                     // de complete
  uint64_t* bar_out = bars + 5;                    // dv, dk, dq complete
  uint64_t* bar_g = bars + 6;                      // Gg complete
  uint64_t* bar_e = bars + 7;                      // E in shared memory has been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
  int* abort_flag = reinterpret_cast<int*>(bars + 9);
  int* sNext = abort_flag + 1;                     // the chunk after this one
  int* sReady = abort_flag + 2;                    // the predecessor's state was out when E and G were

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int r = 32 * (warp & 3) + lane, w = warp >> 2, rb = warp & 3;
  const int BH = a.B * a.H, M = a.M, total = a.chunks * BH;
  const bool live = r < M;
  const float sl = a.scale_log2;

  if (tid == 0) {
    for (int i = 0; i < 8; ++i) mbar_init(bars + i, 1);
    abort_flag[0] = 0;
    *sNext = atomicAdd(a.sync, 1);
    fence_barrier_init();
    prefetch_tmap(&tmQ); prefetch_tmap(&tmK); prefetch_tmap(&tmV); prefetch_tmap(&tmG);
  }
  if (warp == 1) tmem_alloc<512>(tmem_slot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t row = tmem + ((uint32_t)(rb * 32) << 16);
  constexpr uint32_t cS = 0, cEh = 0, cGh = 64, cGl = 0, cDSh = 0, cDSl = 64, cT = 128, cX = 256, cEl = 384, cDQ = 384, cDV = 448, cAl = cDV;

  const uint32_t id_s = idesc_f16(128, 128, 1, 1, 0, 0);            // A, B K-major, N = 128
  const uint32_t id_mn = idesc_f16(128, 128, 1, 1, 1, 1);           // A, B MN-major, N = 128
  const uint32_t id_tm = idesc_f16(128, 128, 1, 1, 0, 1);           // A in tensor memory, B MN-major, N = 128
  const uint32_t id_td = idesc_f16(128, D, 1, 1, 0, 1);             // the same, N = D
  const uint32_t id_md = idesc_f16(128, D, 1, 1, 1, 1);             // A, B MN-major, N = D
  const uint64_t dQ = smem_desc<ROWB>(smem_u32(sQ)), dK = smem_desc<ROWB>(smem_u32(sK)), dV = smem_desc<ROWB>(smem_u32(sV)),
                 dg = smem_desc<ROWB>(smem_u32(sg)), dAR = smem_desc<ROWB>(smem_u32(sAR)), dRl = smem_desc<ROWB>(smem_u32(sG));
  const uint64_t dE = smem_desc_mn128(smem_u32(sE), kHalf, 1024), dG = smem_desc_mn128(smem_u32(sG), kHalf, 1024),
                 dXh = smem_desc_mn128(smem_u32(sXh), kHalf, 1024), dXl = smem_desc_mn128(smem_u32(sXl), kHalf, 1024);

  // Chunk `ticket` in the order of the counter: its tiles and its prefix.  acc0 rows come by asynchronous copies (each
  // thread fetches the pieces it will scale), (m, l) of latent r in registers.
  float2 ml0 = make_float2(-INFINITY, 0.f);
  auto fetch = [&](int ticket) {
    const int c = a.chunks - 1 - ticket / BH, bh = ticket % BH;
    const int b = bh / a.H, h = bh % a.H;
    if (warp == 0 && elect_one()) {
      mbar_expect_tx(bar_ld, 4 * kTile);
      tma_load_4d(sQ, &tmQ, bar_ld, 0, 0, h, a.q_batched ? b : 0);            // rows past M arrive as zeros
      tma_load_4d(sK, &tmK, bar_ld, 0, c * 128, h, b);                        // rows past N arrive as zeros
      tma_load_4d(sV, &tmV, bar_ld, 0, c * 128, h, b);
      tma_load_4d(sg, &tmG, bar_ld, 0, c * 128, h, b);
    }
    __syncwarp();
    const long long prow = (((long long)c * a.B + b) * a.H + h) * M;
    if (live) {
      const uint4* src = reinterpret_cast<const uint4*>(a.pacc + (prow + r) * D) + w * NP;
#pragma unroll
      for (int i = 0; i < NP; ++i)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(sAR + swz_off<ROWB>(r, w * NP + i))), "l"(src + i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    ml0 = a.pml[prow + min(r, M - 1)];
  };

  int ticket = *sNext;
  if (ticket < total) fetch(ticket);
  int out_c = 0, out_bh = -1;                      // the chunk whose dv, dk are staged
  for (uint32_t ph = 0;; ph ^= 1) {
    // also: the results of the chunk before are out of tensor memory, and staged
    const bool stop = __syncthreads_or(*reinterpret_cast<volatile int*>(abort_flag)) != 0 || ticket >= total;
    if (warp == 1 && elect_one()) {
      if (out_bh >= 0) {                           // rows past N are outside the tensor map
        tma_store_4d(&tmDV, sG, 0, out_c * 128, out_bh % a.H, out_bh / a.H);
        tma_store_4d(&tmDK, sG + kTile, 0, out_c * 128, out_bh % a.H, out_bh / a.H);
      }
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    if (stop) {
      if (ticket < total) mbar_wait(bar_ld, ph, a.status, abort_flag);         // giving up: let the loads in flight land first
      break;
    }
    const int c = a.chunks - 1 - ticket / BH, bh = ticket % BH;
    const int n0 = c * 128;
    const int cnt = min(128, a.N - n0);
    const bool last = c == a.chunks - 1;           // nothing behind it: no state to take over
    const bool full = cnt == 128 && M == 128;
    const uint32_t in = cnt >= 32 * (w + 1) ? ~0u : cnt <= 32 * w ? 0u : (1u << (cnt - 32 * w)) - 1u;   // tokens that exist

    if (warp == 0) {
      mbar_wait_hot(bar_ld, ph, a.status, abort_flag);
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) mma_ss(tmem + cS, dQ + 2 * kk, dK + 2 * kk, id_s, kk > 0);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) mma_ss(tmem + cT, dK + 2 * kk, dQ + 2 * kk, id_s, kk > 0);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) mma_ss(tmem + cX, dV + 2 * kk, dg + 2 * kk, id_s, kk > 0);
        mma_commit(bar_s);
      }
      __syncwarp();
    }
    uint4 al[NP];                                  // remainders of this thread's piece of acc0
    {
      const uint4* src = reinterpret_cast<const uint4*>(a.plo + ((((long long)c * a.B * a.H + bh) * M) + min(r, M - 1)) * D) + w * NP;
#pragma unroll
      for (int i = 0; i < NP; ++i) al[i] = __ldcs(src + i);
    }
    const float m0l = ml0.x * kLog2e;              // the record keeps m in natural-log units
    const float l0 = ml0.y;
    mbar_wait_hot(bar_s, ph, a.status, abort_flag);
    tc_fence_after();
    // ---- token r over 32 latents: maximum and sum.  latent r over its 32 tokens: maximum ----
    uint32_t v[32], hi[16], lo[16];
    tmem_ld32(row + cT + 32 * w, v);
    tmem_wait_ld_on(v);
    {
      float mx = -INFINITY, su = 0.f;
      if (full) {
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 32; ++j) m4[j & 3] = fmaxf(m4[j & 3], __uint_as_float(v[j]));
        mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sl;
#pragma unroll
        for (int j = 0; j < 32; ++j) s4[j & 3] += ex2(fmaf(__uint_as_float(v[j]), sl, -mx));
        su = (s4[0] + s4[1]) + (s4[2] + s4[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) if (32 * w + j < M) mx = fmaxf(mx, __uint_as_float(v[j]) * sl);
#pragma unroll
        for (int j = 0; j < 32; ++j) if (32 * w + j < M) su += ex2(fmaf(__uint_as_float(v[j]), sl, -mx));
      }
      sPart[w * 128 + r] = make_float2(mx, su);
    }
    tmem_ld32(row + cS + 32 * w, v);
    tmem_wait_ld_on(v);
    const float first = fmaxf(m0l, __uint_as_float(v[0]) * sl);     // w == 0: the running maximum after the chunk's first token
    {
      float mp = -INFINITY;
      if (full) {
        float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int j = 0; j < 32; ++j) m4[j & 3] = fmaxf(m4[j & 3], __uint_as_float(v[j]));
        mp = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sl;
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) if (in >> j & 1) mp = fmaxf(mp, __uint_as_float(v[j]) * sl);
      }
      sMuP[w * 128 + r] = mp;
    }
    if (tid == 256) *sNext = atomicAdd(a.sync, 1);                  // read at the end of this chunk
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    // ---- A_mt = E_mt u_m w_t with u_m = 2^(mu_m - c0), w_t = 2^(c0 - cmax_t) / csum_t, c0 = cmax of the first token ----
    const float c0 = fmaxf(fmaxf(sPart[0].x, sPart[128].x), fmaxf(sPart[256].x, sPart[384].x));
    if (w == 0) {
      const float2 p0 = sPart[r], p1 = sPart[128 + r], p2 = sPart[256 + r], p3 = sPart[384 + r];
      const float cm = fmaxf(fmaxf(p0.x, p1.x), fmaxf(p2.x, p3.x));
      float cs = p0.y * ex2(p0.x - cm);            // (an empty quarter has maximum -inf and sum 0)
      if (p1.y > 0.f) cs += p1.y * ex2(p1.x - cm);
      if (p2.y > 0.f) cs += p2.y * ex2(p2.x - cm);
      if (p3.y > 0.f) cs += p3.y * ex2(p3.x - cm);
      sWt[r] = r < cnt ? __fdividef(ex2(c0 - cm), cs) : 0.f;
      if (r < cnt && fabsf(c0 - cm) > 50.f) a.redo[bh] = 1;
    }
    const float mu = fmaxf(fmaxf(m0l, fmaxf(sMuP[r], sMuP[128 + r])), fmaxf(sMuP[256 + r], sMuP[384 + r]));
    const float aa = m0l == -INFINITY ? 0.f : ex2(m0l - mu);
    if (w == 0 && live && (mu - first > 64.f || fabsf(mu - c0) > 50.f)) a.redo[bh] = 1;
    const float um = live ? ex2(fminf(fmaxf(mu - c0, -60.f), 60.f)) : 0.f;
#pragma unroll
    for (int i = 0; i < NP; ++i) {                 // a acc0 in place, its remainder where Gg will be
      uint4* at = reinterpret_cast<uint4*>(sAR + swz_off<ROWB>(r, w * NP + i));
      uint32_t ow[4] = {0u, 0u, 0u, 0u}, lw[4] = {0u, 0u, 0u, 0u};
      if (live) {
        const uint4 s4 = *at;
        const uint32_t sw[4] = {s4.x, s4.y, s4.z, s4.w}, tw[4] = {al[i].x, al[i].y, al[i].z, al[i].w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float2 f = Op16<__nv_bfloat16>::unpack(sw[u]), g = Op16<__nv_bfloat16>::unpack(tw[u]);
          split2((f.x + g.x) * aa, (f.y + g.y) * aa, ow[u], lw[u]);
        }
      }
      *at = make_uint4(ow[0], ow[1], ow[2], ow[3]);
      tmem_st4(row + cAl + 4 * (w * NP + i), lw);
    }
    // ---- E ----
    float e[32];
    {
      float s4[4] = {0.f, 0.f, 0.f, 0.f};
      if (full) {
#pragma unroll
        for (int j = 0; j < 32; ++j) e[j] = ex2(fmaf(__uint_as_float(v[j]), sl, -mu));
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) e[j] = live && (in >> j & 1) ? ex2(fmaf(__uint_as_float(v[j]), sl, -mu)) : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 32; ++j) s4[j & 3] += e[j];
      sRow[w * 128 + r] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
#pragma unroll
      for (int j = 0; j < 16; ++j) hi[j] = pack_bf16(e[2 * j], e[2 * j + 1]);
      put_row(sE, r, w, hi);
    }
    // dv, dk of the chunk before have left sG (the thread that sent them waits here)
    if (warp == 1) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncthreads();
    tmem_st16(row + cEh + 16 * w, hi);             // every row of S has been read
#pragma unroll
    for (int j = 0; j < 16; ++j)                   // what the 16 bits of E left over, for C and W
      hi[j] = pack_bf16(e[2 * j] - __uint_as_float(hi[j] << 16), e[2 * j + 1] - __uint_as_float(hi[j] & 0xffff0000u));
    tmem_st16(row + cEl + 16 * w, hi);
    put_row(sXh, r, w, hi);                        // until W is complete; then X
    // ---- l, A, G ----
    const float4* wt4 = reinterpret_cast<const float4*>(sWt + 32 * w);
    float il[32];                                  // 1 / l
    {
      float l = aa * l0;                           // l before this quarter's tokens
      if (w > 0) l += sRow[r];
      if (w > 1) l += sRow[128 + r];
      if (w > 2) l += sRow[256 + r];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 wt = wt4[q];
        const float ws[4] = {wt.x, wt.y, wt.z, wt.w};
        float g[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = 4 * q + u;
          l += e[j];
          il[j] = l > 0.f ? rcp(l) : 0.f;          // l = 0: a latent row past M, or a chunk that is flagged and redone
          g[u] = e[j] * (um * ws[u]) * il[j];
        }
        split2(g[0], g[1], lo[2 * q], hi[2 * q]);
        split2(g[2], g[3], lo[2 * q + 1], hi[2 * q + 1]);
      }
      tmem_st16(row + cGh + 16 * w, lo);
      put_row(sG, r, w, lo);
      put_row(sXl, r, w, hi);
    }
    if (tid == kRowT - 1) *sReady = last || ld_acquire(a.sync + 1 + (c + 1) * BH + bh) != 0;
    tmem_wait_st();
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {           // over the latents
          mma_ss(tmem + cT, dE + 128 * kk, dG + 128 * kk, id_mn, kk > 0);
          mma_ss(tmem + cT, dXh + 128 * kk, dG + 128 * kk, id_mn, true);
          mma_ss(tmem + cT, dE + 128 * kk, dXl + 128 * kk, id_mn, true);
        }
        mma_commit(bar_w);
      }
      __syncwarp();
    }
    const bool ready = *reinterpret_cast<volatile int*>(sReady) != 0;

    // ---- X of token r, masked to t >= r, packed over the remainders; then W^T likewise, in place, while C is formed ----
    tmem_ld32(row + cX + 32 * w, v);
    tmem_wait_ld_on(v);
    split_upper(v, w, rb, lane, hi, lo);
    mbar_wait_hot(bar_w, ph, a.status, abort_flag);
    put_row(sXh, r, w, hi);
    put_row(sXl, r, w, lo);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) {
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) mma_ts(tmem + cX, tmem + cAl + 8 * kk, dg + 2 * kk, id_s, kk > 0);
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) mma_ss(tmem + cX, dAR + 2 * kk, dg + 2 * kk, id_s, true);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {           // contraction over the tokens n, 16 per product
          mma_ts(tmem + cX, tmem + cEh + 8 * kk, dXh + 128 * kk, id_tm, true);
          mma_ts(tmem + cX, tmem + cEh + 8 * kk, dXl + 128 * kk, id_tm, true);
          mma_ts(tmem + cX, tmem + cEl + 8 * kk, dXh + 128 * kk, id_tm, true);
        }
        mma_commit(bar_c);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) mma_ts(tmem + cDV, tmem + cGh + 8 * kk, dg + (uint64_t)(kk * ROWB), id_td, kk > 0);
      }
      __syncwarp();
    }
    tmem_ld32(row + cT + 32 * w, v);
    tmem_wait_ld_on(v);
    split_upper(v, w, rb, lane, hi, lo);
    tmem_st16(row + cT + 32 * w, hi);
    tmem_st16(row + cT + 32 * w + 16, lo);

    // ---- c, sums of G c and A c; dS = E de + bb ----
    mbar_wait_hot(bar_c, ph, a.status, abort_flag);
    tc_fence_after();
    float bb[32];
    {
      float hs[2];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t cv[16], gl[8];
        float gcv[16], ac[16];
        tmem_ld16(row + cX + 32 * w + 16 * hf, cv);
        wait_ld16(cv);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 wt = wt4[4 * hf + q];
          const float ws[4] = {wt.x, wt.y, wt.z, wt.w};
          float g[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int j = 4 * q + u;
            g[u] = e[16 * hf + j] * (um * ws[u]) * il[16 * hf + j];  // as above: gl is what its 16 bits left over
            ac[j] = g[u] * __uint_as_float(cv[j]);                   // A c = (A / l) C
            gcv[j] = ac[j] * il[16 * hf + j];
          }
          uint32_t drop;
          split2(g[0], g[1], drop, gl[2 * q]);
          split2(g[2], g[3], drop, gl[2 * q + 1]);
        }
        tmem_st8(row + cGl + 16 * w + 8 * hf, gl);                   // over E packed: C is complete
        float run = 0.f;
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          run += gcv[j];
          bb[16 * hf + j] = fmaf(-e[16 * hf + j], run, ac[j]);
        }
        hs[hf] = run;
        const float d = lane_sums16(ac, lane);
        if (lane < 16) sDel[rb * 128 + 32 * w + 16 * hf + lane] = d;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) bb[j] = fmaf(-e[j], hs[1], bb[j]);
      sGc[w * 128 + r] = hs[0] + hs[1];
    }
    // ---- the state of the later chunks ----
    float4* const cp = a.carry + ((long long)bh * (D / 4) + w * (DQ / 4)) * 128 + r;
    float2* const cml = a.carry_ml + (long long)bh * 256 + r;
    float4 st[DQ / 4];
    float2 rnu = make_float2(0.f, 0.f);
    auto take = [&] {
      rnu = __ldcg(cml + 128 * ((c + 1) & 1));
#pragma unroll
      for (int p = 0; p < DQ / 4; ++p) st[p] = __ldcg(cp + p * 128);
    };
#pragma unroll
    for (int p = 0; p < DQ / 4; ++p) st[p] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ready && !last) take();
    if (!ready && tid == kRowT - 1) {
      const int* flag = a.sync + 1 + (c + 1) * BH + bh;
      const long long t0 = clock64();
      while (ld_acquire(flag) == 0) {
        if (clock64() - t0 > (1LL << 31)) {
          if (a.status) atomicOr(a.status, kErrWaitTimeout);
          *reinterpret_cast<volatile int*>(abort_flag) = 1;
          break;
        }
      }
    }
    tmem_wait_st();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) mma_ts(tmem + cDV, tmem + cGl + 8 * kk, dg + (uint64_t)(kk * ROWB), id_td, true);
        mma_commit(bar_g);
      }
      __syncwarp();
    }
    if (!ready) take();
    float after, gc_all;                           // sums of G c: the quarters behind this one, the chunk
    {
      const float g0 = sGc[r], g1 = sGc[128 + r], g2 = sGc[256 + r], g3 = sGc[384 + r];
      gc_all = (g0 + g1) + (g2 + g3);
      after = w == 0 ? (g1 + g2) + g3 : w == 1 ? g2 + g3 : w == 2 ? g3 : 0.f;
    }
    if (w == 1) sDelta[r] = (sDel[r] + sDel[128 + r]) + (sDel[256 + r] + sDel[384 + r]);
    const float wf = last ? 0.f : ex2(mu - rnu.y);
    const float rin = wf * rnu.x;
    {
      uint32_t gg[DQ], rp[DQ / 2], rl[DQ / 2];
      mbar_wait_hot(bar_g, ph, a.status, abort_flag);
      tc_fence_after();
      if constexpr (DQ == 16) tmem_ld16(row + cDV + DQ * w, gg);
      else tmem_ld8(row + cDV + DQ * w, gg);
      tmem_wait_ld();
#pragma unroll
      for (int p = 0; p < DQ / 4; ++p) {
        const float4 in4 = make_float4(st[p].x * wf, st[p].y * wf, st[p].z * wf, st[p].w * wf);
        split2(in4.x, in4.y, rp[2 * p], rl[2 * p]);
        split2(in4.z, in4.w, rp[2 * p + 1], rl[2 * p + 1]);
        if (c > 0)
          cp[p * 128] = make_float4(in4.x + __uint_as_float(gg[4 * p]), in4.y + __uint_as_float(gg[4 * p + 1]),
                                    in4.z + __uint_as_float(gg[4 * p + 2]), in4.w + __uint_as_float(gg[4 * p + 3]));
      }
#pragma unroll
      for (int i = 0; i < NP; ++i) {               // Rin over a acc0, its remainder over G: C and W are complete
        *reinterpret_cast<uint4*>(sAR + swz_off<ROWB>(r, w * NP + i)) = make_uint4(rp[4 * i], rp[4 * i + 1], rp[4 * i + 2], rp[4 * i + 3]);
        *reinterpret_cast<uint4*>(sG + swz_off<ROWB>(r, w * NP + i)) = make_uint4(rl[4 * i], rl[4 * i + 1], rl[4 * i + 2], rl[4 * i + 3]);
      }
      if (w == 0 && c > 0) cml[128 * (c & 1)] = make_float2(rin - gc_all, mu);
    }
    tmem_wait_st();
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (tid == 32 && c > 0) {                      // every thread's part of the state is ordered before this by the barrier
      __threadfence();
      st_release(a.sync + 1 + c * BH + bh, 1);
    }
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
          mma_ss(tmem + cX, dAR + 2 * kk, dV + 2 * kk, id_s, kk > 0);
          mma_ss(tmem + cX, dRl + 2 * kk, dV + 2 * kk, id_s, true);
        }
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {           // contraction over the tokens t: X as a K-major operand
          const uint64_t kh = smem_desc<128>(smem_u32(sXh) + (kk >> 2) * kHalf) + 2 * (kk & 3);
          const uint64_t kl = smem_desc<128>(smem_u32(sXl) + (kk >> 2) * kHalf) + 2 * (kk & 3);
          mma_ts(tmem + cX, tmem + cGh + 8 * kk, kh, id_s, true);
          mma_ts(tmem + cX, tmem + cGh + 8 * kk, kl, id_s, true);
          mma_ts(tmem + cX, tmem + cGl + 8 * kk, kh, id_s, true);
        }
        mma_commit(bar_de);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          mma_ss(tmem + cDV, dE + 128 * kk, dAR + (uint64_t)(kk * ROWB), id_md, kk > 0);
          mma_ss(tmem + cDV, dE + 128 * kk, dRl + (uint64_t)(kk * ROWB), id_md, true);
        }
        mma_commit(bar_e);
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {           // W packed in place: 16 columns of values, 16 of remainders per quarter
          const uint32_t wp = tmem + cT + 32 * (kk >> 1) + 8 * (kk & 1);
          mma_ts(tmem + cDV, wp, dg + (uint64_t)(kk * ROWB), id_td, true);
          mma_ts(tmem + cDV, wp + 16, dg + (uint64_t)(kk * ROWB), id_td, true);
        }
      }
      __syncwarp();
    }
    {
      const float4* dl4 = reinterpret_cast<const float4*>(sDelta + 32 * w);
      const float rr = rin - after;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 wt = wt4[q], dl = dl4[q];
        const float ws[4] = {wt.x, wt.y, wt.z, wt.w}, ds[4] = {dl.x, dl.y, dl.z, dl.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) bb[4 * q + u] = fmaf(e[4 * q + u], fmaf(-um, ws[u] * ds[u], rr), bb[4 * q + u]);
      }
    }

    // ---- dS ----
    mbar_wait_hot(bar_de, ph, a.status, abort_flag);
    tc_fence_after();
    tmem_ld32(row + cX + 32 * w, v);
    tmem_wait_ld_on(v);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      split2(fmaf(e[2 * j], __uint_as_float(v[2 * j]), bb[2 * j]), fmaf(e[2 * j + 1], __uint_as_float(v[2 * j + 1]), bb[2 * j + 1]), hi[j], lo[j]);
    tmem_st16(row + cDSh + 16 * w, hi);
    tmem_st16(row + cDSl + 16 * w, lo);
    put_row(sXh, r, w, hi);                        // over X: de is complete
    put_row(sXl, r, w, lo);
    mbar_wait_hot(bar_e, ph, a.status, abort_flag);
#pragma unroll
    for (int j = 0; j < 16; ++j) {                 // the remainder of E over E, for dv
      uint32_t eh;
      split2(e[2 * j], e[2 * j + 1], eh, lo[j]);
    }
    put_row(sE, r, w, lo);
    tmem_wait_st();
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          mma_ss(tmem + cDV, dE + 128 * kk, dAR + (uint64_t)(kk * ROWB), id_md, true);
          mma_ss(tmem + cX, dXh + 128 * kk, dQ + (uint64_t)(kk * ROWB), id_md, kk > 0);              // dk over de
          mma_ss(tmem + cX, dXl + 128 * kk, dQ + (uint64_t)(kk * ROWB), id_md, true);
          mma_ts(tmem + cDQ, tmem + cDSh + 8 * kk, dK + (uint64_t)(kk * ROWB), id_td, kk > 0);
          mma_ts(tmem + cDQ, tmem + cDSl + 8 * kk, dK + (uint64_t)(kk * ROWB), id_td, true);
        }
        mma_commit(bar_out);
      }
      __syncwarp();
    }
    const int next = *reinterpret_cast<volatile int*>(sNext);

    // ---- results: dv, dk of token r to their staging tiles, dq of latent r to this chunk's partial ----
    mbar_wait_hot(bar_out, ph, a.status, abort_flag);
    tc_fence_after();
    if (next < total) fetch(next);                 // every operand tile is free
    {
      uint32_t t1[DQ], t2[DQ], t3[DQ];
      if constexpr (DQ == 16) { tmem_ld16(row + cDV + DQ * w, t1); tmem_ld16(row + cX + DQ * w, t2); tmem_ld16(row + cDQ + DQ * w, t3); }
      else { tmem_ld8(row + cDV + DQ * w, t1); tmem_ld8(row + cX + DQ * w, t2); tmem_ld8(row + cDQ + DQ * w, t3); }
      tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        uint32_t o[4], d[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          o[u] = pack_bf16(__uint_as_float(t1[8 * q + 2 * u]), __uint_as_float(t1[8 * q + 2 * u + 1]));
          d[u] = pack_bf16(__uint_as_float(t2[8 * q + 2 * u]) * a.scale, __uint_as_float(t2[8 * q + 2 * u + 1]) * a.scale);
        }
        const uint32_t off = swz_off<ROWB>(r, w * NP + q);
        *reinterpret_cast<uint4*>(sG + off) = make_uint4(o[0], o[1], o[2], o[3]);
        *reinterpret_cast<uint4*>(sG + kTile + off) = make_uint4(d[0], d[1], d[2], d[3]);
      }
      if (live) {
        float4* po = a.dq_part + (((long long)c * BH + bh) * (D / 4) + w * (DQ / 4)) * 128 + r;
#pragma unroll
        for (int p = 0; p < DQ / 4; ++p)
          po[p * 128] = make_float4(__uint_as_float(t3[4 * p]), __uint_as_float(t3[4 * p + 1]), __uint_as_float(t3[4 * p + 2]), __uint_as_float(t3[4 * p + 3]));
      }
    }
    fence_proxy_async();
    tc_fence_before();
    out_c = c; out_bh = bh;
    ticket = next;
  }
  if (warp == 1) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");     // the staged tiles are written before the CTA ends
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc<512>(tmem);
}

// dq[h][m][d] = scale * (sum over the chunks, and over the batch where it shares its latents) of the partials
// [part][H or B*H][D/4][128] of four columns each.  A block takes 32 latents of one (head, four columns); its eight warps
// take every eighth partial with coalesced 512-byte reads, and their sums meet in shared memory.
template <int D>
__global__ void __launch_bounds__(256)
k_causal_dq_sum(const float4* __restrict__ part, int parts, int heads, int M, float scale, float* __restrict__ dq) {
  grid_dep_sync();
  __shared__ float4 acc[8][32];
  const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
  const int m = blockIdx.x * 32 + lane, d4 = blockIdx.y, hd = blockIdx.z;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (m < M) {
    const float4* p = part + ((long long)hd * (D / 4) + d4) * 128 + m;
    const long long step = (long long)heads * (D / 4) * 128;
#pragma unroll 4
    for (int i = wq; i < parts; i += 8) {
      const float4 x = __ldcs(p + i * step);
      s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w;
    }
  }
  acc[wq][lane] = s;
  __syncthreads();
  if (wq == 0 && m < M) {
#pragma unroll
    for (int i = 1; i < 8; ++i) { s.x += acc[i][lane].x; s.y += acc[i][lane].y; s.z += acc[i][lane].z; s.w += acc[i][lane].w; }
    *reinterpret_cast<float4*>(dq + ((long long)hd * M + m) * D + 4 * d4) = make_float4(s.x * scale, s.y * scale, s.z * scale, s.w * scale);
  }
}

constexpr size_t up256(size_t x) { return (x + 255) & ~size_t(255); }

struct BwdLayout {
  int chunks;
  size_t sync, carry_ml, carry, part, sub, total;
};
BwdLayout layout(const FlareProblem* p) {
  BwdLayout L;
  const size_t BH = (size_t)p->B * p->H;
  L.chunks = (p->N + 127) / 128;
  size_t at = 0;
  auto take = [&](size_t bytes) { const size_t o = at; at += up256(bytes); return o; };
  L.sync = take((1 + (size_t)L.chunks * BH + BH) * sizeof(int));    // counter, flags, redo: cleared together
  L.carry_ml = take(BH * 2 * 128 * sizeof(float2));
  L.carry = take(BH * (p->D / 4) * 128 * sizeof(float4));
  L.part = take((size_t)L.chunks * BH * (p->D / 4) * 128 * sizeof(float4));
  L.sub = take(4 * BH * p->M * (p->D + 2) * sizeof(float));
  L.total = at + 256;
  return L;
}

template <int D>
int launch_bwd(const FlareProblem* p, const void* q, const void* k, const void* v, const void* dy, void* dk, void* dv,
               const CausalBwdTcArgs& a, cudaStream_t st) {
  CUtensorMap tmQ, tmK, tmV, tmG, tmDK, tmDV;
  const uint64_t e = 2;
  const bool qb = p->q_stride[0] != 0;
  auto tokens = [&](CUtensorMap* m, const void* t, const int64_t* s) {
    return make_tile_map(m, t, 1, D, (uint64_t)p->N, (uint64_t)p->H, (uint64_t)p->B, s[2] * e, s[1] * e,
                         (p->B > 1 ? s[0] : s[1] * p->H) * e, 128);
  };
  if (!make_tile_map(&tmQ, q, 1, D, (uint64_t)p->M, (uint64_t)p->H, (uint64_t)(qb ? p->B : 1), p->q_stride[2] * e,
                     p->q_stride[1] * e, (qb ? p->q_stride[0] : p->q_stride[1] * p->H) * e, 128) ||
      !tokens(&tmK, k, p->k_stride) || !tokens(&tmV, v, p->v_stride) || !tokens(&tmG, dy, p->dy_stride) ||
      !tokens(&tmDK, dk, p->dk_stride) || !tokens(&tmDV, dv, p->dv_stride))
    return FLARE_EUNSUPPORTED;
  constexpr int smem = 5 * 128 * 2 * D + 8 * kHalf + 13 * 1024 + 256 + 1024;
  if (tc_set_dyn_smem(reinterpret_cast<const void*>(&k_causal_bwd_tc<D>), smem) != FLARE_OK) return FLARE_ECUDA;
  const long long n = (long long)a.chunks * a.B * a.H;
  const int grid = (int)(n < num_sms() ? n : num_sms());
  k_causal_bwd_tc<D><<<grid, kRowT, smem, st>>>(tmQ, tmK, tmV, tmG, tmDK, tmDV, a);       // behind a memset: a plain launch
  return cudaPeekAtLastError() == cudaSuccess ? FLARE_OK : FLARE_ECUDA;
}

}  // namespace

bool causal_bwd_tc_supported(const FlareProblem* p, const void* q, const void* k, const void* v, const void* dy,
                             const void* dk, const void* dv) {
  FlareProblem t = *p;
  auto with_y = [&](const int64_t* s) { for (int i = 0; i < 3; ++i) t.y_stride[i] = s[i]; return &t; };
  return causal_tc_walk_supported(with_y(p->dy_stride), q, k, v, dy) && causal_tc_walk_supported(with_y(p->dk_stride), q, k, v, dk) &&
         causal_tc_walk_supported(with_y(p->dv_stride), q, k, v, dv);
}

size_t causal_bwd_tc_workspace(const FlareProblem* p) { return layout(p).total; }

int causal_bwd_tc(const FlareProblem* p, const void* q, const void* k, const void* v, const void* dy, const __nv_bfloat16* pacc,
                  const __nv_bfloat16* plo, const float2* pml, float* dq32, bool sum_batch, void* dk, void* dv, void* workspace, cudaStream_t st) {
  const BwdLayout L = layout(p);
  char* ws = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255));
  const int BH = p->B * p->H;
  CausalBwdTcArgs a;
  a.B = p->B; a.H = p->H; a.N = p->N; a.M = p->M;
  a.chunks = L.chunks;
  a.scale = p->scale; a.scale_log2 = p->scale * kLog2e;
  a.q_batched = p->q_stride[0] != 0;
  a.pacc = pacc; a.plo = plo; a.pml = pml;
  a.dq_part = reinterpret_cast<float4*>(ws + L.part);
  a.carry = reinterpret_cast<float4*>(ws + L.carry);
  a.carry_ml = reinterpret_cast<float2*>(ws + L.carry_ml);
  a.sync = reinterpret_cast<int*>(ws + L.sync);
  a.redo = a.sync + 1 + (size_t)L.chunks * BH;
  a.status = tc_status_ptr();
  if (cudaMemsetAsync(a.sync, 0, (1 + (size_t)L.chunks * BH + BH) * sizeof(int), st) != cudaSuccess) return FLARE_ECUDA;
  int rc = p->D == 32 ? launch_bwd<32>(p, q, k, v, dy, dk, dv, a, st) : launch_bwd<64>(p, q, k, v, dy, dk, dv, a, st);
  if (rc != FLARE_OK) return rc;
  rc = causal_bwd_redo(p, q, k, v, dy, pacc, plo, pml, a.redo, reinterpret_cast<float*>(a.dq_part), L.chunks, dk, dv, reinterpret_cast<float*>(ws + L.sub), st);
  if (rc != FLARE_OK) return rc;
  const int heads = sum_batch ? p->H : BH, parts = L.chunks * (sum_batch ? p->B : 1);
  const dim3 grid((unsigned)((p->M + 31) / 32), (unsigned)(p->D / 4), (unsigned)heads);
  if (p->D == 32) launch_dep(k_causal_dq_sum<32>, grid, dim3(256), 0, st, a.dq_part, parts, heads, p->M, p->scale, dq32);
  else launch_dep(k_causal_dq_sum<64>, grid, dim3(256), 0, st, a.dq_part, parts, heads, p->M, p->scale, dq32);
  return cudaPeekAtLastError() == cudaSuccess ? FLARE_OK : FLARE_ECUDA;
}

}  // namespace flare
