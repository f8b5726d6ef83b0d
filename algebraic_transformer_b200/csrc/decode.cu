// Single-query asinh-power attention against a KV cache (Tq = 1, all keys visible).
//
// HBM-bound: every K and V row is read from HBM exactly once.  Keys are split over CTAs
// (grid = splits x heads x batch); inside a CTA a producer warp streams 32-key K and V tiles
// into a shared-memory ring with TMA (192 KB an SM, in one or two CTAs), and four or six consumer warps take
// the tiles in turn, each with a state of its own (running maximum m, normaliser l, accumulator;
// weight w = (rho(x) rho(-m))^n, the max-shifted weight of src/algebraic/algebraic.py:186-204), so
// no step of the key loop involves the whole CTA and nothing but the ring's barriers paces it.
//
// What bounded the loop before was instruction issue, not HBM: eight lanes shared a key's products
// and all eight evaluated its weight, 200 instructions of a warp for 8 keys of head_dim 64, so caches of
// a few thousand keys streamed at 3.9 TB/s.  Now both products run on the tensor cores as
// mma.sync.m16n8k16, and a warp spends on 32 keys what it spent on 8:
//   scores   A = q in every one of the first eight rows, B = K rows as they lie in shared memory
//            (bf16 x bf16 is exact in fp32, as the scalar products were); every row of the result holds the
//            32 scores, lane (r, i) = (lane / 4, lane % 4) those of keys 2 i, 2 i + 1 of each block of eight;
//   weights  lane (r, i) evaluates the one key 8 (r / 2) + 2 i + r % 2;
//   output   A rows 0, 1, 2 = the three bf16 that add up to the fp32 weight, 8 bits of it each, so that the
//            accumulator rows 0, 1 and 2 add up to what fp32 weights would give; B = V rows through ldmatrix.trans.
//            The remaining rows of A are ignored.  The normaliser adds the fp32 weights.
//            (With two parts, 16 of the 24 bits, the error before the output's rounding was ten times that of fp32
//            products: 1.1e-6 against 1.1e-7 rms of the terms' size with two keys and n = 2, 1.16e-7 now; of
//            5.2 million outputs over 64 to 60000 keys 8935 were not the nearest bf16, 4790 with fp32 products, 4871 now.  The
//            third part costs nothing at head_dim 64 and on single CTAs, 2 to 4 % where two CTAs of head_dim 128 share an
//            SM: 16 x 12 x 3000 x 128 57.9 -> 59.0-60.4 us, 32 x 24 x 300 x 128 33.0 -> 34.4.)
// Single-row products leave 13 of the 16 rows idle, which costs nothing: the tensor pipe is at a few percent.
//
// The warp states are merged once at the end with the exact rescale (rho(m_a) rho(-m))^n.  A CTA
// that holds a whole head writes the output row; otherwise it writes its (acc, m, l) state and the split
// that finishes last for its (batch, head) merges the states, with the sink, and writes the output
// row: one launch.  "Last" is decided by an arrival word per (batch, head) that carries the call's
// number, so that nothing has to be zeroed between calls (a word left by another call counts as
// zero arrivals).  All mbarrier waits are bounded; the row of a (batch, head) whose wait ran out is NaN, and the status
// word, where there is one, says ALG_DEV_TIMEOUT.
//
// Measured (CUDA graph, before -> now): 16 x 16 heads x 1900 keys x 64 31.7 -> 21.7 us = 5.7 TB/s, 1 x 16 x 32768 x 128
// 55.5 -> 47.5 = 5.65 TB/s, 16 x 12 x 3000 x 128 73 -> 59, 32 x 24 x 64 x 64 15.4 -> 9.6, 1 x 12 x 333 x 64 9.7 -> 8.2, of which
// about 8 is a launch, the first tile's way and the merge.
#include "common.cuh"
#include "launchers.h"
#include "sm100_ptx.cuh"

namespace alg {
namespace {

using namespace sm100;

constexpr int TILE = 32;                        // keys of a ring slot: one consumer warp's step
constexpr int SPLIT_UNIT = 64;                  // splits are whole multiples of this many keys
constexpr int PANEL = TILE * 128;               // 64 columns of a tile, 128-byte swizzle
// Tile t lies in slot t % STAGES and belongs to warp t % CWARPS.  STAGES is a multiple of CWARPS, so that every slot
// belongs to ONE warp: a warp that waited for a slot whose previous tile is another warp's could look at the slot's
// barrier while that tile is still on its way, and would take the phase before it for its own.
template <int D, int CTAS> struct Cfg {
  static constexpr int PANELS = D / 64, TILE_BYTES = PANELS * PANEL;
  static constexpr int STAGES = 24 / PANELS / CTAS;    // 192 KB of K and V tiles per SM
  static constexpr int CWARPS = D == 64 ? 4 : 6, CONSUMERS = CWARPS * 32, NTHREADS = CONSUMERS + 32;
  static_assert(STAGES % CWARPS == 0, "a slot belongs to one warp");
  static_assert(CONSUMERS >= D, "a thread per output column in the merges");
};
constexpr int MAX_CWARPS = 6, MAX_STAGES = 12;

struct __align__(16) DecodeCtl {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES];
  int abort_flag;
  int tile_ok;
  int last_split;
  float m[MAX_CWARPS], l[MAX_CWARPS];
};

template <class C> constexpr size_t decode_smem() { return size_t(C::STAGES) * 2 * C::TILE_BYTES + sizeof(DecodeCtl) + 1024; }

template <int N> __device__ __forceinline__ void consumer_sync() { asm volatile("bar.sync 1, %0;" ::"n"(N) : "memory"); }

// four 8x8 bf16 matrices; lane i gives the address of row i % 8 of matrix i / 8
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_trans(uint32_t addr, uint32_t* r) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// c[0..1] (rows 0-7) += A B with rows 8-15 of A zero
__device__ __forceinline__ void mma_top(float* c, uint32_t a0, uint32_t a2, uint32_t b0, uint32_t b1) {
  float x, y;                                   // rows 8-15 of the result: zero
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%5}, {%7,%8}, {%0,%1,%9,%9};"
               : "+f"(c[0]), "+f"(c[1]), "=f"(x), "=f"(y) : "r"(a0), "r"(0u), "r"(a2), "r"(b0), "r"(b1), "f"(0.f));
}

constexpr int MAX_SPLITS = 1024;

// Merge the splits (and the sink) of one (batch, head); called by every thread of the CTA that
// arrived last, thread d < D owns output column d.  `scratch`: 2 * MAX_SPLITS floats of shared memory.
template <int D>
__device__ __forceinline__ void decode_combine(const DecodeParams& p, int b, int h, float* scratch) {
  float* s_f = scratch;                          // rescale factor per split
  float* s_l = scratch + MAX_SPLITS;
  float* s_red = scratch + 2 * MAX_SPLITS;       // D / 32 partial maxima
  const int bh = b * p.H + h;
  const float* part = p.part + int64_t(bh) * p.splits * (D + 2);
  const bool has_sink = p.sink != nullptr;
  const float bs = has_sink ? p.sink[h] * p.inv_c : -1e30f;
  const bool mine = threadIdx.x < D;
  float mm = bs;                                 // all loads below are independent of one another
  if (mine) {
    for (int s = threadIdx.x; s < p.splits; s += D) {
      const float ms = __ldcg(part + s * (D + 2) + D);      // written by other CTAs: read past L1
      s_f[s] = ms;
      s_l[s] = __ldcg(part + s * (D + 2) + D + 1);
      mm = fmaxf(mm, ms);
    }
    mm = warp_max(mm);
    if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = mm;
  }
  __syncthreads();
  mm = s_red[0];
#pragma unroll
  for (int i = 1; i < D / 32; ++i) mm = fmaxf(mm, s_red[i]);
  const float ns = rho_stable(-mm);
  if (mine) {
    for (int s = threadIdx.x; s < p.splits; s += D) {
      const float ms = s_f[s];
      s_f[s] = (ms > -1e29f) ? pow2n_rt(rho_stable(ms) * ns, p.log2n) : 0.f;
    }
  }
  __syncthreads();
  if (!mine) return;
  float lt = has_sink ? pow2n_rt(rho_stable(bs) * ns, p.log2n) : 0.f;
  float at = 0.f;
#pragma unroll 8
  for (int s = 0; s < p.splits; ++s) {
    lt = fmaf(s_f[s], s_l[s], lt);
    at = fmaf(s_f[s], __ldcg(part + s * (D + 2) + threadIdx.x), at);
  }
  reinterpret_cast<__nv_bfloat16*>(p.o)[int64_t(bh) * D + threadIdx.x] = __float2bfloat16_rn(at / lt);
}

template <int D, int CTAS>
__global__ void __launch_bounds__(Cfg<D, CTAS>::NTHREADS, CTAS)
decode_partial_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                      const DecodeParams p) {
  using C = Cfg<D, CTAS>;
  constexpr int STAGES = C::STAGES, TILE_BYTES = C::TILE_BYTES, CWARPS = C::CWARPS;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  DecodeCtl* ctl = reinterpret_cast<DecodeCtl*>(smem + size_t(STAGES) * 2 * TILE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int k_begin = split * p.keys_per_split;
  const int k_end = min(p.Tk, k_begin + p.keys_per_split);
  const int ntiles = k_end > k_begin ? (k_end - k_begin + TILE - 1) / TILE : 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&ctl->full[s], 1); mbar_init(&ctl->empty[s], 1); }
    ctl->abort_flag = 0;
    ctl->tile_ok = 1;
    fence_barrier_init();
  }
  if (threadIdx.x == C::CONSUMERS) { tma_prefetch_desc(&tm_k); tma_prefetch_desc(&tm_v); }
  __syncthreads();
  griddep_wait();                               // launched as a programmatic dependent of the kernel ahead in the stream
  const BoundedWait bw{&ctl->abort_flag, p.wait_ns};

  if (warp == CWARPS) {                         // producer warp
    if (lane == 0) {
      uint32_t stage = 0, phase = 1;
      const int loads = min(ntiles, p.max_loads);
      for (int t = 0; t < loads; ++t) {
        if (!bw.wait(&ctl->empty[stage], phase)) break;
        unsigned char* dst = smem + size_t(stage) * 2 * TILE_BYTES;
        mbar_arrive_expect_tx(&ctl->full[stage], 2 * TILE_BYTES);
        tma_load_5d(dst, &tm_k, &ctl->full[stage], 0, k_begin + t * TILE, 0, h, b);
        tma_load_5d(dst + TILE_BYTES, &tm_v, &ctl->full[stage], 0, k_begin + t * TILE, 0, h, b);
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
      }
    }
  } else {
    const int r = lane >> 2, i = lane & 3;      // row and column pair of an mma result
    uint32_t qa[D / 16][2];                     // A fragments of q: columns 2 i, 2 i + 1 and 8 further of each 16
    const uint32_t* q32 = reinterpret_cast<const uint32_t*>(static_cast<const __nv_bfloat16*>(p.q) + (int64_t(b) * p.H + h) * D);
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) { qa[ks][0] = q32[ks * 8 + i]; qa[ks][1] = q32[ks * 8 + 4 + i]; }
    float acc[D / 8][2];                        // rows 0, 1, 2: the three parts of the weights times V
#pragma unroll
    for (int c = 0; c < D / 8; ++c) acc[c][0] = acc[c][1] = 0.f;
    float m_ref = -1e30f, shift = 0.f, l_part = 0.f;
    // addresses within a panel; a 16-byte chunk c of row `key` lies at chunk c ^ (key % 8)
    const uint32_t ring = smem_u32(smem);
    const uint32_t k_row = uint32_t(lane & 7) * 128, k_chunk = uint32_t(lane >> 3);              // + 8 keys, + 4 chunks
    const uint32_t v_row = uint32_t(((lane >> 3) & 1) * 8 + (lane & 7)) * 128, v_chunk = uint32_t(lane >> 4);   // + 16 keys, + 2
    const uint32_t swz = uint32_t(lane & 7);
    const int own = 8 * (r >> 1) + 2 * i + (r & 1);                                              // the key this lane evaluates
    const bool odd = (r & 1) != 0;
    const uint32_t part = uint32_t(i) | (r == 0 ? 0u : r == 1 ? 4u : 8u);                        // the lane that has this row's part of a weight
    bool ok = true;
    for (int t = warp; t < ntiles; t += CWARPS) {
      const int stage = t % STAGES;
      if (!__all_sync(0xffffffffu, bw.wait(&ctl->full[stage], uint32_t(t / STAGES) & 1u))) { ok = false; break; }
      const uint32_t sk = ring + uint32_t(stage) * (2 * TILE_BYTES), sv = sk + TILE_BYTES;
      float sc[4][2];
#pragma unroll
      for (int n = 0; n < 4; ++n) sc[n][0] = sc[n][1] = 0.f;
#pragma unroll
      for (int kq = 0; kq < D / 32; ++kq) {     // 32 columns of K a load
#pragma unroll
        for (int n = 0; n < 4; ++n) {           // eight keys
          uint32_t kb[4];
          ldsm4(sk + (kq >> 1) * PANEL + n * 1024 + k_row + (((uint32_t(kq & 1) * 4 + k_chunk) ^ swz) << 4), kb);
          mma_top(sc[n], qa[2 * kq][0], qa[2 * kq][1], kb[0], kb[1]);
          mma_top(sc[n], qa[2 * kq + 1][0], qa[2 * kq + 1][1], kb[2], kb[3]);
        }
      }
      const float e0 = (r & 1) ? sc[0][1] : sc[0][0], e1 = (r & 1) ? sc[1][1] : sc[1][0];
      const float e2 = (r & 1) ? sc[2][1] : sc[2][0], e3 = (r & 1) ? sc[3][1] : sc[3][0];
      const float f0 = (r & 2) ? e1 : e0, f1 = (r & 2) ? e3 : e2;
      const float x = (k_begin + t * TILE + own < k_end) ? ((r & 4) ? f1 : f0) * p.scale : -1e30f;
      const float tmax = warp_max(x);
      if (tmax > m_ref) {                                    // warp-uniform
        const float ns = rho_stable(-tmax);
        const float alpha = (m_ref > -1e29f) ? pow2n_rt(rho_stable(m_ref) * ns, p.log2n) : 0.f;
        l_part *= alpha;
#pragma unroll
        for (int c = 0; c < D / 8; ++c) { acc[c][0] *= alpha; acc[c][1] *= alpha; }
        m_ref = tmax;
        shift = ns;
      }
      const float w = (x > -1e29f) ? pow2n_rt(rho_stable(x) * shift, p.log2n) : 0.f;
      l_part += w;
      // w = h + m + lo, three bf16 that carry all 24 bits of it.  Two neighbouring keys' lanes (even and odd row) exchange
      // halves: the even one then has both keys' h, the odd one both m, either both lo, which also go to the
      // lanes of the neighbouring block of eight keys.  One shuffle per block then serves rows 0, 1 and 2.
      const float h = __bfloat162float(__float2bfloat16_rn(w)), m = __bfloat162float(__float2bfloat16_rn(w - h)), lo = w - h - m;
      const uint32_t kept = pack_bf16(odd ? m : h, lo);
      const uint32_t got = __shfl_xor_sync(0xffffffffu, pack_bf16(odd ? h : m, lo), 4);
      const uint32_t lead = __byte_perm(kept, got, odd ? 0x1054u : 0x5410u);
      const uint32_t rest = __shfl_xor_sync(0xffffffffu, __byte_perm(kept, got, odd ? 0x3276u : 0x7632u), 8);
#pragma unroll
      for (int ks = 0; ks < 2; ++ks) {          // sixteen keys
        uint32_t wa[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {           // keys 2 i, 2 i + 1 of block 2 ks + j
          const int block = 2 * ks + j;
          wa[j] = __shfl_sync(0xffffffffu, (r >> 1) == block ? lead : rest, (block * 8) ^ int(part));
        }
#pragma unroll
        for (int c = 0; c < D / 8; c += 2) {    // sixteen columns of V a load
          uint32_t vb[4];
          ldsm4_trans(sv + (c >> 3) * PANEL + ks * 2048 + v_row + (((uint32_t(c & 7) + v_chunk) ^ swz) << 4), vb);
          mma_top(acc[c], wa[0], wa[1], vb[0], vb[1]);
          mma_top(acc[c + 1], wa[0], wa[1], vb[2], vb[3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->empty[stage]);      // this warp is done with the stage
    }
    // ---- this warp's state: rows 0, 1 and 2 together, then merge the warps
    __syncwarp();
    l_part = warp_sum(l_part);
    consumer_sync<C::CONSUMERS>();                          // ring no longer read: reuse it as scratch
    float* s_acc = reinterpret_cast<float*>(smem);         // [warps][D]
#pragma unroll
    for (int c = 0; c < D / 8; ++c) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float mid = __shfl_down_sync(0xffffffffu, acc[c][e], 4), low = __shfl_down_sync(0xffffffffu, acc[c][e], 8);
        // an infinite V meets a zero part of a weight as NaN: the leading part has the answer then
        if (r == 0) s_acc[warp * D + c * 8 + 2 * i + e] = isinf(acc[c][e]) ? acc[c][e] : acc[c][e] + (mid + low);
      }
    }
    if (lane == 0) { ctl->m[warp] = m_ref; ctl->l[warp] = l_part; if (!ok) ctl->tile_ok = 0; }
    consumer_sync<C::CONSUMERS>();
    if (threadIdx.x < D) {
      const bool fine = ctl->tile_ok != 0;                    // a wait that ran out leaves a row of NaN, not one of fewer keys
      const float nan = __int_as_float(0x7fc00000);
      const bool sunk = p.splits == 1 && p.sink != nullptr;   // the sink joins here when this CTA has the whole head
      const float bs = sunk ? p.sink[h] * p.inv_c : -1e30f;
      float mm = bs;
#pragma unroll
      for (int wv = 0; wv < CWARPS; ++wv) mm = fmaxf(mm, ctl->m[wv]);
      const float ns = rho_stable(-mm);
      float a = 0.f, l = sunk ? pow2n_rt(rho_stable(bs) * ns, p.log2n) : 0.f;
#pragma unroll
      for (int wv = 0; wv < CWARPS; ++wv) {
        const float mw = ctl->m[wv];
        const float f = (mw > -1e29f) ? pow2n_rt(rho_stable(mw) * ns, p.log2n) : 0.f;
        a = fmaf(f, s_acc[wv * D + threadIdx.x], a);
        l = fmaf(f, ctl->l[wv], l);
      }
      if (p.splits == 1) {
        reinterpret_cast<__nv_bfloat16*>(p.o)[(int64_t(b) * p.H + h) * D + threadIdx.x] = __float2bfloat16_rn(fine ? a / l : nan);
      } else {
        float* out = p.part + ((int64_t(b) * p.H + h) * p.splits + split) * (D + 2);
        out[threadIdx.x] = fine ? a : 0.f;
        if (threadIdx.x == 0) {
          out[D] = fine ? mm : -1e30f;
          out[D + 1] = fine ? l : nan;                      // reaches the merged row as 0 * NaN
        }
        __threadfence();                                   // the state is visible before this split counts as arrived
      }
    }
  }
  __syncthreads();
  // ---- arrival: the split that completes the count merges all states of its (batch, head)
  if (threadIdx.x == 0 && p.splits == 1) ctl->last_split = 0;
  if (threadIdx.x == 0 && p.splits > 1) {
    unsigned long long* word = p.arrivals + (int64_t(b) * p.H + h);
    unsigned long long seen = *reinterpret_cast<volatile unsigned long long*>(word), next;
    for (;;) {                                             // at most `splits` contenders, each retries a few times
      next = ((seen >> 16) == p.call) ? seen + 1 : ((p.call << 16) | 1ull);
      const unsigned long long prev = atomicCAS(word, seen, next);
      if (prev == seen) break;
      seen = prev;
    }
    ctl->last_split = int(next & 0xffffull) == p.splits ? 1 : 0;
    // the last one leaves the word at zero: a replay of this very launch (a captured graph carries the
    // same call number) starts counting afresh
    if (ctl->last_split) *reinterpret_cast<volatile unsigned long long*>(word) = 0ull;
    __threadfence();
  }
  __syncthreads();
  if (ctl->last_split) decode_combine<D>(p, b, h, reinterpret_cast<float*>(smem));
  __syncthreads();
  if (ctl->abort_flag != 0 && threadIdx.x == 0) {
    if (p.status != nullptr) atomicExch(p.status, ALG_DEV_TIMEOUT);
    const uint64_t t0 = global_timer_ns();                 // let issued loads land before the CTA retires
    while (global_timer_ns() - t0 < 200000ull) { }
  }
}

int make_kv_map(CUtensorMap* tm, const void* base, const Strides3& s, int B, int H, int T, int D) {
  // 64 columns a panel: one copy brings a tile's panels one behind the other
  const uint64_t dims[5] = {64, uint64_t(T), uint64_t(D / 64), uint64_t(H), uint64_t(B)};
  const uint64_t strides[4] = {uint64_t(s.t), 64, uint64_t(s.h), uint64_t(s.b)};
  const uint32_t box[5] = {64, TILE, uint32_t(D / 64), 1, 1};
  return make_tmap_bf16(tm, base, 5, dims, strides, box, true);
}

template <int D, int CTAS>
int launch_d(const DecodeParams& p, cudaStream_t stream) {
  using C = Cfg<D, CTAS>;
  static_assert(CTAS * (decode_smem<C>() + 1024) <= 233472, "shared memory of an SM");
  CUtensorMap tk, tv;
  if (int rc = make_kv_map(&tk, p.k, p.ks, p.B, p.H, p.Tk, D)) return rc;
  if (int rc = make_kv_map(&tv, p.v, p.vs, p.B, p.H, p.Tk, D)) return rc;
  auto kern = decode_partial_kernel<D, CTAS>;
  static PerDeviceOnce configured;
  if (int rc = configured.run([&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(decode_smem<C>())); })) return rc;
  ALG_CUDA_TRY(launch_dependent(kern, dim3(p.splits, p.H, p.B), dim3(C::NTHREADS), decode_smem<C>(), stream, tk, tv, p));
  count_launch();
  return ALG_OK;
}

}  // namespace

// CTAs that share an SM (and its 192 KB of ring).  head_dim 64: two (one: 16 x 16 heads x 1900 keys 21.7 -> 33.3 us).
// head_dim 128: one CTA needs no register spills and halves the states to merge, two start and end more smoothly
// beside each other; what decides is how full the last round of CTAs is.  Heads up to the SM count are split to fill
// one round, and heads that take an odd number of rounds of single CTAs would waste half a round in pairs: one.
// Measured, two -> one: 1 x 16 x 32768 57 -> 47.5 us, 7 x 6 x 5000 30.2 -> 24.0, 16 x 24 x 1000 (3 rounds) 47.9 -> 39.9;
// 16 x 12 x 500 (2 rounds) 13.6 -> 15.0, 32 x 24 x 300 (6 rounds) 33.6 -> 41.2.  75 to 147 heads in single CTAs are one
// unsplit CTA each and leave SMs idle, which loses nothing to speak of: the CTAs' rings together already
// draw what HBM gives (4 x 24 x 8192 59.4 us = 6.8 TB/s on 96 SMs, 5 x 16 x 8192 56.8 us = 5.9 TB/s on 80).
static int ctas_per_sm(int D, int B, int H) {
  const int sms = sm_count();
  return D == 128 && ((int64_t(B) * H + sms - 1) / sms) % 2 == 1 ? 1 : 2;
}

// Splits are whole 64-key units, and at least two of them (four tiles: fewer would leave consumer warps
// without one and only add states to merge).  The grid is ONE wave where heads allow (a second wave
// would pay the ring's start-up latency again: 62 -> 56 us on a 32768-key cache), never more splits than the
// merging CTA's table.
int decode_splits(int D, int B, int H, int Tk) {
  const int bh = B * H > 0 ? B * H : 1;
  const int units = (Tk + SPLIT_UNIT - 1) / SPLIT_UNIT;
  int s = sm_count() * ctas_per_sm(D, B, H) / bh;
  if (s > (units + 1) / 2) s = (units + 1) / 2;
  if (s > MAX_SPLITS) s = MAX_SPLITS;
  if (s < 1) s = 1;
  const int units_per_split = (units + s - 1) / s;
  return (units + units_per_split - 1) / units_per_split;
}

int decode_keys_per_split(int D, int B, int H, int Tk) {
  const int units = (Tk + SPLIT_UNIT - 1) / SPLIT_UNIT;
  const int s = decode_splits(D, B, H, Tk);
  return ((units + s - 1) / s) * SPLIT_UNIT;
}

int launch_decode(const DecodeParams& p, cudaStream_t stream) {
  if (p.B == 0 || p.H == 0) return ALG_OK;
  const int ctas = ctas_per_sm(p.D, p.B, p.H);
  if (p.D == 64) return launch_d<64, 2>(p, stream);
  if (p.D == 128) return ctas == 1 ? launch_d<128, 1>(p, stream) : launch_d<128, 2>(p, stream);
  set_error("decode needs head_dim 64 or 128, got %d", p.D);
  return ALG_ERR_UNSUPPORTED;
}

}  // namespace alg
