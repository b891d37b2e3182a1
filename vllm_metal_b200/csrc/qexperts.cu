// Routed experts with affine-quantized weights: choice of the experts, rows grouped and staged as fp16, the products of all
// experts in two persistent tcgen05 launches, weighted sum.  Nothing is read back to the host.
//
// The products: weights fill the M side (128 rows of a tile: 64 gate + 64 up rows of the same features on the way in, 128
// features on the way out) and an expert's rows the N side (16 .. 192 of them, in steps of 16: its rows are split evenly over
// as few tiles as hold them), so packed weights cross HBM once and are unpacked once for up to 192 rows.
//
//   8 warps                unpack: half a weight row of 64 columns a thread; int4 / int8 -> s * q + b (one rounding to fp16)
//                          -> the A ring in tensor memory
//   8 warps                epilogue: bias, activation, stores; two accumulators, so the next item's products overlap it
//   1 warp                 packed words (ring) and the whole rows' scales and biases of an item (one bulk copy each: rows are
//                          contiguous, however odd K / group is)
//   1 warp                 the rows of x, by TMA from the grouped fp16 copy
//   1 warp                 tcgen05.mma, A from tensor memory
//
// The accumulators' additions drop bits, the more of them in a chain the more: a result that is one chain of K = 2880 is not the
// rounding of the float64 sum over the same fp16 weights in 0.13 % (int4) to 0.19 % (int8) of cases, as in the dense GEMM above 64
// rows; a GEMM of few rows, which splits K, has 0.04 to 0.06 %.  So narrow tiles deal their steps out to four accumulators (two for
// 64 rows) which the epilogue adds up: 0.04 to 0.06 % (64 rows 0.07 to 0.10).  32 rows 166 -> 168 us a block, 128 rows 168 -> 174.  The
// sums of every step in registers instead, 0.02 %, took 197 and 201.
//
// A word's nibbles come out as (k_i, k_{i+4}) pairs; the grouped copy holds its columns in that order, so that no permutation
// of weights is needed, neither at load time nor here.
//
// Few rows are bound by the single warps' hand-offs, whose time does not shrink with the work between them: a step of 256 columns
// (SK = 4) instead of 64 and one copy of x for it took a way in of 32 experts of 2880 x 2880, int4 in groups of 64, 32 rows in all
// from 146 to 94 us (words 265 MB, scales and biases 33 MB: 46 us of HBM).  Then 57 % of the issue slots are taken, 37 % of HBM and
// 8 % of the tensor pipe.  Many rows need the finer ring more (two steps of 128 columns are all that tensor memory has left beside
// 192 rows): 1024 rows, 183 us with steps of 64 columns, 204 with 128; with fast exponentials in the epilogue, whose instructions
// compete with the unpacking, 169.  Counters: profiles/expert_products_ncu.txt.
#include "../../include/b200_hybrid_ops.h"
#include "qdequant.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>

namespace b200 {
namespace qx {
using namespace tc;

constexpr int kPacked = 128 * 128;  // bytes of a packed stage: 128 rows x 128 B
constexpr int kMaxA = 6;            // steps of A in tensor memory, at most: what two accumulators leave
constexpr int kMaxX = 16;           // of x in shared memory, at most
constexpr int kMaxTile = 192;       // rows of x a tile holds: two accumulators and the A ring fill tensor memory
constexpr int kSmemMax = 232448;
constexpr int kMaxExperts = 1024;
constexpr int kBarBytes = 704;
constexpr int kUnpackWarps = 8;     // a second set gained nothing
constexpr int kEpiSets = 2;         // sets of four epilogue warps; one: 183 us instead of 169
constexpr int kThreads = kUnpackWarps * 32 + kEpiSets * 128 + 96;

struct Params {
  const int32_t *pairs, *first, *tiles;
  const uint16_t* scales[2];  // gated: gate, up
  const uint16_t* biases[2];
  const __nv_bfloat16* bias[2];
  void* out;
  int64_t out_stride;
  int total, experts, n_out, groups, num_kb, max_tiles;
  int cap, box, ps, nx, na, nbuf, act, chains;
  int* status;  // on the host; set to 1 if a wait ran out or the plan did not fit together
};

// That word, one for the process: a launch that fails writes it, the host looks after it has waited for the stream anyway.
static int* status_word(bool make) {
  static std::atomic<int*> word{nullptr};
  static std::mutex lock;
  int* w = word.load(std::memory_order_acquire);
  if (w || !make) return w;
  std::lock_guard<std::mutex> hold(lock);
  w = word.load(std::memory_order_acquire);
  if (w) return w;
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // an allocation is no part of a capture that may be under way
  const bool swapped = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
  void* p = nullptr;
  const cudaError_t e = cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped);
  if (swapped) cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) return nullptr;
  w = static_cast<int*>(p);
  *w = 0;
  word.store(w, std::memory_order_release);
  return w;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}

struct Item {
  int expert, n0, row0, nrows;
};

// The last expert whose running count of tiles is not past i (empty ones are stepped over).
__device__ __forceinline__ int expert_of_tile(const int* tiles, int n, int i) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tiles[mid] <= i) lo = mid; else hi = mid;
  }
  return lo;
}

template <int FEATURES>
__device__ __forceinline__ Item item_at(const Params& p, const int* tiles, const int* first, int ft, int i) {
  Item w;
  w.expert = expert_of_tile(tiles, p.experts, i / ft);
  const int nt = tiles[w.expert + 1] - tiles[w.expert], n = first[w.expert + 1] - first[w.expert];
  const int local = i - tiles[w.expert] * ft, f = local / nt, tile = local - f * nt;
  const int per = ((n + nt - 1) / nt + 15) & ~15;
  w.n0 = f * FEATURES;
  w.row0 = first[w.expert] + tile * per;
  w.nrows = min(per, n - tile * per);
  return w;
}

__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
__device__ __forceinline__ float clamp_f16(float v) { return fminf(fmaxf(v, -65504.f), 65504.f); }

// Activations of the rounded projections, in fp32 but for the exponential and the quotient, which are the fast ones: by CUDA's error
// bounds some 5 + 1.2 |g| last bits (2^-21 near nought, 2^-16 at g = -88), in front of a rounding to the 8 bits of bf16.
__device__ __forceinline__ float activate(int act, float g, float u) {
  if (act == 1) {  // clipped SwiGLU: alpha 1.702, limit 7
    g = g > 7.f ? 7.f : g;
    u = u > 7.f ? 7.f : u < -7.f ? -7.f : u;
    return g * __fdividef(1.f, 1.f + __expf(-1.702f * g)) * (u + 1.f);
  }
  return g * __fdividef(1.f, 1.f + __expf(-g)) * u;
}

// SK: 64-column blocks of a step of the A ring and of x.
template <int BITS, int G, bool GATED, int SK>
__global__ void __launch_bounds__(kThreads, 1)
expert_qgemm_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap u_map,
                    const __grid_constant__ CUtensorMap x_map, const Params p) {
  constexpr int FEATURES = GATED ? 64 : 128, A_COLS = 32 * SK;
  constexpr int KB_PER_P = 1024 / BITS / 64;     // 64-column blocks of a packed stage
  constexpr int U = SK < 2 ? SK : 2;             // that a thread unpacks at a time
  constexpr int CH_T = BITS / 4;                 // 16-byte packed chunks a thread unpacks per block
  constexpr int W_EPI = kUnpackWarps, W_W = W_EPI + 4 * kEpiSets, W_X = W_W + 1, W_MMA = W_W + 2;
  extern __shared__ __align__(1024) uint8_t raw[];
  const uint32_t base = (smem_u32(raw) + 1023u) & ~1023u;
  const uint32_t xb = p.cap * 128 * SK, row_bytes = p.groups * 2, half_sb = 128 * row_bytes, sb_bytes = 2 * half_sb;
  const uint32_t sm_x = base + p.ps * kPacked, sm_sb = sm_x + p.nx * xb, sm_ex = sm_sb + p.nbuf * sb_bytes;
  const uint32_t sm_bar = sm_ex + (GATED ? kEpiSets * 8192 : 0);
  const uint32_t bar_full_p = sm_bar, bar_empty_p = bar_full_p + 64, bar_full = bar_empty_p + 64, bar_empty = bar_full + 8 * kMaxA;
  const uint32_t bar_acc = bar_empty + 8 * kMaxA, bar_free = bar_acc + 16, bar_full_sb = bar_free + 16, bar_empty_sb = bar_full_sb + 16;
  const uint32_t bar_full_x = bar_empty_sb + 16, bar_empty_x = bar_full_x + 8 * kMaxX, tmem_ptr = bar_empty_x + 8 * kMaxX;
  uint8_t* gen = raw + (sm_bar - smem_u32(raw));
  volatile uint32_t* tmem_gen = reinterpret_cast<volatile uint32_t*>(gen + (tmem_ptr - sm_bar));
  volatile int* sfail = reinterpret_cast<volatile int*>(gen + (tmem_ptr - sm_bar) + 4);
  int* tiles = reinterpret_cast<int*>(gen + kBarBytes);
  int* first = tiles + p.experts + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, chains = SK == 4 ? p.chains : 1;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.ps; ++i) {
      mbar_init(bar_full_p + 8 * i, 1);
      mbar_init(bar_empty_p + 8 * i, kUnpackWarps);
    }
    for (int i = 0; i < p.na; ++i) {
      mbar_init(bar_full + 8 * i, 8);
      mbar_init(bar_empty + 8 * i, 1);
    }
    for (int i = 0; i < p.nx; ++i) {
      mbar_init(bar_full_x + 8 * i, 1);
      mbar_init(bar_empty_x + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar_acc + 8 * i, 1);
      mbar_init(bar_free + 8 * i, 4 * kEpiSets);
      mbar_init(bar_full_sb + 8 * i, 1);
      mbar_init(bar_empty_sb + 8 * i, kUnpackWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *sfail = 0;
  }
  if (warp == W_MMA) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_ptr), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  // The plan is checked on the way in: running counts from nought to all rows that fit together, so that whatever they hold, every
  // row below is a row of the operands and every row of the result is written.
  for (int i = threadIdx.x; i <= p.experts; i += blockDim.x) {
    const int t = p.tiles[i], f = p.first[i];
    tiles[i] = t;
    first[i] = f;
    const int tn = i < p.experts ? p.tiles[i + 1] : t, fn = i < p.experts ? p.first[i + 1] : p.total;
    if (t < 0 || f < 0 || t > p.max_tiles || f > p.total || (i == 0 && (t != 0 || f != 0)) || (i == p.experts && f != p.total) ||
        (i < p.experts && (fn < f || tn - t != (fn - f + p.cap - 1) / p.cap)))
      *sfail = 1;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_gen;
  const int ft = (p.n_out + FEATURES - 1) / FEATURES;
  const bool sound = *sfail == 0;
  const int items = sound ? tiles[p.experts] * ft : 0;
  __syncthreads();
  bool ok = true;

  if (warp == W_W) {
    // ===== packed words; scales and biases =====
    int st = 0, it = 0, issued = 0, sb_issued = 0;
    uint32_t ph = 1;
    const int stages = (p.num_kb + KB_PER_P - 1) / KB_PER_P;
    for (int i = blockIdx.x; ok && i < items; i += gridDim.x, ++it) {
      const Item w = item_at<FEATURES>(p, tiles, first, ft, i);
      const int live = GATED ? 128 : min(128, p.n_out - w.n0);  // weight rows: 64 or 128
      const int r0 = w.expert * p.n_out + w.n0;
      const int buf = p.nbuf == 2 ? it & 1 : 0, use = p.nbuf == 2 ? it >> 1 : it;
      if (!(ok = mbar_wait_or_fail(bar_empty_sb + 8 * buf, (use & 1) ^ 1))) break;
      if (elect_one()) {
        const uint32_t bar = bar_full_sb + 8 * buf, dst = sm_sb + buf * sb_bytes;
        mbar_expect_tx(bar, 2 * live * row_bytes);
        const int64_t at = (int64_t)r0 * p.groups;
        if (GATED) {
          bulk_load(dst, p.scales[0] + at, 64 * row_bytes, bar);
          bulk_load(dst + 64 * row_bytes, p.scales[1] + at, 64 * row_bytes, bar);
          bulk_load(dst + half_sb, p.biases[0] + at, 64 * row_bytes, bar);
          bulk_load(dst + half_sb + 64 * row_bytes, p.biases[1] + at, 64 * row_bytes, bar);
        } else {
          bulk_load(dst, p.scales[0] + at, live * row_bytes, bar);
          bulk_load(dst + half_sb, p.biases[0] + at, live * row_bytes, bar);
        }
      }
      __syncwarp();
      ++sb_issued;
      for (int s = 0; s < stages; ++s) {
        if (!(ok = mbar_wait_parked_or_fail(bar_empty_p + 8 * st, ph))) break;
        if (elect_one()) {
          const uint32_t bar = bar_full_p + 8 * st, dst = base + st * kPacked;
          mbar_expect_tx(bar, live * 128);
          tma_load_2d(dst, &w_map, bar, s * 32, r0);
          if (live > 64) tma_load_2d(dst + kPacked / 2, GATED ? &u_map : &w_map, bar, s * 32, GATED ? r0 : r0 + 64);
        }
        __syncwarp();
        ++issued;
        if (++st == p.ps) st = 0, ph ^= 1;
      }
    }
    if (!ok) {
      if (lane == 0) *sfail = 1;
      // the copies in flight land before the CTA's memory goes away
      for (int j = min(issued, p.ps); j > 0; --j) {
        if (--st < 0) st = p.ps - 1, ph ^= 1;
        mbar_wait_or_fail(bar_full_p + 8 * st, ph ^ 1);
      }
      for (int j = max(0, sb_issued - p.nbuf); j < sb_issued; ++j)
        mbar_wait_or_fail(bar_full_sb + 8 * (p.nbuf == 2 ? j & 1 : 0), (p.nbuf == 2 ? j >> 1 : j) & 1);
    }
  } else if (warp == W_X) {
    // ===== rows of x =====
    int st = 0, issued = 0;
    uint32_t ph = 1;
    for (int i = blockIdx.x; ok && i < items; i += gridDim.x) {
      const Item w = item_at<FEATURES>(p, tiles, first, ft, i);
      const int boxes = (w.nrows + p.box - 1) / p.box;
      for (int kb = 0; kb < p.num_kb; kb += SK) {
        if (!(ok = mbar_wait_parked_or_fail(bar_empty_x + 8 * st, ph))) break;
        if (elect_one()) {
          const uint32_t bar = bar_full_x + 8 * st, dst = sm_x + st * xb;
          mbar_expect_tx(bar, boxes * p.box * 128 * SK);  // columns past K arrive as zeros
          if constexpr (SK > 1) {
            tma_load_3d(dst, &x_map, bar, 0, w.row0, kb);  // one box is the whole tile
          } else {
            for (int j = 0; j < boxes; ++j) tma_load_3d(dst + j * p.box * 128, &x_map, bar, 0, w.row0 + j * p.box, kb);
          }
        }
        __syncwarp();
        ++issued;
        if (++st == p.nx) st = 0, ph ^= 1;
      }
    }
    // the last products' arrivals find the CTA still there; after a failure the copies in flight land
    for (int j = min(issued, p.nx); j > 0; --j) {
      if (--st < 0) st = p.nx - 1, ph ^= 1;
      if (!mbar_wait_or_fail((ok ? bar_empty_x : bar_full_x) + 8 * st, ph ^ 1) && ok) ok = false;
    }
    if (!ok && lane == 0) *sfail = 1;
  } else if (warp == W_MMA) {
    // ===== products =====
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t x_desc = make_smem_desc(sm_x);
    const uint32_t a0 = tb + 2 * chains * p.cap, half = p.cap * 8;  // a 64-column block of x, in the descriptor's units
    int st = 0, xs = 0, it = 0;
    uint32_t ph = 0, xph = 0;
    for (int i = blockIdx.x; ok && i < items; i += gridDim.x, ++it) {
      const Item w = item_at<FEATURES>(p, tiles, first, ft, i);
      const uint32_t idesc = make_idesc(0, 128, (w.nrows + 15) & ~15), d = tb + (it & 1) * chains * p.cap;
      if (!(ok = mbar_wait_or_fail(bar_free + 8 * (it & 1), ((it >> 1) & 1) ^ 1))) break;
      int chain = 0;
      for (int kb = 0; kb < p.num_kb; kb += SK) {
        // both looked at at once, then waited for what was not ready
        const bool rx = mbar_try_wait(bar_full_x + 8 * xs, xph), ra = mbar_try_wait(bar_full + 8 * st, ph);
        ok = (rx || mbar_wait_or_fail(bar_full_x + 8 * xs, xph)) && (ra || mbar_wait_or_fail(bar_full + 8 * st, ph));
        if (!ok) break;
        tc_fence_after();
        if (elect_one()) {
          const uint64_t x = x_desc + xs * (xb >> 4);
          const uint32_t a = a0 + st * A_COLS;
#pragma unroll
          for (int h = 0; h < SK; ++h)
            if (h == 0 || kb + h < p.num_kb) {
#pragma unroll
              for (int k = 0; k < 4; ++k)
                tc_mma_f16_ts(d + chain * p.cap, a + 32 * h + 8 * k, x + h * half + 2 * k, idesc,
                              h == 0 && k == 0 ? (kb >= chains * SK ? 1u : 0u) : 1u);
            }
          tc_commit(bar_empty_x + 8 * xs);
          tc_commit(bar_empty + 8 * st);
          if (kb + SK >= p.num_kb) tc_commit(bar_acc + 8 * (it & 1));
        }
        __syncwarp();
        if (++st == p.na) st = 0, ph ^= 1;
        if (++xs == p.nx) xs = 0, xph ^= 1;
        if (++chain == chains) chain = 0;
      }
    }
    if (!ok && lane == 0) *sfail = 1;
  } else if (warp < W_EPI) {
    // ===== unpack =====
    const int r = threadIdx.x & 127, hsel = (threadIdx.x >> 7) & 1;
    const uint32_t xr = r & 7, tm_a = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 2 * chains * p.cap + hsel * 16;
    int pst = 0, it = 0, slot = 0;
    uint32_t pph = 0, sph = 1;
    for (int i = blockIdx.x; ok && i < items; i += gridDim.x, ++it) {
      const int buf = p.nbuf == 2 ? it & 1 : 0, use = p.nbuf == 2 ? it >> 1 : it;
      if (!(ok = mbar_wait_or_fail(bar_full_sb + 8 * buf, use & 1))) break;
      const uint32_t srow = sm_sb + buf * sb_bytes + r * row_bytes;
      for (int kb0 = 0; ok && kb0 < p.num_kb; kb0 += KB_PER_P) {
        if (!(ok = mbar_wait_or_fail(bar_full_p + 8 * pst, pph))) break;
        const uint32_t prow = base + pst * kPacked + r * 128;
#pragma unroll
        for (int j = 0; j < KB_PER_P; j += U) {
          const int kb = kb0 + j;
          if (kb >= p.num_kb) continue;
          const int part = (kb / U) % (SK / U);  // of the step
          const bool last = part == SK / U - 1 || kb + U >= p.num_kb;
          uint4 pk[U][CH_T];
          uint16_t sr[U], br[U];
#pragma unroll
          for (int h = 0; h < U; ++h) {  // past K's end: whatever the stage holds, multiplied by nothing
#pragma unroll
            for (int c = 0; c < CH_T; ++c)
              asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                           : "=r"(pk[h][c].x), "=r"(pk[h][c].y), "=r"(pk[h][c].z), "=r"(pk[h][c].w)
                           : "r"(prow + (((uint32_t)((j + h) * 2 * CH_T + hsel * CH_T + c) ^ xr) << 4)));
            const uint32_t g = G >= 64 ? (uint32_t)(kb + h) * 64 / G : (uint32_t)(kb + h) * 2 + hsel;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(sr[h]) : "r"(srow + 2 * g));
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(br[h]) : "r"(srow + half_sb + 2 * g));
          }
          uint32_t av[16 * U];
#pragma unroll
          for (int h = 0; h < U; ++h) {
            const float sf = qtc::Cvt<__nv_bfloat16>::to_f(sr[h]), bf = qtc::Cvt<__nv_bfloat16>::to_f(br[h]);
            const __half2 s2 = __float2half2_rn(sf), b2 = __float2half2_rn(bf);
            uint32_t* o = av + 16 * h;
#pragma unroll
            for (int c = 0; c < CH_T; ++c) {
              const uint32_t words[4] = {pk[h][c].x, pk[h][c].y, pk[h][c].z, pk[h][c].w};
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                if constexpr (BITS == 4) {
                  const uint4 v = qtc::dequant_word4<__half, true>(words[k], s2, b2);
                  o[4 * k] = v.x; o[4 * k + 1] = v.y; o[4 * k + 2] = v.z; o[4 * k + 3] = v.w;
                } else {
                  const uint2 v = qtc::dequant_word8<__half>(words[k], sf, bf);
                  o[8 * c + 2 * k] = v.x; o[8 * c + 2 * k + 1] = v.y;
                }
              }
            }
          }
          if (part == 0 && !(ok = mbar_wait_or_fail(bar_empty + 8 * slot, sph))) break;
          tc_fence_after();
#pragma unroll
          for (int h = 0; h < U; ++h) tmem_st16_nowait(tm_a + slot * A_COLS + 32 * (U * part + h), av + 16 * h);
          if (last) {
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_full + 8 * slot);
            if (++slot == p.na) slot = 0, sph ^= 1;
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_empty_p + 8 * pst);
        if (++pst == p.ps) pst = 0, pph ^= 1;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_empty_sb + 8 * buf);
    }
    if (!ok && lane == 0) *sfail = 1;
  } else {
    // ===== epilogue: thread = weight row of the tile; the sets of four warps take columns in turn =====
    const int q = warp & 3, r = q * 32 + lane, set = (warp - W_EPI) >> 2;
    const uint32_t tm = tmem + ((uint32_t)(q * 32) << 16);
    const int used = min(chains, (p.num_kb + SK - 1) / SK);
    int it = 0, flip = 0;
    for (int i = blockIdx.x; i < items; i += gridDim.x, ++it) {
      const Item w = item_at<FEATURES>(p, tiles, first, ft, i);
      const int which = GATED ? r >> 6 : 0, feature = w.n0 + (GATED ? r & 63 : r);
      const __nv_bfloat16* bp = p.bias[which];
      const float bias = bp != nullptr && feature < p.n_out ? __bfloat162float(bp[(int64_t)w.expert * p.n_out + feature]) : 0.f;
      ok = mbar_wait_parked_or_fail(bar_acc + 8 * (it & 1), (it >> 1) & 1);
      if constexpr (GATED) {  // a set's warps meet below: they go on together or not at all
        uint32_t all = ok;
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %0, 0;\n\tbar.red.and.pred q, %1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                     : "+r"(all) : "r"(1 + set) : "memory");
        ok = all != 0;
      }
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tm + (it & 1) * chains * p.cap;
      auto sums = [&](uint32_t col, uint32_t (&v)[16]) {
        tmem_ld<16>(d + col, v);
        for (int j = 1; j < used; ++j) {
          uint32_t t[16];
          tmem_ld<16>(d + j * p.cap + col, t);
#pragma unroll
          for (int c = 0; c < 16; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) + __uint_as_float(t[c]));
        }
      };
      if constexpr (GATED) {
        __half* out = reinterpret_cast<__half*>(p.out);
        for (int c0 = set * 32; c0 < w.nrows; c0 += 32 * kEpiSets) {
          uint32_t mine[16], other[16] = {};
          // gate lanes finish the first 16 columns, up lanes the second: each hands its other 16 over
          const bool second = c0 + 16 < w.nrows;  // the last 32 columns may hold one sixteen only
          if (second || !which) sums(c0 + which * 16, mine);
          if (second || which) sums(c0 + (which ? 0 : 16), other);
          const uint32_t ex = sm_ex + set * 8192 + (flip & 1) * 4096;
#pragma unroll
          for (int c = 0; c < 16; c += 2) {
            const __nv_bfloat162 v = __floats2bfloat162_rn(__uint_as_float(other[c]) + bias, __uint_as_float(other[c + 1]) + bias);
            asm volatile("st.shared.b32 [%0], %1;" ::"r"(ex + which * 2048 + (c / 2) * 256 + (r & 63) * 4),
                         "r"(*reinterpret_cast<const uint32_t*>(&v)) : "memory");
          }
          asm volatile("bar.sync %0, 128;" ::"r"(1 + set) : "memory");
          ++flip;
          if (!second && which) continue;
          const int cols = min(16, w.nrows - c0 - which * 16);
          constexpr int PAIR = BITS == 4 ? 4 : 1;  // the lane whose feature is the next column of the copy
          const bool odd = lane & PAIR;
          const int at = BITS == 4 ? (feature & ~7) + 2 * (feature & 3) : feature & ~1;
          const int64_t row = w.row0 + c0 + which * 16;
#pragma unroll
          for (int c = 0; c < 16; c += 2) {
            uint32_t t;
            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(t) : "r"(ex + (which ^ 1) * 2048 + (c / 2) * 256 + (r & 63) * 4) : "memory");
            float h[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float a = round_bf16(__uint_as_float(mine[c + e]) + bias), b = __uint_as_float(e ? t & 0xffff0000u : t << 16);
              h[e] = clamp_f16(round_bf16(which ? activate(p.act, b, a) : activate(p.act, a, b)));
            }
            // two lanes swap a column each: one 4-byte store of two features a lane for two columns
            const float got = __shfl_xor_sync(0xffffffffu, odd ? h[0] : h[1], PAIR);
            const __half2 v = odd ? __floats2half2_rn(got, h[1]) : __floats2half2_rn(h[0], got);
            const int col = c + (odd ? 1 : 0);
            if (col < cols) *reinterpret_cast<__half2*>(out + (row + col) * p.out_stride + at) = v;
          }
        }
      } else {
        __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + (feature & ~1);
        const bool odd = lane & 1, live = feature < p.n_out;
        for (int c0 = set * 16; c0 < w.nrows; c0 += 16 * kEpiSets) {
          uint32_t u[16];
          sums(c0, u);
          const int place = (int)min((uint32_t)p.pairs[w.row0 + min(c0 + (lane & 15), w.nrows - 1)], (uint32_t)p.total - 1);
#pragma unroll
          for (int c = 0; c < 16; c += 2) {
            const float a = __uint_as_float(u[c]) + bias, b = __uint_as_float(u[c + 1]) + bias;
            const float got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
            const __nv_bfloat162 v = odd ? __floats2bfloat162_rn(got, b) : __floats2bfloat162_rn(a, got);
            const int col = c + (odd ? 1 : 0);
            const int64_t row = __shfl_sync(0xffffffffu, place, col);
            if (live && c0 + col < w.nrows) *reinterpret_cast<__nv_bfloat162*>(out + row * p.out_stride) = v;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_free + 8 * (it & 1));
    }
    if (!ok && lane == 0) *sfail = 1;
  }
  tc_fence_before();
  __syncthreads();
  if (*sfail) {
    // What should have been written here is NaN (0x7fff in both types), never what the memory held: everything for a plan that
    // does not fit together, else this CTA's items.
    const uint32_t nan2 = 0x7fff7fffu;
    auto fill = [&](int64_t row, int col) { *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.out) + row * p.out_stride + col) = nan2; };
    if (!sound) {
      const int half = p.n_out / 2;
      for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (int64_t)p.total * half; i += (int64_t)gridDim.x * blockDim.x)
        fill(i / half, (int)(i % half) * 2);
    }
    for (int i = blockIdx.x; i < items; i += gridDim.x) {
      const Item w = item_at<FEATURES>(p, tiles, first, ft, i);
      for (int j = threadIdx.x; j < w.nrows * (FEATURES / 2); j += blockDim.x) {
        const int r = w.row0 + j / (FEATURES / 2), c = w.n0 + j % (FEATURES / 2) * 2;
        if (c < p.n_out) fill(GATED ? r : (int64_t)min((uint32_t)p.pairs[r], (uint32_t)p.total - 1), c);
      }
    }
    if (threadIdx.x == 0) {
      *reinterpret_cast<volatile int*>(p.status) = 1;
      __threadfence_system();
    }
  }
  if (warp == W_MMA) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
}

// ---- rows grouped by expert, as fp16 --------------------------------------------------------------------------
// y[i] = x[pairs[i] / top], saturated; with `permute` every eight columns in the order 0 4 1 5 2 6 3 7.
__global__ void __launch_bounds__(256)
group_rows_kernel(const __nv_bfloat16* x, const int32_t* pairs, __half* y, int total, int top, int cols, int64_t x_stride, int permute) {
  pdl_trigger();
  pdl_wait();
  const int vec = cols >> 3;
  const int64_t n = (int64_t)total * vec;
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
    const int r = (int)(i / vec), c = (int)(i - (int64_t)r * vec) * 8;
    const int src = (int)min((uint32_t)pairs[r], (uint32_t)total - 1) / top;
    const uint4 v = *reinterpret_cast<const uint4*>(x + src * x_stride + c);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    __half h[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float f = clamp_f16(__uint_as_float(k & 1 ? w[k / 2] & 0xffff0000u : w[k / 2] << 16));
      h[k] = __float2half_rn(f);
    }
    uint4 o;
    __half2* o2 = reinterpret_cast<__half2*>(&o);
#pragma unroll
    for (int k = 0; k < 4; ++k) o2[k] = permute ? __halves2half2(h[k], h[k + 4]) : __halves2half2(h[2 * k], h[2 * k + 1]);
    *reinterpret_cast<uint4*>(y + (int64_t)r * cols + c) = o;
  }
}

// ---- weighted sum over a row's experts ----------------------------------------------------------------------
__global__ void __launch_bounds__(256)
weighted_sum_kernel(const __nv_bfloat16* y, const float* weights, __nv_bfloat16* out, int rows, int top, int cols) {
  pdl_trigger();
  pdl_wait();
  const int vec = cols >> 3;
  const int64_t n = (int64_t)rows * vec;
  for (int64_t i = blockIdx.x * 256ll + threadIdx.x; i < n; i += gridDim.x * 256ll) {
    const int64_t r = i / vec, c = (i - r * vec) * 8;
    float acc[8] = {};
    for (int j = 0; j < top; ++j) {
      const float s = weights[r * top + j];
      const uint4 v = *reinterpret_cast<const uint4*>(y + (r * top + j) * cols + c);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int k = 0; k < 8; ++k) acc[k] = fmaf(s, __uint_as_float(k & 1 ? w[k / 2] & 0xffff0000u : w[k / 2] << 16), acc[k]);
    }
    uint4 o;
    __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int k = 0; k < 4; ++k) o2[k] = __floats2bfloat162_rn(acc[2 * k], acc[2 * k + 1]);
    *reinterpret_cast<uint4*>(out + r * cols + c) = o;
  }
}

// ---- router product and choice --------------------------------------------------------------------------------
// A block has 16 rows and all experts; its warps split K and add up through shared memory.  A decode step's few blocks are bound
// by the way to L2, round by round: with WARPS = 32 (16 for more than 32 experts, by registers) 32 x 2880 by
// 32 experts takes 9.6 us, with 8 warps 20.3.  Products are exact; the tensor cores add them up in 32 bits, in chains of
// K / WARPS.  A logit on the edge between two bf16 values may so go another way than with another order of the sum: of 4096 rows,
// 9 at 2880 columns by 32 experts have a logit that is not float64's, by an fp32 product with a library 23; 4096 by 64: 13 and 29;
// 2048 by 128: 4 and 3.  Both operands are read in 16-byte pieces, so the columns of a 32-wide step go to the two products in
// another order than they lie in, the same for both.
constexpr int kRouteTop = 32;

template <int NT, int WARPS>  // NT: blocks of 8 experts
__global__ void __launch_bounds__(WARPS * 32)
route_kernel(const __nv_bfloat16* x, const __nv_bfloat16* w, const __nv_bfloat16* bias, int32_t* chosen, float* scores, int rows,
             int width, int experts, int top, int64_t x_stride, int over_all, int norm) {
  extern __shared__ float red[];  // [warps][16 rows][NT * 8 + 1]
  constexpr int EP = NT * 8 + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, row0 = blockIdx.x * 16;
  pdl_trigger();
  pdl_wait();
  float acc[NT][4] = {};
  const __nv_bfloat16* x0 = x + (int64_t)min(row0 + g, rows - 1) * x_stride + t * 8;
  const __nv_bfloat16* x1 = x + (int64_t)min(row0 + g + 8, rows - 1) * x_stride + t * 8;
#pragma unroll 1
  for (int k = warp * 32; k < width; k += WARPS * 32) {
    const uint4 a = *reinterpret_cast<const uint4*>(x0 + k), b = *reinterpret_cast<const uint4*>(x1 + k);
    uint4 v[NT];
#pragma unroll
    for (int n = 0; n < NT; ++n) v[n] = *reinterpret_cast<const uint4*>(w + (int64_t)min(n * 8 + g, experts - 1) * width + t * 8 + k);
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                   : "+f"(acc[n][0]), "+f"(acc[n][1]), "+f"(acc[n][2]), "+f"(acc[n][3])
                   : "r"(a.x), "r"(b.x), "r"(a.y), "r"(b.y), "r"(v[n].x), "r"(v[n].y));
      asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                   : "+f"(acc[n][0]), "+f"(acc[n][1]), "+f"(acc[n][2]), "+f"(acc[n][3])
                   : "r"(a.z), "r"(b.z), "r"(a.w), "r"(b.w), "r"(v[n].z), "r"(v[n].w));
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int c = 0; c < 4; ++c) red[(warp * 16 + g + (c >> 1) * 8) * EP + n * 8 + t * 2 + (c & 1)] = acc[n][c];
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * NT * 8; i += WARPS * 32) {  // the logits, over the first warp's part
    const int r = i / (NT * 8), e = i - r * (NT * 8);
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) s += red[(k * 16 + r) * EP + e];
    if (bias != nullptr && e < experts) s += __bfloat162float(bias[e]);
    red[r * EP + e] = round_bf16(s) + 0.f;  // one zero: -0 and 0 tie
  }
  __syncthreads();
  constexpr int PER = (NT * 8 + 31) / 32;  // experts a lane looks after
  for (int r = warp; r < 16; r += WARPS) {
    const int row = row0 + r;
    if (row >= rows) break;
    float v[PER], m = -INFINITY;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int e = lane + 32 * j;
      v[j] = -INFINITY;
      if (e < experts) {
        v[j] = red[r * EP + e];
        m = fmaxf(m, v[j]);
      }
    }
    if (over_all) {  // softmax over all experts before the choice
      m = warp_max(m);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < PER; ++j)
        if (lane + 32 * j < experts) sum += v[j] = expf(v[j] - m);
      sum = warp_sum(sum);
#pragma unroll
      for (int j = 0; j < PER; ++j) v[j] = v[j] / sum;
    }
    uint32_t left = 0;  // bit j: expert lane + 32 j can be chosen
#pragma unroll
    for (int j = 0; j < PER; ++j) left |= lane + 32 * j < experts ? 1u << j : 0u;
    float mine = -INFINITY;  // lane j: the value of choice j
    for (int c = 0; c < top; ++c) {
      uint32_t best = 0;
      int at = 0x7fffffff;
      float val = 0.f;
#pragma unroll
      for (int j = PER - 1; j >= 0; --j) {  // largest first, NaN before all, ties to the lowest number
        const uint32_t bits = __float_as_uint(v[j]);
        const uint32_t key = v[j] != v[j] ? 0xffffffffu : bits ^ ((int32_t)bits < 0 ? 0xffffffffu : 0x80000000u);
        if ((left >> j & 1) && key >= best) best = key, at = lane + 32 * j, val = v[j];
      }
      const uint32_t top_key = __reduce_max_sync(0xffffffffu, best);
      const int e = __reduce_min_sync(0xffffffffu, best == top_key ? at : 0x7fffffff);
      val = __shfl_sync(0xffffffffu, val, e & 31);
      if (lane == (e & 31)) left &= ~(1u << (e >> 5));
      if (lane == c) mine = val;
      if (lane == 0) chosen[(int64_t)row * top + c] = min(e, experts - 1);
    }
    if (!over_all) {
      const float largest = __shfl_sync(0xffffffffu, mine, 0), e = lane < top ? expf(mine - largest) : 0.f;
      mine = e / warp_sum(e);
    } else if (norm) {
      mine = mine / warp_sum(lane < top ? mine : 0.f);
    }
    if (lane < top) scores[(int64_t)row * top + lane] = mine;
  }
}

// ---- host ---------------------------------------------------------------------------------------------------
struct Rings {
  int cap, sk, ps, nx, nbuf, smem;
};

constexpr int kCaps[] = {16, 32, 64, 96, 128, 160, kMaxTile};
constexpr int kNumCaps = 7;

// Accumulators that a result's steps of K go to in turn: what fits beside two steps of A, for tiles whose GEMM split K before.
static int chains_of(int cap) { return cap <= 32 ? 4 : cap <= 64 ? 2 : 1; }

// Rings beside tiles of `cap` rows: three stages of packed words and the x of two steps (narrow tiles) or four 64-column blocks
// (wide ones) at least, with the scales of two items if they fit.
static bool rings_of(Rings& o, int cap, int experts, int k, int group, bool gated) {
  const int sb = 2 * 128 * (k / group) * 2, sk = cap <= 64 ? 4 : 1, xb = cap * 128 * sk;
  for (int nbuf = 2; nbuf >= 1; --nbuf) {
    const int room = kSmemMax - (1024 + nbuf * sb + (gated ? kEpiSets * 8192 : 0) + kBarBytes + 8 * (experts + 1));
    int ps = 3, nx = sk == 4 ? 2 : 4;
    if (room < ps * kPacked + nx * xb) continue;
    auto left = [&] { return room - ps * kPacked - nx * xb; };
    while (nx < (sk == 4 ? 3 : 6) && left() >= xb) ++nx;
    while (ps < 6 && left() >= kPacked) ++ps;
    while (nx < (sk == 4 ? 4 : 8) && left() >= xb) ++nx;
    o = {cap, sk, ps, nx, nbuf, kSmemMax - left()};
    return true;
  }
  return false;
}

// The tile that holds most experts' rows at once when they spread as if drawn (mean and three deviations), smaller where the
// rings would not fit beside it.
static int choose_cap(int rows, int top, int experts, int k, int group, bool gated) {
  const double mean = (double)rows * top / experts;
  const double want = mean + 3.0 * std::sqrt(mean);
  int c = kNumCaps - 1;
  while (c > 0 && (kCaps[c - 1] >= want || kCaps[c - 1] >= rows)) --c;
  Rings r;
  for (; c >= 0; --c)
    if (rings_of(r, kCaps[c], experts, k, group, gated)) return kCaps[c];
  return 0;
}

template <int BITS, int G, bool GATED, int SK>
static int launch_steps(const b200_qexpert_product_args& a, const Rings& ring, cudaStream_t st) {
  auto kern = expert_qgemm_kernel<BITS, G, GATED, SK>;
  static int configured[16] = {0};
  int dev = 0;
  B200_CUDA_OK(cudaGetDevice(&dev));
  if (configured[dev & 15] < ring.smem) {
    B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
    configured[dev & 15] = kSmemMax;
  }
  CUtensorMap w, u, x;
  const uint64_t words = (uint64_t)a.k * BITS / 32, w_rows = (uint64_t)a.experts * a.n_out;
  const int box = SK == 4 ? ring.cap : ring.cap / 2;  // a narrow tile's whole step is one copy, a wide one is copied as far as it is full
  int rc = make_map_2d(&w, CU_TENSOR_MAP_DATA_TYPE_UINT32, a.w, words, w_rows, words * 4, 32, 64, CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (rc == B200_OK)
    rc = make_map_2d(&u, CU_TENSOR_MAP_DATA_TYPE_UINT32, GATED ? a.up_w : a.w, words, w_rows, words * 4, 32, 64,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (rc == B200_OK)
    rc = make_map_slabs(&x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.x, 64, a.total, a.k / 64, 2, (uint64_t)a.k * 2, box, SK,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  if (rc != B200_OK) return rc;
  Params p{};
  p.pairs = a.pairs;
  p.first = a.first;
  p.tiles = a.tiles;
  p.scales[0] = (const uint16_t*)a.scales;
  p.biases[0] = (const uint16_t*)a.biases;
  p.bias[0] = (const __nv_bfloat16*)a.bias;
  p.scales[1] = (const uint16_t*)a.up_scales;
  p.biases[1] = (const uint16_t*)a.up_biases;
  p.bias[1] = (const __nv_bfloat16*)a.up_bias;
  p.out = a.out;
  p.out_stride = a.n_out;
  p.total = a.total;
  p.experts = a.experts;
  p.n_out = a.n_out;
  p.groups = a.k / G;
  p.num_kb = a.k / 64;
  p.max_tiles = a.total / ring.cap + (a.experts < a.total ? a.experts : a.total);
  p.cap = ring.cap;
  p.box = box;
  p.ps = ring.ps;
  p.nx = ring.nx;
  p.chains = chains_of(ring.cap);
  p.na = std::min((512 - 2 * p.chains * ring.cap) / (32 * SK), kMaxA);
  p.nbuf = ring.nbuf;
  p.act = a.activation;
  p.status = status_word(true);
  if (!p.status) return set_error(B200_ERR_CUDA, "qexpert_product: no pinned memory for the status word");
  constexpr int FEATURES = GATED ? 64 : 128;
  const int64_t items = (int64_t)p.max_tiles * ((a.n_out + FEATURES - 1) / FEATURES);
  const int sms = sm_count() > 0 ? sm_count() : 148;
  B200_CUDA_OK(launch_pdl(kern, dim3(items < sms ? (int)items : sms), dim3(kThreads), ring.smem, st, w, u, x, p));
  return check_launch("expert_qgemm_kernel");
}

template <int BITS, int G, bool GATED>
static int launch(const b200_qexpert_product_args& a, const Rings& ring, cudaStream_t st) {
  return ring.sk == 4 ? launch_steps<BITS, G, GATED, 4>(a, ring, st) : launch_steps<BITS, G, GATED, 1>(a, ring, st);
}

template <bool GATED>
static int dispatch(const b200_qexpert_product_args& a, const Rings& r, cudaStream_t st) {
  switch (a.bits * 256 + a.group_size) {
    case 4 * 256 + 32: return launch<4, 32, GATED>(a, r, st);
    case 4 * 256 + 64: return launch<4, 64, GATED>(a, r, st);
    case 4 * 256 + 128: return launch<4, 128, GATED>(a, r, st);
    case 8 * 256 + 32: return launch<8, 32, GATED>(a, r, st);
    case 8 * 256 + 64: return launch<8, 64, GATED>(a, r, st);
    case 8 * 256 + 128: return launch<8, 128, GATED>(a, r, st);
    default: return set_error(B200_ERR_INVALID_ARGUMENT, "qexpert_product: bits %d, group %d", a.bits, a.group_size);
  }
}

static bool aligned(const void* p) { return ((uintptr_t)p & 15) == 0; }

}  // namespace qx
}  // namespace b200

using namespace b200;

extern "C" {

int b200_qexpert_tile_rows(int rows, int top, int experts, int n_out, int k, int group_size, int gated) {
  if (rows < 1 || top < 1 || experts < 1 || experts > qx::kMaxExperts || n_out < 64 || n_out % 64 || k < 64 || k % 64 ||
      !(group_size == 32 || group_size == 64 || group_size == 128) || k % group_size || (int64_t)experts * n_out >= (1ll << 31))
    return 0;
  return qx::choose_cap(rows, top, experts, k, group_size, gated != 0);
}

int b200_qexpert_product(const b200_qexpert_product_args* a, void* stream) {
  B200_CHECK_ARG(a && a->x && a->w && a->scales && a->biases && a->out && a->pairs && a->first && a->tiles,
                 "qexpert_product: null pointer argument");
  B200_CHECK_ARG(!a->gated || (a->up_w && a->up_scales && a->up_biases), "qexpert_product: a gate without its other half");
  B200_CHECK_ARG(b200_qexpert_tile_rows(1, 1, a->experts, a->n_out, a->k, a->group_size, a->gated) > 0 && (a->bits == 4 || a->bits == 8) &&
                     a->activation >= 0 && a->activation <= 1 && a->total >= 0,
                 "qexpert_product: %d experts of %d x %d, %d bits in groups of %d", a->experts, a->n_out, a->k, a->bits, a->group_size);
  const void* all[] = {a->x, a->w, a->scales, a->biases, a->out, a->up_w, a->up_scales, a->up_biases};
  for (const void* q : all) B200_CHECK_ARG(qx::aligned(q), "qexpert_product: operands start on 16 bytes");
  if (a->total == 0) return B200_OK;
  if (tc::encode_fn() == nullptr) return set_error(B200_ERR_UNSUPPORTED, "qexpert_product: no tensor maps from the driver");
  qx::Rings r;
  bool cap_ok = false;
  for (int c : qx::kCaps) cap_ok |= c == a->tile_rows;
  B200_CHECK_ARG(cap_ok && qx::rings_of(r, a->tile_rows, a->experts, a->k, a->group_size, a->gated != 0),
                 "qexpert_product: tiles of %d rows", a->tile_rows);
  return a->gated ? qx::dispatch<true>(*a, r, (cudaStream_t)stream) : qx::dispatch<false>(*a, r, (cudaStream_t)stream);
}

int b200_qexpert_status(int reset) {
  volatile int* w = qx::status_word(false);
  if (!w) return 0;
  const int v = *w;
  if (reset) *w = 0;
  return v;
}

int b200_qexpert_failed(void) { return cudaDeviceSynchronize() != cudaSuccess ? 1 : b200_qexpert_status(0); }

int b200_qexpert_rows(const void* x, const int32_t* pairs, void* y, int total, int top, int cols, int64_t x_stride, int permute, void* stream) {
  B200_CHECK_ARG(x && pairs && y && top >= 1 && cols >= 8 && cols % 8 == 0 && x_stride % 8 == 0 && qx::aligned(x) && qx::aligned(y),
                 "qexpert_rows: rows of whole 16-byte units");
  if (total <= 0) return B200_OK;
  const int64_t n = ((int64_t)total * (cols / 8) + 255) / 256;
  B200_CUDA_OK(launch_pdl(qx::group_rows_kernel, dim3((unsigned)(n < 148 * 8 ? n : 148 * 8)), dim3(256), 0, (cudaStream_t)stream,
                          (const __nv_bfloat16*)x, pairs, (__half*)y, total, top, cols, x_stride, permute));
  return check_launch("group_rows_kernel");
}

int b200_qexpert_sum(const void* y, const float* weights, void* out, int rows, int top, int cols, void* stream) {
  B200_CHECK_ARG(y && weights && out && top >= 1 && cols >= 8 && cols % 8 == 0 && qx::aligned(y) && qx::aligned(out),
                 "qexpert_sum: rows of whole 16-byte units");
  if (rows <= 0) return B200_OK;
  const int64_t n = ((int64_t)rows * (cols / 8) + 255) / 256;
  B200_CUDA_OK(launch_pdl(qx::weighted_sum_kernel, dim3((unsigned)(n < 148 * 8 ? n : 148 * 8)), dim3(256), 0, (cudaStream_t)stream,
                          (const __nv_bfloat16*)y, weights, (__nv_bfloat16*)out, rows, top, cols));
  return check_launch("weighted_sum_kernel");
}

int b200_qexpert_route(const void* x, const void* w, const void* bias, int32_t* chosen, float* scores, int rows, int width, int experts,
                       int top, int64_t x_stride, int over_all, int norm, void* stream) {
  B200_CHECK_ARG(x && w && chosen && scores, "qexpert_route: null pointer argument");
  B200_CHECK_ARG(experts >= 1 && experts <= 128 && top >= 1 && top <= experts && top <= qx::kRouteTop && width >= 32 && width % 32 == 0 &&
                     x_stride % 8 == 0 && qx::aligned(x) && qx::aligned(w),
                 "qexpert_route: %d of %d experts (at most 32 of 128) over %d columns", top, experts, width);
  if (rows <= 0) return B200_OK;
  auto go = [&](auto kern, int nt, int warps) -> int {
    const int smem = warps * 16 * (nt * 8 + 1) * 4;
    if (smem > 48 * 1024) B200_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    B200_CUDA_OK(launch_pdl(kern, dim3((rows + 15) / 16), dim3(warps * 32), smem, (cudaStream_t)stream, (const __nv_bfloat16*)x,
                            (const __nv_bfloat16*)w, (const __nv_bfloat16*)bias, chosen, scores, rows, width, experts, top, x_stride,
                            over_all, norm));
    return check_launch("route_kernel");
  };
  return experts <= 32   ? go(qx::route_kernel<4, 32>, 4, 32)
         : experts <= 64 ? go(qx::route_kernel<8, 16>, 8, 16)
                         : go(qx::route_kernel<16, 16>, 16, 16);
}

static size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

size_t b200_qexpert_block_workspace_bytes(int rows, int width, int ff, int experts, int top) {
  const size_t pairs = (size_t)rows * top;
  return 3 * up256(pairs * 4) + 2 * up256((size_t)(experts + 1) * 4) + 2 * up256(pairs * width * 2) + up256(pairs * ff * 2);
}

int b200_qexpert_block(const b200_qexpert_block_args* a, void* stream) {
  B200_CHECK_ARG(a && a->x && a->router_w && a->out && a->workspace, "qexpert_block: null pointer argument");
  if (a->rows <= 0) return B200_OK;
  const int in = b200_qexpert_tile_rows(a->rows, a->top, a->experts, a->ff, a->width, a->group_size, 1);
  const int back = b200_qexpert_tile_rows(a->rows, a->top, a->experts, a->width, a->ff, a->group_size, 0);
  if (!in || !back || a->experts > 128 || a->top > a->experts || a->top > qx::kRouteTop || a->x_stride % 8 || !qx::aligned(a->x) ||
      !qx::aligned(a->router_w) || (int64_t)a->rows * a->top >= (1ll << 31) || tc::encode_fn() == nullptr)
    return set_error(B200_ERR_UNSUPPORTED, "qexpert_block: sizes or alignment");
  for (const b200_qexpert_matrix* m : {&a->gate, &a->up, &a->down})
    if (!qx::aligned(m->w) || !qx::aligned(m->scales) || !qx::aligned(m->biases))
      return set_error(B200_ERR_UNSUPPORTED, "qexpert_block: alignment");
  B200_CHECK_ARG(a->workspace_bytes >= b200_qexpert_block_workspace_bytes(a->rows, a->width, a->ff, a->experts, a->top),
                 "qexpert_block: workspace of %zu bytes", a->workspace_bytes);
  const size_t pairs_n = (size_t)a->rows * a->top;
  char* at = reinterpret_cast<char*>(a->workspace);
  auto take = [&](size_t n) {
    char* p = at;
    at += up256(n);
    return p;
  };
  int32_t* chosen = (int32_t*)take(pairs_n * 4);
  float* scores = (float*)take(pairs_n * 4);
  int32_t* pairs = (int32_t*)take(pairs_n * 4);
  int32_t* first = (int32_t*)take((size_t)(a->experts + 1) * 4);
  int32_t* tiles = (int32_t*)take((size_t)(a->experts + 1) * 4);
  void* xs = take(pairs_n * a->width * 2);
  void* y = take(pairs_n * a->width * 2);
  void* h = take(pairs_n * a->ff * 2);
  const int tile = in < back ? in : back;
  int rc = b200_qexpert_route(a->x, a->router_w, a->router_bias, chosen, scores, a->rows, a->width, a->experts, a->top, a->x_stride,
                              a->over_all, a->norm, stream);
  if (rc == B200_OK) rc = b200_expert_plan(chosen, pairs, first, tiles, a->rows, a->experts, a->top, tile, stream);
  if (rc == B200_OK) rc = b200_qexpert_rows(a->x, pairs, xs, (int)pairs_n, a->top, a->width, a->x_stride, a->bits == 4, stream);
  b200_qexpert_product_args p{};
  p.x = xs;
  p.w = a->gate.w;
  p.scales = a->gate.scales;
  p.biases = a->gate.biases;
  p.bias = a->gate.bias;
  p.up_w = a->up.w;
  p.up_scales = a->up.scales;
  p.up_biases = a->up.biases;
  p.up_bias = a->up.bias;
  p.out = h;
  p.pairs = pairs;
  p.first = first;
  p.tiles = tiles;
  p.total = (int)pairs_n;
  p.experts = a->experts;
  p.n_out = a->ff;
  p.k = a->width;
  p.bits = a->bits;
  p.group_size = a->group_size;
  p.tile_rows = tile;
  p.gated = 1;
  p.activation = a->activation;
  if (rc == B200_OK) rc = b200_qexpert_product(&p, stream);
  p.x = h;
  p.w = a->down.w;
  p.scales = a->down.scales;
  p.biases = a->down.biases;
  p.bias = a->down.bias;
  p.up_w = nullptr;
  p.up_scales = p.up_biases = p.up_bias = nullptr;
  p.out = y;
  p.n_out = a->width;
  p.k = a->ff;
  p.gated = 0;
  if (rc == B200_OK) rc = b200_qexpert_product(&p, stream);
  if (rc == B200_OK) rc = b200_qexpert_sum(y, scores, a->out, a->rows, a->top, a->width, stream);
  return rc;
}

}  // extern "C"
