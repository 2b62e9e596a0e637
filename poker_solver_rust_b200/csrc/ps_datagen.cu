// Device side of the turn-datagen boundary pipeline: the reach-weighted
// average of boundary-value-network outputs over the 48 river cards, with card
// blocking (cfvnet/src/datagen/gpu_boundary_eval.rs:207-269 does it on the
// host in f64, and it is that pipeline's measured bottleneck).
//
// For boundary item i, player p (opponent o), river r of the 48 cards not on
// the item's 4-card board and combo c:
//   w_o[r]  = sum over combos c' without card r of reach_o[c']          (f64)
//   cfv_p[h] = (pot + stack) * sum_{r not in hand h} w_o[r] * net[i][p][r][c(h)]
//                              / sum_{r not in hand h} w_o[r]            (0 if the sum is 0)
// Player 0 is weighted by IP reach, player 1 by OOP reach, as in the reference.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ps_launch.hpp"

namespace ps {

constexpr int kRivers = 48;
constexpr int kCombos = 1326;

// (c1, c2), c1 < c2, of a combo index (inverse of card.rs:50-55): c1 is the
// last card whose first combo, c1 * (103 - c1) / 2, is at most idx
__device__ __forceinline__ void combo_cards(int idx, int& c1, int& c2) {
  int a = (int)((103.f - sqrtf((float)(10609 - 8 * idx))) * 0.5f);
  if (a * (103 - a) / 2 > idx) --a;
  if ((a + 1) * (102 - a) / 2 <= idx) ++a;
  c1 = a;
  c2 = idx - a * (101 - a) / 2 + 1;
}
// combo index of two distinct cards (card.rs:50-55)
__device__ __forceinline__ int combo_index(int a, int b) {
  const int lo = a < b ? a : b, hi = a < b ? b : a;
  return lo * (101 - lo) / 2 + hi - 1;
}

// The 48 cards not on a 4-card board, ascending; pos: the place of card c in
// that order (kRivers if it is on the board).
__device__ __forceinline__ int river_pos(const uint8_t* bd, int c) {
  int k = c;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (bd[i] == c) return kRivers;
    k -= bd[i] < c;
  }
  return k;
}

// f64 weight of every river for one item and player: the opponent's reach on
// the combos free of the river card (total minus the 51 combos holding it).
// Whole block; s_w [kRivers], s_red [32] shared; ends with a barrier.
__device__ void river_weights(const uint8_t* bd, const float* ro, double* s_w, double* s_red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double t = 0.0;
  for (int c = threadIdx.x; c < kCombos; c += blockDim.x) t += (double)ro[c];
  for (int s = 16; s > 0; s >>= 1) t += __shfl_down_sync(0xffffffffu, t, s);
  if (lane == 0) s_red[warp] = t;
  __syncthreads();
  double total = 0.0;
  for (int w = 0; w < nw; ++w) total += s_red[w];
  for (int c = warp; c < 52; c += nw) {  // a warp per card
    const int k = river_pos(bd, c);
    if (k == kRivers) continue;
    double blocked = 0.0;
    for (int x = lane; x < 52; x += 32)
      if (x != c) blocked += (double)ro[combo_index(x, c)];
    for (int s = 16; s > 0; s >>= 1) blocked += __shfl_down_sync(0xffffffffu, blocked, s);
    if (lane == 0) s_w[k] = total - blocked;
  }
  __syncthreads();
}

// Two adjacent network outputs (an even first index, so the pair is aligned).
__device__ __forceinline__ float2 net_pair(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 net_pair(const __nv_bfloat16* p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}
__device__ __forceinline__ float net_one(const float* p) { return *p; }
__device__ __forceinline__ float net_one(const __nv_bfloat16* p) { return __bfloat162float(*p); }

// One block per (item, player), two hands per thread and round (224 threads:
// three rounds cover the 663 pairs with 9 idle slots): bound by the read of the
// network's outputs, the f64 conversions close behind.  The 48 rows of a column
// pair are read sixteen at a time; whether a river blocks a hand is a bit of a
// mask, so no branch stands around a load.  One value at a time behind such a
// branch, 1024 items took 122 us of kernel time for 260 MB of bf16 outputs
// instead of 99.
constexpr int kReduceThreads = 224;
__device__ __forceinline__ uint64_t blocked_rivers(const uint8_t* bd, int combo) {
  int c1, c2;
  combo_cards(combo, c1, c2);
  const int k1 = river_pos(bd, c1), k2 = river_pos(bd, c2);
  return (1ull << k1 | 1ull << k2) & ((1ull << kRivers) - 1);  // (kRivers: the card is on the board)
}
// The sum of the weights of the rivers that do not block a hand: the sum of all
// less the blocked ones (at most two), added up directly where the difference
// would cancel.
__device__ __forceinline__ double free_weight(const double* s_w, double all, uint64_t blocked) {
  double d = all;
  for (uint64_t m = blocked; m; m &= m - 1) d -= s_w[__ffsll((long long)m) - 1];
  if (d > 1e-3 * all) return d;
  d = 0.0;
#pragma unroll 1
  for (int r = 0; r < kRivers; ++r)
    if (!(blocked >> r & 1)) d += s_w[r];
  return d;
}
__device__ __forceinline__ double all_weights(const double* s_w) {
  double d = 0.0;
#pragma unroll 8
  for (int r = 0; r < kRivers; ++r) d += s_w[r];
  return d;
}
template <typename T>
__global__ void __launch_bounds__(kReduceThreads) k_boundary_river_reduce(const __grid_constant__ ItemMeta meta,
                                                                          const T* __restrict__ net,
                                                                          const float* __restrict__ reach,
                                                                          const int32_t* __restrict__ hands, int H,
                                                                          float* __restrict__ out, bool pairs) {
  const int item = blockIdx.x >> 1, p = blockIdx.x & 1, o = p ^ 1;
  __shared__ double s_w[kRivers];
  __shared__ double s_red[32];
  const uint8_t* bd = meta.board[item];
  river_weights(bd, reach + ((size_t)item * 2 + o) * kCombos, s_w, s_red);
  const T* np_ = net + ((size_t)item * 2 + p) * kRivers * kCombos;
  const double scale = (double)meta.a[item], all = all_weights(s_w);
  float* dst = out + ((size_t)item * 2 + p) * H;
  for (int h = 2 * threadIdx.x; h < H; h += 2 * blockDim.x) {
    const bool two = h + 1 < H;
    const int ca = hands[h], cb = two ? hands[h + 1] : -1;
    const bool oka = ca >= 0 && ca < kCombos, okb = cb >= 0 && cb < kCombos;  // not a combo: no value
    const uint64_t ma = blocked_rivers(bd, oka ? ca : 0), mb = blocked_rivers(bd, okb ? cb : 0);
    const bool pair = pairs && oka && cb == ca + 1 && !(ca & 1);  // pairs: the outputs are aligned to two values
    const T* pa = np_ + (oka ? ca : 0);
    const T* pb = np_ + (okb ? cb : 0);
    double na = 0.0, nb = 0.0;
    constexpr int kRows = 16;
#pragma unroll 1
    for (int r0 = 0; r0 < kRivers; r0 += kRows) {
      float2 v[kRows];
      if (pair) {
#pragma unroll
        for (int u = 0; u < kRows; ++u) v[u] = net_pair(pa + (size_t)(r0 + u) * kCombos);
      } else {
#pragma unroll
        for (int u = 0; u < kRows; ++u)
          v[u] = make_float2(net_one(pa + (size_t)(r0 + u) * kCombos), net_one(pb + (size_t)(r0 + u) * kCombos));
      }
      const unsigned ka = (unsigned)(ma >> r0), kb = (unsigned)(mb >> r0);
#pragma unroll
      for (int u = 0; u < kRows; ++u) {
        const double w = s_w[r0 + u];
        if (!(ka >> u & 1)) na += w * (double)v[u].x;
        if (!(kb >> u & 1)) nb += w * (double)v[u].y;
      }
    }
    const double da = free_weight(s_w, all, ma), db = free_weight(s_w, all, mb);
    dst[h] = oka && da > 0.0 ? (float)(na / da * scale) : 0.0f;
    if (two) dst[h + 1] = okb && db > 0.0 ? (float)(nb / db * scale) : 0.0f;
  }
}

// The average's gradient with respect to the network's outputs, in f64 from
// f32 inputs: gy[i][p][r][c] = w[r] * (g[i][p][c] * scale / sum of w over the
// rivers free of c's cards), where the river is one of them 0 times the
// bracket: a gradient that is not finite shows there too, as in the formula.
// One block per (item, player), a column pair per thread and round: bound by
// the write of gy, which four blocks an SM do fastest (512 items 102 us a call,
// 107 with the seven that its registers allow, 110 with five and six); the
// launch asks for kGradPad bytes of shared memory that nothing uses.
constexpr int kGradPad = 47 * 1024;
__global__ void __launch_bounds__(kReduceThreads) k_river_average_grad(const __grid_constant__ ItemMeta meta,
                                                            const float* __restrict__ reach,
                                                            const float* __restrict__ g, float* __restrict__ gy,
                                                            bool pairs) {
  const int item = blockIdx.x >> 1, p = blockIdx.x & 1, o = p ^ 1;
  __shared__ double s_w[kRivers];
  __shared__ double s_red[32];
  const uint8_t* bd = meta.board[item];
  river_weights(bd, reach + ((size_t)item * 2 + o) * kCombos, s_w, s_red);
  const double scale = (double)meta.a[item], all = all_weights(s_w);
  const float* gi = g + ((size_t)item * 2 + p) * kCombos;
  float* go = gy + ((size_t)item * 2 + p) * kRivers * kCombos;
  for (int c = 2 * threadIdx.x; c < kCombos; c += 2 * blockDim.x) {  // kCombos is even
    const uint64_t ma = blocked_rivers(bd, c), mb = blocked_rivers(bd, c + 1);
    const double da = free_weight(s_w, all, ma), db = free_weight(s_w, all, mb);
    const double ka = da > 0.0 ? (double)gi[c] * scale / da : 0.0, kb = db > 0.0 ? (double)gi[c + 1] * scale / db : 0.0;
    const float za = (float)(0.0 * ka), zb = (float)(0.0 * kb);
#pragma unroll 1
    for (int r0 = 0; r0 < kRivers; r0 += 8) {
      const unsigned xa = (unsigned)(ma >> r0), xb = (unsigned)(mb >> r0);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const double w = s_w[r0 + u];
        const float2 v = make_float2(xa >> u & 1 ? za : (float)(w * ka), xb >> u & 1 ? zb : (float)(w * kb));
        float* at = go + (size_t)(r0 + u) * kCombos + c;
        if (pairs) {  // gy is aligned to two values
          *reinterpret_cast<float2*>(at) = v;
        } else {
          at[0] = v.x;
          at[1] = v.y;
        }
      }
    }
  }
}

// One block per boundary item (spot, ordinal), both players: between the
// spot's hand-order rows (stride vstride) and the item's 1326-combo rows.
__global__ void k_boundary_combo(const SpotDev* __restrict__ spots, const int2* __restrict__ items, int which,
                                 const float* __restrict__ in, float* __restrict__ out) {
  const int2 it = items[blockIdx.x];
  const SpotDev& sp = spots[it.x];
  for (int p = 0; p < 2; ++p) {
    const uint8_t* cards = sp.cards[p];
    const size_t hrow = ((size_t)it.y * 2 + p) * sp.vstride;
    const size_t crow = ((size_t)blockIdx.x * 2 + p) * kCombos;
    if (which == BC_SET_VALUES) {
      float* dst = const_cast<float*>(sp.bcfv) + hrow;
      const float* src = in + crow;
      for (int h = threadIdx.x; h < sp.vstride; h += blockDim.x)
        dst[h] = h < sp.H[p] ? src[combo_index(cards[2 * h], cards[2 * h + 1])] : 0.f;
    } else {
      const float* from = which == BC_REACH ? sp.breach : sp.bgrad;
      float* dst = out + crow;
      for (int c = threadIdx.x; c < kCombos; c += blockDim.x) dst[c] = 0.f;
      __syncthreads();
      if (from)
        for (int h = threadIdx.x; h < sp.H[p]; h += blockDim.x)
          dst[combo_index(cards[2 * h], cards[2 * h + 1])] = from[hrow + h];
      __syncthreads();
    }
  }
}

cudaError_t launch_boundary_combo(const SpotDev* spots, const int2* items, int nitems, int which,
                                  const float* in, float* out, cudaStream_t s) {
  if (nitems <= 0) return cudaSuccess;
  k_boundary_combo<<<nitems, 256, 0, s>>>(spots, items, which, in, out);
  return cudaGetLastError();
}

// One block per spot, both players: between the spot's hand-order vectors and
// its 1326-combo rows.
__global__ void k_spot_combo(const SpotDev* __restrict__ spots, int which, const float* __restrict__ in,
                             float* __restrict__ out) {
  const SpotDev& sp = spots[blockIdx.x];
  for (int p = 0; p < 2; ++p) {
    const uint8_t* cards = sp.cards[p];
    const size_t crow = ((size_t)blockIdx.x * 2 + p) * kCombos;
    if (which == SC_COT) {
      float* dst = sp.adj_g[p];
      for (int h = threadIdx.x; h < sp.hs[p]; h += blockDim.x)
        dst[h] = h < sp.H[p] ? in[crow + combo_index(cards[2 * h], cards[2 * h + 1])] : 0.f;
    } else {
      const float* from = which == SC_ROOT ? sp.root_out[p] : sp.adj_dw[p];
      float* dst = out + crow;
      for (int c = threadIdx.x; c < kCombos; c += blockDim.x) dst[c] = 0.f;
      __syncthreads();
      if (from)
        for (int h = threadIdx.x; h < sp.H[p]; h += blockDim.x)
          dst[combo_index(cards[2 * h], cards[2 * h + 1])] = from[h];
      __syncthreads();
    }
  }
}

cudaError_t launch_spot_combo(const SpotDev* spots, int n, int which, const float* in, float* out,
                              cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_spot_combo<<<n, 256, 0, s>>>(spots, which, in, out);
  return cudaGetLastError();
}

// Input rows of the boundary network, one block per item: bound by the write
// of the rows.  A thread owns one 16-byte vector of the row (4 f32 or 8 bf16
// values) for all 48 rivers and both players: it keeps the vector's reach
// values converted and their hands' cards in registers, and per river only
// clears the hands holding the river card and stores the vector twice.
// Choosing each value of each row by its segment, 733 items took 202 us for
// 383 MB of bf16 rows instead of 91.  The vectors that reach into the 68
// board, rank, pot, stack and player columns are made value by value, their
// rows spread over the block.
constexpr int kEncodeThreads = 352;
template <bool BF16>
__global__ void __launch_bounds__(kEncodeThreads) k_boundary_encode(const __grid_constant__ ItemMeta meta,
                                                                    const float* __restrict__ reach,
                                                                    void* __restrict__ out, bool whole) {
  constexpr int E = BF16 ? 8 : 4;  // values per vector
  constexpr int kVec = kBoundaryInput / E, kPlain = 2 * kCombos / E;
  const int item = blockIdx.x;
  __shared__ uint8_t s_river[kRivers];
  const uint8_t* bd = meta.board[item];
  for (int c = threadIdx.x; c < 52; c += blockDim.x) {
    const int k = river_pos(bd, c);
    if (k < kRivers) s_river[k] = (uint8_t)c;
  }
  const uint64_t bmask = (1ull << bd[0]) | (1ull << bd[1]) | (1ull << bd[2]) | (1ull << bd[3]);
  const float* rr = reach + (size_t)item * 2 * kCombos;
  // boundary_evaluator.rs:35-36, :54-56 in f32
  const float pot = meta.a[item], stack = meta.b[item];
  const float total = __fadd_rn(pot, stack);
  const float norm = total > 0.f ? total : 1.f;
  const float fpot = __fdiv_rn(pot, norm), fstack = __fdiv_rn(stack, norm);
  const unsigned ranks4 = (1u << (bd[0] >> 2)) | (1u << (bd[1] >> 2)) | (1u << (bd[2] >> 2)) | (1u << (bd[3] >> 2));
  uint4* o0 = reinterpret_cast<uint4*>(out) + (size_t)item * 2 * kRivers * kVec;
  uint4* o1 = o0 + (size_t)kRivers * kVec;
  auto bits = [](float x) {
    return BF16 ? (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(x)) : __float_as_uint(x);
  };
  auto put = [&](uint4* at, uint4 w) {
    if (!BF16 || whole) {
      *at = w;
    } else {  // bf16 rows aligned to 8 bytes only
      reinterpret_cast<uint2*>(at)[0] = make_uint2(w.x, w.y);
      reinterpret_cast<uint2*>(at)[1] = make_uint2(w.z, w.w);
    }
  };
  auto pack = [](const uint32_t (&x)[E]) {
    return BF16 ? make_uint4(x[0] | x[1] << 16, x[2 % E] | x[3 % E] << 16, x[4 % E] | x[5 % E] << 16,
                             x[6 % E] | x[7 % E] << 16)
                : make_uint4(x[0], x[1], x[2], x[3]);
  };
  __syncthreads();
  // the vectors that hold board, rank, pot, stack and player columns
  constexpr int kTail = kVec - kPlain;
  for (int i = threadIdx.x; i < 2 * kRivers * kTail; i += blockDim.x) {
    const int ri = i / kTail, q = kPlain + i - ri * kTail;
    const int player = ri >= kRivers, river = s_river[player ? ri - kRivers : ri];
    const uint64_t b5 = bmask | (1ull << river);
    const unsigned ranks = ranks4 | (1u << (river >> 2));
    uint32_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int f = E * q + e;
      float y;
      if (f < 2 * kCombos) {
        int a, b;
        combo_cards(f - kCombos, a, b);
        y = a == river || b == river ? 0.f : rr[f];
      } else if (f < 2 * kCombos + 52) {
        y = (b5 >> (f - 2 * kCombos) & 1) ? 1.f : 0.f;
      } else if (f < 2 * kCombos + 65) {
        y = (ranks >> (f - 2 * kCombos - 52) & 1) ? 1.f : 0.f;
      } else {
        y = f == kBoundaryInput - 3 ? fpot : f == kBoundaryInput - 2 ? fstack : (float)player;
      }
      x[e] = bits(y);
    }
    put(o0 + (size_t)ri * kVec + q, pack(x));  // the second player's rows follow the first's
  }
  for (int q = threadIdx.x; q < kPlain; q += blockDim.x) {
    uint32_t v[E];
    int c1[E], c2[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int f = E * q + e;
      v[e] = bits(rr[f]);
      combo_cards(f < kCombos ? f : f - kCombos, c1[e], c2[e]);
    }
#pragma unroll 4
    for (int ri = 0; ri < kRivers; ++ri) {
      const int river = s_river[ri];
      uint32_t x[E];
#pragma unroll
      for (int e = 0; e < E; ++e) x[e] = c1[e] == river || c2[e] == river ? 0u : v[e];
      const uint4 w = pack(x);
      put(o0 + (size_t)ri * kVec + q, w);
      put(o1 + (size_t)ri * kVec + q, w);
    }
  }
}

cudaError_t launch_boundary_encode(int n, const ItemMeta& meta, const float* reach, void* out, int bf16,
                                   cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (bf16)
    k_boundary_encode<true><<<n, kEncodeThreads, 0, s>>>(meta, reach, out, ((uintptr_t)out & 15) == 0);
  else
    k_boundary_encode<false><<<n, kEncodeThreads, 0, s>>>(meta, reach, out, true);
  return cudaGetLastError();
}

// Training records (cfvnet datagen/storage.rs:5-57), one block per (spot,
// player), packed byte by byte (the format is unaligned):
//   [board_size u8][board][pot f32][stack f32][player u8][game_value f32]
//   [oop_range f32 x1326][ip_range f32 x1326][cfvs f32 x1326][valid_mask u8 x1326]
// with the values of the GPU river datagen (datagen/domain/pipeline.rs:353-411):
// cfvs[c] = (f64(f32(rootcfv[h] * num_combinations)) - pot/2) / (pot/2) for the
// hands of the player's list, 0 elsewhere; valid_mask marks the hands of
// either player's list (one mask for both records);
// game_value = sum over combos of range * cfv, in f32, in combo order.
__device__ __forceinline__ void put_bytes(uint8_t* dst, const void* src, int n) {
  const uint8_t* s = static_cast<const uint8_t*>(src);
  for (int i = 0; i < n; ++i) dst[i] = s[i];
}

__global__ void k_pack_records(const SpotDev* __restrict__ spots, const float* __restrict__ ranges,
                               const RecordMeta* __restrict__ meta, uint8_t* __restrict__ out) {
  const int spot = blockIdx.x >> 1, player = blockIdx.x & 1;
  const SpotDev& sp = spots[spot];
  const RecordMeta m = meta[spot];
  const int bs = m.board_size;
  const size_t rsize = 1 + bs + 4 + 4 + 1 + 4 + 3 * 4 * kCombos + kCombos;
  uint8_t* rec = out + (size_t)blockIdx.x * rsize;
  __shared__ float s_cfv[kCombos];
  __shared__ uint8_t s_valid[kCombos];
  for (int c = threadIdx.x; c < kCombos; c += blockDim.x) {
    s_cfv[c] = 0.f;
    s_valid[c] = 0;
  }
  __syncthreads();
  const double half = 0.5 * (double)m.pot;
  const double norm = half > 0.0 ? half : 1.0;
  const float comb = (float)sp.num_combinations;
  const uint8_t* cards = sp.cards[player];
  for (int h = threadIdx.x; h < sp.H[player]; h += blockDim.x) {
    const int c = combo_index(cards[2 * h], cards[2 * h + 1]);
    const float ev = __fmul_rn(sp.root_out[player][h], comb);
    s_cfv[c] = (float)(((double)ev - half) / norm);
  }
  // one mask for both records: the hands of either player (pipeline.rs:366-377)
  for (int q = 0; q < 2; ++q)
    for (int h = threadIdx.x; h < sp.H[q]; h += blockDim.x)
      s_valid[combo_index(sp.cards[q][2 * h], sp.cards[q][2 * h + 1])] = 1;
  __syncthreads();
  const float* rg = ranges + (size_t)spot * 2 * kCombos;
  uint8_t* body = rec + 1 + bs + 13;
  for (int i = threadIdx.x; i < 3 * kCombos; i += blockDim.x) {
    const float v = i < 2 * kCombos ? rg[i] : s_cfv[i - 2 * kCombos];
    put_bytes(body + 4 * i, &v, 4);
  }
  for (int c = threadIdx.x; c < kCombos; c += blockDim.x) body[12 * kCombos + c] = s_valid[c];
  if (threadIdx.x == 0) {
    const float* own = rg + (size_t)player * kCombos;
    float gv = 0.f;
    for (int c = 0; c < kCombos; ++c) gv = __fadd_rn(gv, __fmul_rn(own[c], s_cfv[c]));
    rec[0] = (uint8_t)bs;
    for (int k = 0; k < bs; ++k) rec[1 + k] = m.board[k];
    put_bytes(rec + 1 + bs, &m.pot, 4);
    put_bytes(rec + 5 + bs, &m.stack, 4);
    rec[9 + bs] = (uint8_t)player;
    put_bytes(rec + 10 + bs, &gv, 4);
  }
}

cudaError_t launch_pack_records(const SpotDev* spots, int n, const float* ranges, const RecordMeta* meta,
                                uint8_t* out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_pack_records<<<2 * n, 256, 0, s>>>(spots, ranges, meta, out);
  return cudaGetLastError();
}

cudaError_t launch_boundary_river_reduce(int n, const ItemMeta& meta, const void* net, int net_bf16,
                                         const float* reach, const int32_t* hands, int H, float* out,
                                         cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  if (net_bf16)
    k_boundary_river_reduce<__nv_bfloat16><<<2 * n, kReduceThreads, 0, s>>>(meta, static_cast<const __nv_bfloat16*>(net), reach,
                                                                 hands, H, out, ((uintptr_t)net & 3) == 0);
  else
    k_boundary_river_reduce<float><<<2 * n, kReduceThreads, 0, s>>>(meta, static_cast<const float*>(net), reach, hands, H, out,
                                                         ((uintptr_t)net & 7) == 0);
  return cudaGetLastError();
}

cudaError_t launch_river_average_grad(int n, const ItemMeta& meta, const float* reach, const float* g, float* gy,
                                      cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_river_average_grad<<<2 * n, kReduceThreads, kGradPad, s>>>(meta, reach, g, gy, ((uintptr_t)gy & 7) == 0);
  return cudaGetLastError();
}

// First layer of a boundary network (a Linear over the 2720 input values)
// for every input row of boundary_encode, without writing the rows: for item
// i, player p and river card r,
//   W x = W_reach [oop|ip] - sum over combos holding r of W_reach[., c] reach[c]
//         + board / rank one-hot columns + pot, stack, player columns (+ bias)
// base[i] = W_reach [oop|ip] and percard[i][k] (the sum over the combos
// holding card k) come from the caller's GEMMs; without base it is half the
// sum of percard over the 52 cards (every combo holds two), in f64.  One block
// per item, V adjacent columns per thread for all 48 rivers and both players,
// the river-independent part in registers: bound by the read of percard and
// the write of the rows.  With an index division per element and one column at
// a time, 1024 items of 500 columns took 127 us; 57 us now, base included.
// out [n][2][48][h].
template <int V>
struct Cols {
  float x[V];
};
template <int V>
__device__ __forceinline__ Cols<V> ld_cols(const float* p) {
  Cols<V> c;
  if (V == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    c.x[0] = v.x;
    c.x[V - 1] = v.y;
  } else {
    c.x[0] = *p;
  }
  return c;
}
template <bool BF16, int V>
__device__ __forceinline__ void st_cols(void* out, size_t at, const float (&v)[V]) {
  if (BF16) {
    __nv_bfloat16* o = static_cast<__nv_bfloat16*>(out) + at;
    if (V == 2)
      *reinterpret_cast<__nv_bfloat162*>(o) = __floats2bfloat162_rn(v[0], v[V - 1]);
    else
      *o = __float2bfloat16_rn(v[0]);
  } else {
    float* o = static_cast<float*>(out) + at;
    if (V == 2)
      *reinterpret_cast<float2*>(o) = make_float2(v[0], v[V - 1]);
    else
      *o = v[0];
  }
}
template <bool BF16, int V>
__global__ void __launch_bounds__(256) k_boundary_first_layer(const __grid_constant__ ItemMeta meta,
                                                              const float* __restrict__ base,
                                                              const float* __restrict__ percard,
                                                              const float* __restrict__ wcols,
                                                              const float* __restrict__ bias, int h,
                                                              void* __restrict__ out) {
  __shared__ uint8_t s_river[kRivers];
  const int item = blockIdx.x;
  const uint8_t* bd = meta.board[item];
  const unsigned ranks4 = (1u << (bd[0] >> 2)) | (1u << (bd[1] >> 2)) | (1u << (bd[2] >> 2)) | (1u << (bd[3] >> 2));
  for (int c = threadIdx.x; c < 52; c += blockDim.x) {
    const int k = river_pos(bd, c);
    if (k < kRivers) s_river[k] = (uint8_t)c;
  }
  __syncthreads();
  const float pot = meta.a[item], stack = meta.b[item];
  const float total = __fadd_rn(pot, stack);
  const float norm = total > 0.f ? total : 1.f;
  const float fpot = __fdiv_rn(pot, norm), fstack = __fdiv_rn(stack, norm);
  const float* pc = percard + (size_t)item * 52 * h;
  const size_t o0 = (size_t)item * 2 * kRivers * h, o1 = o0 + (size_t)kRivers * h;
  for (int j = V * threadIdx.x; j < h; j += V * blockDim.x) {
    Cols<V> c;
    if (base) {
      c = ld_cols<V>(base + (size_t)item * h + j);
    } else {
      double t[V] = {};
#pragma unroll 13
      for (int k = 0; k < 52; ++k) {
        const Cols<V> x = ld_cols<V>(pc + (size_t)k * h + j);
#pragma unroll
        for (int e = 0; e < V; ++e) t[e] += (double)x.x[e];
      }
#pragma unroll
      for (int e = 0; e < V; ++e) c.x[e] = (float)(0.5 * t[e]);
    }
    auto col = [&](int k) { return ld_cols<V>(wcols + (size_t)k * h + j); };
    auto plus = [&](const Cols<V>& x) {
#pragma unroll
      for (int e = 0; e < V; ++e) c.x[e] += x.x[e];
    };
#pragma unroll
    for (int k = 0; k < 4; ++k) plus(col(bd[k]));
    for (int q = 0; q < 13; ++q)
      if (ranks4 >> q & 1) plus(col(52 + q));
    const Cols<V> wpot = col(65), wstack = col(66), wplayer = col(67);
#pragma unroll
    for (int e = 0; e < V; ++e)
      c.x[e] = c.x[e] + fpot * wpot.x[e] + fstack * wstack.x[e] + (bias ? bias[j + e] : 0.f);
#pragma unroll 4
    for (int ri = 0; ri < kRivers; ++ri) {
      const int r = s_river[ri];
      const Cols<V> x = ld_cols<V>(pc + (size_t)r * h + j), w = col(r), k = col(52 + (r >> 2));
      const bool fresh = !(ranks4 >> (r >> 2) & 1);  // the river brings a rank the board lacks
      float v[V], v1[V];
#pragma unroll
      for (int e = 0; e < V; ++e) {
        v[e] = c.x[e] - x.x[e] + w.x[e];
        if (fresh) v[e] += k.x[e];
        v1[e] = v[e] + wplayer.x[e];
      }
      st_cols<BF16, V>(out, o0 + (size_t)ri * h + j, v);
      st_cols<BF16, V>(out, o1 + (size_t)ri * h + j, v1);
    }
  }
}

cudaError_t launch_boundary_first_layer(int n, const ItemMeta& meta, const float* base, const float* percard,
                                        const float* wcols, const float* bias, int h, void* out, int bf16,
                                        cudaStream_t s) {
  if (n <= 0 || h <= 0) return cudaSuccess;
  if (h > kMaxFirstLayerWidth) return cudaErrorInvalidValue;
  // column pairs where every row starts on one
  const uintptr_t f32 = (uintptr_t)base | (uintptr_t)percard | (uintptr_t)wcols | (bf16 ? 0 : (uintptr_t)out);
  const bool two = h % 2 == 0 && (f32 & 7) == 0 && ((uintptr_t)out & 3) == 0;
  auto k = bf16 ? (two ? k_boundary_first_layer<true, 2> : k_boundary_first_layer<true, 1>)
                : (two ? k_boundary_first_layer<false, 2> : k_boundary_first_layer<false, 1>);
  k<<<n, 256, 0, s>>>(meta, base, percard, wcols, bias, h, out);
  return cudaGetLastError();
}

}  // namespace ps
