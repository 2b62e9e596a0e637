// Situation sampling on the device: boards, pot / stack and two R(S,p) ranges
// per situation (cfvnet datagen/sampler.rs:30-60, :142-205 and
// datagen/range_gen.rs:18-167), one block per situation.
//
// Random numbers: a counter-based SplitMix64 stream (Vigna's published
// generator), key(i) = mix(seed + (i + 1) * G), draw(i, c) = mix(key(i) +
// (c + 1) * G), so that every draw of every situation is addressable and the
// R(S,p) recursion runs in parallel.  The reference draws from rand's ChaCha8
// in recursion order; the distribution is the same, the stream is not.
// Counters: board cards from 0, pot / stack from 1 << 16, range r's split at
// the node covering sorted positions [lo, hi) at ((r + 1) << 32) | lo << 12 | hi.
#include <cuda_runtime.h>
#include <stdint.h>

#include "ps_launch.hpp"

namespace ps {

namespace {

constexpr int kCombosS = 1326;
constexpr uint64_t kGolden = 0x9E3779B97F4A7C15ull;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ uint64_t draw(uint64_t key, uint64_t ctr) { return mix64(key + (ctr + 1) * kGolden); }

// uniform integer in [0, n) from the top 32 bits (multiply-shift)
__device__ __forceinline__ int draw_int(uint64_t key, uint64_t ctr, uint32_t n) {
  return (int)(((draw(key, ctr) >> 32) * (uint64_t)n) >> 32);
}

// uniform double in [0, 1) with 53 random bits
__device__ __forceinline__ double draw_unit(uint64_t key, uint64_t ctr) {
  return (double)(draw(key, ctr) >> 11) * 0x1.0p-53;
}

__device__ __forceinline__ int top_bits(int x, int n) {  // the n highest set bits of x
  int r = 0;
  for (int k = 0; k < n && x; ++k) {
    const int b = 1 << (31 - __clz(x));
    r |= b;
    x ^= b;
  }
  return r;
}

__device__ __forceinline__ int straight_top(int ranks) {  // top-rank bit of a 5-rank run (wheel: the five)
  const int run = ranks & (ranks << 1) & (ranks << 2) & (ranks << 3) & (ranks << 4);
  if (run) return top_bits(run, 1);
  return (ranks & 0x100F) == 0x100F ? 1 << 3 : 0;
}

// Cards by count: the rank sets with at least one, two, three and four cards,
// and the ranks held in each suit (13 bits each, suit s from bit 16 s).
struct Counts {
  int c1, c2, c3, c4;
  uint64_t suits;
  __device__ __forceinline__ Counts() : c1(0), c2(0), c3(0), c4(0), suits(0) {}
  __device__ __forceinline__ void add(int card) {
    const int b = 1 << (card >> 2);
    c4 |= c3 & b;
    c3 |= c2 & b;
    c2 |= c1 & b;
    c1 |= b;
    suits |= (uint64_t)b << (16 * (card & 3));
  }
};

__device__ __forceinline__ int drop2(int x) {  // x without its two lowest bits
  x &= x - 1;
  return x & (x - 1);
}

// 7-card value with the encoding of range_gen.rs:184-268: category << 26,
// then the ranks that decide within the category (primary set << 13 | kickers).
// fs: the suit with at least five of the cards, or -1.
__device__ __forceinline__ int value7(const Counts& k, int fs) {
  if (fs >= 0) {
    int f = (int)(k.suits >> (16 * fs)) & 0x1FFF;
    const int sf = straight_top(f);
    if (sf) return (8 << 26) | sf;
    const int n = __popc(f);  // 5, 6 or 7
    if (n > 5) f &= f - 1;
    if (n > 6) f &= f - 1;
    return (5 << 26) | f;
  }
  const int b1 = k.c1 & ~k.c2, b2 = k.c2 & ~k.c3, b3 = k.c3 & ~k.c4;
  if (k.c4) return (7 << 26) | (k.c4 << 13) | top_bits(k.c1 ^ k.c4, 1);
  if (b3) {
    if (b3 & (b3 - 1)) {  // two trips
      const int t = top_bits(b3, 1);
      return (6 << 26) | (t << 13) | (b3 ^ t);
    }
    if (b2) return (6 << 26) | (b3 << 13) | top_bits(b2, 1);
  }
  const int st = straight_top(k.c1);
  if (st) return (4 << 26) | st;
  if (b3) return (3 << 26) | (b3 << 13) | drop2(b1);  // four single ranks
  if (b2 & (b2 - 1)) {
    const int two = __popc(b2) > 2 ? b2 & (b2 - 1) : b2;
    return (2 << 26) | (two << 13) | top_bits(k.c1 ^ two, 1);
  }
  if (b2) return (1 << 26) | (b2 << 13) | drop2(b1);  // five single ranks
  return drop2(k.c1);                                 // seven
}

__device__ __forceinline__ void combo_pair(int idx, int& c1, int& c2) {
  // first combo of card a: a (103 - a) / 2
  int a = (int)((103.f - sqrtf((float)(10609 - 8 * idx))) * 0.5f);
  if (a * (103 - a) / 2 > idx) --a;
  if ((a + 1) * (102 - a) / 2 <= idx) ++a;
  c1 = a;
  c2 = idx - a * (101 - a) / 2 + 1;
}

// Ascending sort of kSort keys in shared memory by kThreads threads (bitonic).
// A thread keeps kPer consecutive keys: strides below kPer are exchanged in
// registers, below 32 kPer between the lanes of a warp, and only the six
// strides above that (of 66) through shared memory.
constexpr int kThreads = 256, kSort = 2048, kPer = kSort / kThreads;
__device__ __forceinline__ void order(uint64_t& x, uint64_t& y, bool up) {
  const bool sw = (x > y) == up;
  const uint64_t t = x;
  x = sw ? y : x;
  y = sw ? t : y;
}
__device__ void block_sort(uint64_t* keys) {
  const int t = threadIdx.x, base = t * kPer;
  uint64_t v[kPer];
#pragma unroll
  for (int e = 0; e < kPer; ++e) v[e] = keys[base + e];
#pragma unroll
  for (int e = 0; e < kPer; e += 2) order(v[e], v[e + 1], (e & 2) == 0);
#pragma unroll
  for (int e = 0; e < kPer; e += 4) {
    const bool up = ((base + e) & 4) == 0;
    order(v[e], v[e + 2], up);
    order(v[e + 1], v[e + 3], up);
    order(v[e], v[e + 1], up);
    order(v[e + 2], v[e + 3], up);
  }
#pragma unroll 1
  for (int k = kPer; k <= kSort; k <<= 1) {
    const bool up = (base & k) == 0;
#pragma unroll 1
    for (int j = k >> 1; j >= kPer; j >>= 1) {
      const bool keep_min = ((base & j) == 0) == up;
      if (j >= 32 * kPer) {
        __syncthreads();  // every thread has read the keys of the stride before
#pragma unroll
        for (int e = 0; e < kPer; ++e) keys[e * kThreads + t] = v[e];
        __syncthreads();
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
          const uint64_t o = keys[e * kThreads + (t ^ (j / kPer))];
          v[e] = (o < v[e]) == keep_min ? o : v[e];
        }
      } else {
#pragma unroll
        for (int e = 0; e < kPer; ++e) {
          const uint64_t o = __shfl_xor_sync(0xffffffffu, v[e], j / kPer);
          v[e] = (o < v[e]) == keep_min ? o : v[e];
        }
      }
    }
#pragma unroll
    for (int j = kPer / 2; j > 0; j >>= 1)
#pragma unroll
      for (int e = 0; e < kPer; ++e)
        if (!(e & j)) order(v[e], v[e + j], up);
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kPer; ++e) keys[base + e] = v[e];
  __syncthreads();
}

}  // namespace

// One block per situation.  Bound by integer issue: 46 7-card values per combo
// on a turn board, then the strength order.  The values add one river card to
// the rank and suit sets of the combo's six cards (about 45 instructions), and
// the order is a sort of (value, combo) keys.  Counting each card's ranks anew
// per value and ranking by an all-pairs count, 1500 turn situations took 4.28
// ms of kernel time instead of 0.54.
__global__ void __launch_bounds__(kThreads) k_sample_situations(SamplerParams P, uint8_t* __restrict__ boards, int32_t* __restrict__ pots,
                                    int32_t* __restrict__ stacks, float* __restrict__ ranges, int* err) {
  const int64_t idx = P.first + blockIdx.x;
  const uint64_t key = mix64(P.seed + (uint64_t)(idx + 1) * kGolden);
  __shared__ uint64_t s_key[kSort];    // (value << 11 | combo) in order, past the valid ones all ones
  __shared__ uint16_t s_pos[kCombosS];  // position in the order, kCombosS if blocked
  __shared__ int s_board[5], s_pot, s_stack, s_nvalid, s_bad;
  const int bs = P.board_size;
  if (threadIdx.x == 0) {
    // sampler.rs:142-160: cards by rejection until bs distinct ones
    uint64_t used = 0, ctr = 0;
    int bad = 0;
    for (int k = 0; k < bs; ++k) {
      int c;
      do {
        c = draw_int(key, ctr++, 52);
      } while ((used >> c & 1) && ctr < 4096);
      if (used >> c & 1) bad = 1;
      used |= 1ull << c;
      s_board[k] = c;
    }
    for (int k = bs; k < 5; ++k) s_board[k] = 0;
    // pot and stack (sampler.rs:42-51, :165-205)
    uint64_t pc = 1u << 16;
    int pot = 0, stack = 0;
    if (P.nspr == 0) {
      const int iv = draw_int(key, pc++, (uint32_t)P.npot);
      const int lo = P.pot[iv][0], hi = P.pot[iv][1];
      pot = lo + draw_int(key, pc++, (uint32_t)(hi - lo));
      const int max_stack = P.initial_stack - pot / 2;
      stack = max_stack < 5 ? 5 : 5 + draw_int(key, pc++, (uint32_t)(max_stack - 5 + 1));
    } else {
      const double sf = (double)P.initial_stack;
      bool found = false;
      for (int attempt = 0; attempt < 10000 && !found; ++attempt) {
        const int si = draw_int(key, pc++, (uint32_t)P.nspr);
        const double slo = P.spr[si][0], shi = P.spr[si][1];
        const double spr = slo + draw_unit(key, pc++) * (shi - slo);
        const double pmin = spr > 0.0 ? ceil(5.0 / spr) : ceil(2.0 * (sf - 5.0));
        const double pmax = sf / (spr + 0.5);
        const int flo = (int)fmin(fmax(pmin, 1.0), 1.0e9), fhi = (int)pmax;
        if (flo > fhi) continue;
        int blo[kMaxSamplerIntervals], bhi[kMaxSamplerIntervals], nb = 0;
        for (int k = 0; k < P.npot; ++k) {
          const int lo = max(P.pot[k][0], flo), hi = min(P.pot[k][1], fhi + 1);
          if (lo < hi) {
            blo[nb] = lo;
            bhi[nb] = hi;
            ++nb;
          }
        }
        if (nb == 0) continue;
        const int b = draw_int(key, pc++, (uint32_t)nb);
        const int p = blo[b] + draw_int(key, pc++, (uint32_t)(bhi[b] - blo[b]));
        const int max_stack = P.initial_stack - p / 2;
        if (max_stack < 5) continue;
        const int s = min(max((int)fmin(round(spr * (double)p), 2.0e9), 5), max_stack);
        const double actual = (double)s / (double)p;
        if (actual >= slo && actual < shi) {
          pot = p;
          stack = s;
          found = true;
        }
      }
      if (!found) bad = 1;
    }
    s_pot = pot;
    s_stack = stack;
    s_bad = bad;
  }
  __syncthreads();
  if (s_bad) {
    if (threadIdx.x == 0) atomicExch(err, 1);
    return;
  }
  uint64_t bmask = 0;
  for (int k = 0; k < bs; ++k) bmask |= 1ull << s_board[k];
  // hand strengths (range_gen.rs:18-56): the 7-card value on a 5-card board,
  // its average over the 46 river cards on a 4-card board.  The sum over the
  // rivers stands for the average: every combo has 46, and distinct sums below
  // 2^36 have distinct f64 averages.
  if (threadIdx.x == 0) s_nvalid = 0;
  for (int i = threadIdx.x; i < kSort; i += blockDim.x) {
    uint64_t key = ~0ull;
    if (i < kCombosS) {
      int c1, c2;
      combo_pair(i, c1, c2);
      const uint64_t hm = (1ull << c1) | (1ull << c2);
      s_pos[i] = kCombosS;
      if (!(hm & bmask)) {
        Counts base;
        for (int k = 0; k < bs; ++k) base.add(s_board[k]);
        base.add(c1);
        base.add(c2);
        int fs = -1, four = -1;  // the suit with five or more, and one with exactly four
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int n = __popc((int)(base.suits >> (16 * u)) & 0x1FFF);
          if (n >= 5) fs = u;
          if (n == 4) four = u;
        }
        uint64_t sum = 0;
        if (bs == 5) {
          sum = (uint64_t)value7(base, fs);
        } else {
          for (int r = 0; r < 52; ++r) {
            if ((bmask | hm) >> r & 1) continue;
            Counts c = base;
            c.add(r);
            sum += (uint64_t)value7(c, fs >= 0 ? fs : (r & 3) == four ? four : -1);
          }
        }
        key = sum << 11 | (uint64_t)i;
      }
    }
    s_key[i] = key;
  }
  __syncthreads();
  // the stable ascending order (ties by combo index)
  block_sort(s_key);
  int nv = 0;
  for (int i = threadIdx.x; i < kCombosS; i += blockDim.x)
    if (s_key[i] != ~0ull) {
      s_pos[(int)(s_key[i] & 2047)] = (uint16_t)i;
      ++nv;
    }
  nv = __reduce_add_sync(0xffffffffu, nv);
  if ((threadIdx.x & 31) == 0) atomicAdd(&s_nvalid, nv);
  __syncthreads();
  const int n = s_nvalid;
  // R(S,p) (range_gen.rs:120-167): each node of the recursion over sorted
  // positions [lo, hi) splits its mass p at a uniform point; the larger part
  // goes to the stronger half [lo + len/2, hi).  A combo's mass is the product
  // along its root-to-leaf path, in the recursion's f64 arithmetic.
  const size_t out0 = (size_t)blockIdx.x * 2 * kCombosS;
  for (int r = 0; r < 2; ++r)
    for (int c = threadIdx.x; c < kCombosS; c += blockDim.x) {
      float m = 0.f;
      const int k = s_pos[c];
      if (k < n) {
        int lo = 0, hi = n;
        double p = 1.0;
        while (hi - lo > 1 && p > 0.0) {
          const double u = draw_unit(key, ((uint64_t)(r + 1) << 32) | ((uint64_t)lo << 12) | (uint64_t)hi);
          const double d = u * p, rem = p - d;
          const int mid = lo + (hi - lo) / 2;
          if (k >= mid) {
            p = fmax(d, rem);
            lo = mid;
          } else {
            p = fmin(d, rem);
            hi = mid;
          }
        }
        m = p > 0.0 ? (float)p : 0.f;
      }
      ranges[out0 + (size_t)r * kCombosS + c] = m;
    }
  if (threadIdx.x == 0) {
    for (int k = 0; k < 5; ++k) boards[(size_t)blockIdx.x * 5 + k] = (uint8_t)s_board[k];
    pots[blockIdx.x] = s_pot;
    stacks[blockIdx.x] = s_stack;
  }
}

cudaError_t launch_sample_situations(const SamplerParams& P, int n, uint8_t* boards, int32_t* pots, int32_t* stacks,
                                     float* ranges, int* err, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_sample_situations<<<n, kThreads, 0, s>>>(P, boards, pots, stacks, ranges, err);
  return cudaGetLastError();
}

}  // namespace ps
