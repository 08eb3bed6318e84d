// Contractions on small output tiles: the plain kernel of float64 /
// complex128, and of float32 / complex64 products too small for simt.cu's.
//
// FP64: GB300 issues two FP64 FMAs per clock and SM (1.25 TFLOP/s nominal),
// so a warp's FMA occupies its scheduler for 64 clocks and everything else of
// the loop (shared-memory reads, copies, address arithmetic) hides behind it
// even with one output per thread.  What bounds a product is how evenly its
// FMAs spread over the 152 SMs and how many of them are padding; a 128 x 64
// tile of 256 threads (simt.cu's shape) takes an SM 16 us per 8 k of float64,
// whatever part of it lies inside the output.
// FP32: a small product is a chain of latencies (offsets, operands, sums,
// C), to which a 64 x 128 tile adds the FMAs of its padding.
//   16 x 16 outputs: two per thread;
//   8 x 8 outputs:   one per thread, the two halves of the block taking
//                    alternate k and added in a fixed order at the end, for
//                    outputs with too few tiles to occupy every SM.
// Steps past K are not computed, and a warp whose outputs all lie past the edge
// computes nothing.
// Measured (GB300): complex128 1024^3 8.23 -> 6.95 ms (1.24 TFLOP/s, 98% of
// the two-FMA rate), float64 9216 x 96 x 96 281 -> 190 us a call.
//
// Tiles are gathered through the scatter vectors as in simt.cu (the plain
// form; replaces the reference's include/t1m/t1m.h:432-557 in FP64), each
// operand's unit-stride direction on consecutive threads, through a
// cp.async ring (ring_stages).  Consecutive threads write along C's unit stride.
#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "internal.h"
#include "simt_common.h"
#include "t1m_capi.h"

namespace t1m {
namespace gb300 {
namespace {

constexpr int kThreads = 128;
constexpr int kBK = 16;      // k per stage
// Stages of the copy ring: a small block's time is the latency of its
// copies, so as many as 48 KB of static shared memory hold.
template <class T>
constexpr int ring_stages() { return sizeof(T) == 16 ? 3 : 5; }

__device__ __forceinline__ float flip(float v, uint64_t) { return v; }
__device__ __forceinline__ float2 flip(float2 v, uint64_t sign) {
  v.y = __uint_as_float(__float_as_uint(v.y) ^ static_cast<uint32_t>(sign >> 32));
  return v;
}
// Conjugation by the sign bit: a floating negation of a value that is not an
// FMA operand would go through the FP64 pipe (measured: half as many FP64
// instructions again, complex128 1024^3 10.5 ms against 7.1).
__device__ __forceinline__ double flip(double v, uint64_t) { return v; }
__device__ __forceinline__ double2 flip(double2 v, uint64_t sign) {
  v.y = __longlong_as_double(__double_as_longlong(v.y) ^ static_cast<long long>(sign));
  return v;
}

// A sum of chains: FP32 values with the rounding errors of their additions
// (Knuth's two-sum), so joining four short chains rounds once.  Plain
// additions made outputs of few terms worse than one chain (float32, K = 5,
// entries uniform in [-1, 1]: 5.0e-8 against 4.4e-8).  FP64 joins by plain
// additions: two-sum would take the FP64 pipe longer than a small product.
template <class T>
struct ChainSum {
  T v;
  __device__ __forceinline__ void start(T x) { v = x; }
  __device__ __forceinline__ void join(const ChainSum& o) { v = add(v, o.v); }
  __device__ __forceinline__ T value() const { return v; }
};
__device__ __forceinline__ void two_sum(float& s, float& e, float x, float xe) {
  const float t = __fadd_rn(s, x), u = __fsub_rn(t, s);
  e = __fadd_rn(__fadd_rn(e, xe),
                __fadd_rn(__fsub_rn(s, __fsub_rn(t, u)), __fsub_rn(x, u)));
  s = t;
}
// An infinite, NaN or overflowing sum has no error term.
__device__ __forceinline__ float two_value(float s, float e) {
  return isfinite(e) ? __fadd_rn(s, e) : s;
}
template <>
struct ChainSum<float> {
  float v, e;
  __device__ __forceinline__ void start(float x) { v = x; e = 0.f; }
  __device__ __forceinline__ void join(const ChainSum& o) { two_sum(v, e, o.v, o.e); }
  __device__ __forceinline__ float value() const { return two_value(v, e); }
};
template <>
struct ChainSum<float2> {
  float2 v, e;
  __device__ __forceinline__ void start(float2 x) { v = x; e = make_float2(0.f, 0.f); }
  __device__ __forceinline__ void join(const ChainSum& o) {
    two_sum(v.x, e.x, o.v.x, o.e.x);
    two_sum(v.y, e.y, o.v.y, o.e.y);
  }
  __device__ __forceinline__ float2 value() const {
    return make_float2(two_value(v.x, e.x), two_value(v.y, e.y));
  }
};

// K offsets held in shared memory: looked up per stage, each stage waited for
// its offsets before its copies could start (a 16 x 16 x 512 block: 52 us).
constexpr int kOffsets = 512;

template <class T, int kTile>
struct SmallSmem {
  static constexpr int kPad = 32 / sizeof(T);
  static constexpr int kStages = ring_stages<T>();
  T a[kStages][kBK][kTile + kPad];
  T b[kStages][kBK][kTile + kPad];
  ChainSum<T> part[kTile == 8 ? 64 : 1];  // the second k slice's sums (8 x 8 form)
  int64_t row_a[kTile], col_b[kTile];
  int64_t ka[kOffsets], kb[kOffsets];  // K offsets, a ring of two halves
};

// One output tile over the K range of `split`.  kTile: 16 or 8 rows and
// columns.  kNFast: consecutive threads along n (C unit stride along its
// columns), else along m.
template <class T, int kTile, bool kNFast>
__device__ __forceinline__ void small_tile(const GemmArgs& args, int64_t tile, int64_t split,
                                          SmallSmem<T, kTile>& sm) {
  constexpr int kOut = kTile * kTile >= kThreads ? kTile * kTile / kThreads : 1;
  constexpr int kSlices = kThreads * kOut / (kTile * kTile);  // k slices of the block
  constexpr int kSlow = kTile / kOut;                           // step between a thread's outputs
  auto& As = sm.a;
  auto& Bs = sm.b;
  int64_t* const rowA = sm.row_a;
  int64_t* const colB = sm.col_b;

  const T* __restrict__ A = static_cast<const T*>(args.A);
  const T* __restrict__ B = static_cast<const T*>(args.B);
  const int64_t M = args.M, N = args.N;
  const int64_t tiles_m = (M + kTile - 1) / kTile, tiles_n = (N + kTile - 1) / kTile;
  const int64_t kb = split * args.k_per_split;
  const int64_t K = min(args.K, kb + args.k_per_split);
  T* __restrict__ C = static_cast<T*>(args.C) + split * args.c_split_stride;
  const uint64_t signA = args.flags & kFlagConjA ? uint64_t(1) << 63 : 0;
  const uint64_t signB = args.flags & kFlagConjB ? uint64_t(1) << 63 : 0;
  // Groups of 32 M-tiles sweep N, so blocks running together share operands.
  constexpr int64_t G = 32;
  const int64_t first_m = (tile / (G * tiles_n)) * G;
  const int64_t gsize = min(G, tiles_m - first_m);
  const int64_t r = tile % (G * tiles_n);
  const int64_t m0 = (first_m + r % gsize) * kTile, n0 = (r / gsize) * kTile;

  const int tid = threadIdx.x;
  if (tid < kTile) {
    rowA[tid] = m0 + tid < M ? offs(args.rsA, args.uA_m, m0 + tid) : 0;
  } else if (tid < 2 * kTile) {
    const int n = tid - kTile;
    colB[n] = n0 + n < N ? offs(args.csB, args.uB_n, n0 + n) : 0;
  }

  const bool a_kfast = args.uA_k == 1;
  const bool b_kfast = args.uB_k == 1 || args.uB_n != 1;
  constexpr int kPer = kTile * kBK / kThreads;
  static_assert(kPer * kThreads == kTile * kBK, "stage copies");
  constexpr int kStages = ring_stages<T>();
  // Offsets of k in [k0, k0 + n) into their places of the ring.
  auto look = [&](int64_t k0, int n) {
    for (int i = tid; i < n && k0 + i < K; i += kThreads) {
      const int at = static_cast<int>((k0 + i - kb) % kOffsets);
      sm.ka[at] = offs(args.csA, args.uA_k, k0 + i);
      sm.kb[at] = offs(args.rsB, args.uB_k, k0 + i);
    }
  };
  look(kb, kOffsets);
  __syncthreads();
  auto issue = [&](int64_t k0, int buf) {
    const int at = static_cast<int>((k0 - kb) % kOffsets);
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int idx = tid + p * kThreads;
      const int m = a_kfast ? idx / kBK : idx % kTile;
      const int k = a_kfast ? idx % kBK : idx / kTile;
      const bool in = m0 + m < M && k0 + k < K;
      cp_async_elem<sizeof(T)>(&As[buf][k][m], in ? A + rowA[m] + sm.ka[at + k] : A, in);
    }
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int idx = tid + p * kThreads;
      const int n = b_kfast ? idx / kBK : idx % kTile;
      const int k = b_kfast ? idx % kBK : idx / kTile;
      const bool in = n0 + n < N && k0 + k < K;
      cp_async_elem<sizeof(T)>(&Bs[buf][k][n], in ? B + sm.kb[at + k] + colB[n] : B, in);
    }
  };

  // Outputs of this thread: index `f` along the fast dimension, s + kSlow j
  // along the other.
  const int f = tid % kTile, s = (tid / kTile) % kSlow, slice = tid / (kTile * kSlow);
  const int64_t fast_n = (kNFast ? N - n0 : M - m0), slow_n = (kNFast ? M - m0 : N - n0);
  bool live[kOut];
#pragma unroll
  for (int j = 0; j < kOut; ++j) live[j] = f < fast_n && s + kSlow * j < slow_n;
  // Eight FMA chains per output (k modulo their number, over the slices),
  // joined at the end: shorter chains than one per K range round less, and an
  // unsplit K of 256 has chains of 32 terms, as short as the K ranges that
  // larger tiles split such products into (FP32 with four chains: 20 x 248
  // over 262 3.0e-7 off, 1.5e-7 as seven ranges).  Up to
  // kSerial terms stay in one chain: there the products rounded apart and the
  // sums that join them are more roundings than the chain's.
  constexpr int kAll = 8, kChains = kAll / kSlices;
  constexpr int kSerial = std::is_same_v<T, double>    ? 8
                          : std::is_same_v<T, double2> ? 3
                          : std::is_same_v<T, float>   ? 2
                                                       : 0;
  T part[kOut][kChains];
#pragma unroll
  for (int j = 0; j < kOut; ++j)
#pragma unroll
    for (int u = 0; u < kChains; ++u) part[j][u] = zero<T>();

  const int64_t ksteps = K > kb ? (K - kb + kBK - 1) / kBK : 0;
#pragma unroll
  for (int st = 0; st < kStages - 1; ++st) {
    if (st < ksteps) issue(kb + st * kBK, st);
    cp_async_commit_group();
  }
  for (int64_t st = 0; st < ksteps; ++st) {
    const int buf = static_cast<int>(st % kStages);
    cp_async_wait_group<kStages - 2>();
    __syncthreads();  // stage st has landed for every thread; stage st - 1 is consumed
    const int64_t nxt = st + kStages - 1;
    // The copies enter a new half of the offsets: the other one is refilled
    // (read again no earlier than 256 k later, stages of barriers away).
    if (nxt * kBK % (kOffsets / 2) == 0 && nxt > 0)
      look(kb + nxt * kBK + kOffsets / 2, kOffsets / 2);
    if (nxt < ksteps) issue(kb + nxt * kBK, static_cast<int>(nxt % kStages));
    cp_async_commit_group();
    const int kn = static_cast<int>(min(static_cast<int64_t>(kBK), K - kb - st * kBK));
    auto step = [&](int k, int u) {
      const T x = kNFast ? flip(Bs[buf][k][f], signB) : flip(As[buf][k][f], signA);
#pragma unroll
      for (int j = 0; j < kOut; ++j) {
        if (!live[j]) continue;
        const T y = kNFast ? flip(As[buf][k][s + kSlow * j], signA)
                           : flip(Bs[buf][k][s + kSlow * j], signB);
        if (kNFast) mac(part[j][u], y, x); else mac(part[j][u], x, y);
      }
    };
    if (kn == kBK) {
#pragma unroll
      for (int k = 0; k < kBK; k += kAll)
#pragma unroll
        for (int u = 0; u < kChains; ++u) step(k + u * kSlices + slice, u);
    } else if (K - kb <= kSerial) {
      if (slice == 0)
        for (int k = 0; k < kn; ++k) step(k, 0);
    } else {
      for (int k = 0; k < kn; k += kAll)
#pragma unroll
        for (int u = 0; u < kChains; ++u)
          if (k + u * kSlices + slice < kn) step(k + u * kSlices + slice, u);
    }
  }
  cp_async_wait_group<0>();

  ChainSum<T> acc[kOut];
#pragma unroll
  for (int j = 0; j < kOut; ++j) {
    ChainSum<T> sum[kChains];
#pragma unroll
    for (int u = 0; u < kChains; ++u) sum[u].start(part[j][u]);
#pragma unroll
    for (int w = kChains / 2; w > 0; w /= 2)
#pragma unroll
      for (int u = 0; u < w; ++u) sum[u].join(sum[u + w]);
    acc[j] = sum[0];
  }
  if constexpr (kSlices > 1) {
    static_assert(kOut == 1 && kSlices == 2, "two k slices of one output per thread");
    if (slice > 0) sm.part[tid % (kTile * kTile)] = acc[0];
    __syncthreads();
    if (slice > 0) return;
    acc[0].join(sm.part[tid]);
  }

  const T alpha = scal<T>(args.alpha), beta = scal<T>(args.beta);
  const bool accumulate = args.flags & kFlagAccumulate;
  const bool beta_zero = args.flags & kFlagBetaZero;
#pragma unroll
  for (int j = 0; j < kOut; ++j) {
    if (!live[j]) continue;
    const int64_t m = m0 + (kNFast ? s + kSlow * j : f), n = n0 + (kNFast ? f : s + kSlow * j);
    T* p = C + offs(args.rsC, args.uC_m, m) + offs(args.csC, args.uC_n, n);
    const T ab = mul(alpha, acc[j].value());
    if (accumulate)
      *p = add(*p, ab);
    else if (beta_zero)
      *p = ab;
    else
      *p = add(ab, mul(beta, *p));
  }
}

// Grouped launches: blockIdx.x indexes the concatenated tile lists of
// group[0..nprob) (sorted by tile_begin, split-major within a problem);
// otherwise it is a tile of args0 and blockIdx.y its split.
template <class T, int kTile, bool kGroup>
__global__ void __launch_bounds__(kThreads)
small_contract(const GemmArgs args0, const SimtProblem* group, int nprob) {
  __shared__ __align__(16) SmallSmem<T, kTile> sm;
  __shared__ GemmArgs group_args;
  begin_dependent();
  int64_t tile = blockIdx.x, split = blockIdx.y;
  if constexpr (kGroup) {
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (group[mid].tile_begin <= tile) lo = mid; else hi = mid - 1;
    }
    tile -= group[lo].tile_begin;
    if (threadIdx.x == 0) group_args = group[lo].g;
    __syncthreads();
    const int64_t per = ((group_args.M + kTile - 1) / kTile) * ((group_args.N + kTile - 1) / kTile);
    split = tile / per;
    tile -= split * per;
  }
  const GemmArgs& args = kGroup ? group_args : args0;
  if (args.uC_n == 1 && args.uC_m != 1)
    small_tile<T, kTile, true>(args, tile, split, sm);
  else
    small_tile<T, kTile, false>(args, tile, split, sm);
}

template <class T>
cudaError_t launch(const GemmArgs& g, int tile, int splits, cudaStream_t stream) {
  const int64_t tiles = ((g.M + tile - 1) / tile) * ((g.N + tile - 1) / tile);
  if (tiles == 0) return cudaSuccess;
  if (tiles > 0x7fffffffLL || splits < 1 || splits > 65535) return cudaErrorInvalidConfiguration;
  const dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>(splits));
  return launch_dependent(tile == 16 ? small_contract<T, 16, false> : small_contract<T, 8, false>,
                          grid, dim3(kThreads), 0, stream, g, nullptr, 0);
}

}  // namespace

SmallForm small_form(int dtype, int64_t M, int64_t N, int64_t K, int64_t forced) {
  const bool cplx = dtype == T1M_COMPLEX128 || dtype == T1M_COMPLEX64;
  const bool wide = dtype == T1M_FLOAT64 || dtype == T1M_COMPLEX128;
  const double es = (cplx ? 2 : 1) * (wide ? 8 : 4);
  constexpr double kSms = 152;
  const int64_t ksteps = std::max<int64_t>(1, (K + kBK - 1) / kBK);
  // Large float64 outputs over few k: hundreds of small blocks per SM are all
  // start and end (4000 x 4000 over 8: 498 us against 270 on simt.cu's tile,
  // 1000 x 1000 43 against 28).  Up to 8 k both sum one chain: the same bits.
  const bool brief = dtype == T1M_FLOAT64 && K > 0 && K <= 8;
  SmallForm best{16, 1};
  double best_cost = 1e300;
  // Clocks of the busiest SM: whole blocks per SM times a block's k steps,
  // plus 2000 for the fill of the copy ring and the epilogue, plus, when
  // split, 6000 for the reduction launch and 1 per 8 bytes x SM of partials
  // written and read back.
  auto consider = [&](int tile, double tiles, double per_k, double floor_k, int64_t s) {
    const int64_t per = (ksteps + s - 1) / s;
    const int64_t used = (ksteps + per - 1) / per;
    if (forced <= 0 && used != s) return;  // the same partition as a smaller s
    const double waves = double(static_cast<int64_t>((tiles * used + kSms - 1) / kSms));
    const double k = double(std::min(K, per * kBK));
    double cost = std::max(waves * per_k, floor_k) * k + 2000;
    if (used > 1) cost += 6000 + 2.0 * double(used) * double(M) * double(N) * es / (8 * kSms);
    if (cost < best_cost) {
      best_cost = cost;
      best = {tile, static_cast<int>(used)};
    }
  };
  // More forced ranges than k steps of 16 (other kernels count shorter steps):
  // the tile of as many ranges as there are steps.
  const int64_t first = forced > 0 ? std::min(forced, ksteps) : 1;
  for (int64_t s = first; s <= (forced > 0 ? first : std::min<int64_t>(64, ksteps)); ++s) {
    for (int tile : {16, 8}) {
      const double tiles = double((M + tile - 1) / tile) * double((N + tile - 1) / tile);
      // A block's clocks per k: its FMAs (FP64: two per clock, four per
      // complex product) or the shared-memory reads of its four warps; a
      // stage of 16 k takes at least its latency.
      const double per_k = wide ? double(tile) * tile * (cplx ? 4 : 1) / 2 : (tile == 16 ? 18 : 9);
      // Float64 over at most 8 k: the start and end of a block, 2100 clocks.
      consider(tile, tiles, brief ? std::max(per_k, 2100.0 / double(K)) : per_k, wide ? 0 : 20, s);
    }
    if (brief) {
      // simt.cu's tile: 8192 products per k, always 8 k of them.
      const double tiles = double((M + 127) / 128) * double((N + 63) / 64);
      consider(0, tiles, 8 * 8192 / 2 / double(K), 0, s);
    }
    if (!wide) {
      // simt.cu's tile: 8192 (complex, four FMAs) or 16384 products per k on
      // 128 lanes, two blocks per SM.
      const double tiles = cplx ? double((M + 63) / 64) * double((N + 127) / 128)
                                : double((M + 127) / 128) * double((N + 127) / 128);
      consider(0, tiles, cplx ? 256 : 128, cplx ? 256 : 128, s);
    }
  }
  return best;
}

cudaError_t launch_small(int dtype, int tile, const GemmArgs& g, int splits, cudaStream_t stream) {
  switch (dtype) {
    case T1M_FLOAT32: return launch<float>(g, tile, splits, stream);
    case T1M_FLOAT64: return launch<double>(g, tile, splits, stream);
    case T1M_COMPLEX64: return launch<float2>(g, tile, splits, stream);
    default: return launch<double2>(g, tile, splits, stream);
  }
}

cudaError_t launch_small_group(int dtype, const SimtProblem* dev, int nprob, int64_t total_tiles,
                               cudaStream_t stream) {
  if (total_tiles <= 0) return cudaSuccess;
  if (total_tiles > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
  const GemmArgs none{};
  const dim3 grid(static_cast<unsigned>(total_tiles));
  auto run = [&](auto kernel) {
    return launch_dependent(kernel, grid, dim3(kThreads), 0, stream, none, dev, nprob);
  };
  return dtype == T1M_COMPLEX128 ? run(small_contract<double2, kSmallTile, true>)
                                 : run(small_contract<double, kSmallTile, true>);
}

}  // namespace gb300
}  // namespace t1m
