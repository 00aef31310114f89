// Op-level kernels behind the reference extension's four attention entry
// points: scores + neighbourhood softmax (forward, backward) and the depthwise
// steerable convolution under given weights (forward, backward).
//
// Semantics follow src/gm_attention/nn/fused/attention.h of the reference
// (scores :145-165, softmax :295-316, softmax backward :320-348, depthwise
// message :174-206, its backward :211-232); the kernels themselves are new:
//
//  * scores, head-grouped (H a power of two, the usual case): one or two warps per target, the lanes split into H head
//    groups (narrow heads: several times over, the groups taking the target's edges in turn), every lane owning a few copies
//    of every frequency; four edges' gathers of k_j are in flight; the raw logits go to alpha and the same warps normalise
//    the row in place.
//  * scores, general: one block per target, one WARP per edge with the lanes striding the key row (coalesced
//    128-byte reads of k_j), per-head sums by warp shuffle; the row's logits live in shared memory (or, for very
//    large neighbourhoods, in the alpha output itself) and are normalised there.
//  * softmax backward, conv forward / backward: one warp per target and one LANE per work item -- a (head,
//    frequency, copy) or (frequency, copy): a scalar column or a (re, im) column pair -- listed once per CTA in
//    shared memory.  Where there are few items, groups of lanes take the node's edges in turn and their sums meet by shuffles.
//    Four edges' loads are in flight (conv backward: three), pairs are read as pairs where the addresses allow, atomics only for
//    the scattered dk / dv.
#include "common.cuh"

namespace gmb {
namespace {

constexpr int MAX_H = 8;
constexpr int MAX_F = 8;
constexpr int DESC = 5;

template <typename T> struct Pair;
template <> struct Pair<float> { using type = float2; };
template <> struct Pair<double> { using type = double2; };

// (x, y) at p: one vector access when the address allows it: decided from the address itself, or (VEC) known by the caller
template <bool VEC, typename T>
__device__ __forceinline__ void load_pair(const T* p, T& x, T& y) {
  if (VEC || (reinterpret_cast<uintptr_t>(p) & (2 * sizeof(T) - 1)) == 0) {
    const typename Pair<T>::type t = *reinterpret_cast<const typename Pair<T>::type*>(p);
    x = t.x; y = t.y;
  } else {
    x = p[0]; y = p[1];
  }
}
template <bool VEC, typename T>
__device__ __forceinline__ void store_pair(T* p, T x, T y) {
  if (VEC || (reinterpret_cast<uintptr_t>(p) & (2 * sizeof(T) - 1)) == 0) {
    typename Pair<T>::type t;
    t.x = x; t.y = y;
    *reinterpret_cast<typename Pair<T>::type*>(p) = t;
  } else {
    p[0] = x; p[1] = y;
  }
}
// Whether all of these addresses (as bits set in any of them) are those of pairs
template <typename T> __device__ __forceinline__ bool whole_pairs(uintptr_t bits) { return (bits & (2 * sizeof(T) - 1)) == 0; }
template <typename T> __device__ __forceinline__ uintptr_t bits_of(const T* p) { return reinterpret_cast<uintptr_t>(p); }

// f(t, n, j) for the edges t .. t + n - 1 of a node's `degree` and their sources j that are this turn's of `turns`: U at a time,
// the last ones one at a time; AHEAD: the sources are read while the U edges before them are worked on.
template <int U, bool AHEAD, typename F>
__device__ __forceinline__ void for_edges(int turn, int turns, int degree, const int64_t* source, const F& f) {
  auto single = [&](int t) {
    for (; t < degree; ++t) f(t, std::integral_constant<int, 1>(), [&](int) { return (unsigned)source[t]; });
  };
  if constexpr (AHEAD) {
    unsigned ahead[U];
    auto read = [&](int from) {
#pragma unroll
      for (int u = 0; u < U; ++u) ahead[u] = (unsigned)source[from + u];
    };
    int t = U * turn;
    if (t + U <= degree) read(t);
    for (; t + U <= degree; t += U * turns) {
      unsigned j[U];
#pragma unroll
      for (int u = 0; u < U; ++u) j[u] = ahead[u];
      if (t + U * turns + U <= degree) read(t + U * turns);
      f(t, std::integral_constant<int, U>(), [&](int u) { return j[u]; });
    }
    single(t);
  } else {
    for (int t = U * turn; t < degree; t += U * turns) {
      if (t + U <= degree) f(t, std::integral_constant<int, U>(), [&](int u) { return (unsigned)source[t + u]; });
      else single(t);
    }
  }
}

// ------------------------------------------------------------------ softmax

template <typename T>
struct SoftmaxArgs {
  const T *q, *k, *transport, *bias, *alpha_in, *dalpha;
  const uint8_t* inside;
  const int64_t *desc, *row_ptr, *source;
  T *alpha, *dq, *dk;
  int64_t n_nodes;
  int D, F, orders, H;
  int slots;  // shared-memory logit slots per block (0: keep the logits in alpha)
  int shares;  // grouped scores: groups of a warp's lanes that take a target's edges in turn
  T scale;
};

constexpr int SM_THREADS = 128;

template <typename T>
__global__ void __launch_bounds__(SM_THREADS) softmax_forward_kernel(SoftmaxArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* q_s = reinterpret_cast<T*>(smem_raw);
  T* logit_s = q_s + a.D;
  __shared__ int d_n[MAX_F], d_mult[MAX_F], d_off[MAX_F];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = SM_THREADS / 32;
  if (threadIdx.x < a.F) {
    d_n[threadIdx.x] = (int)a.desc[threadIdx.x * DESC + 0];
    d_mult[threadIdx.x] = (int)a.desc[threadIdx.x * DESC + 1];
    d_off[threadIdx.x] = (int)a.desc[threadIdx.x * DESC + 2];
  }
  for (int64_t i = blockIdx.x; i < a.n_nodes; i += gridDim.x) {
    const int64_t e0 = a.row_ptr[i], e1 = a.row_ptr[i + 1];
    const int deg = (int)(e1 - e0);
    __syncthreads();  // the previous node's reads of q_s / logit_s are done (and d_* are written)
    if (deg == 0) continue;
    for (int c = threadIdx.x; c < a.D; c += SM_THREADS) q_s[c] = a.q[i * a.D + c];
    T* logits = (deg * a.H <= a.slots) ? logit_s : a.alpha + e0 * a.H;
    __syncthreads();
    for (int t = warp; t < deg; t += n_warps) {
      const int64_t e = e0 + t, j = a.source[e];
      const T* k_j = a.k + j * a.D;
      const T* tau_e = a.transport + e * a.orders * 2;
      const T bias = a.bias[e];
      for (int h = 0; h < a.H; ++h) {
        T acc = T(0);
        for (int f = 0; f < a.F; ++f) {
          const int n = d_n[f], a_n = d_mult[f];
          if (n == 0) {
            const int base = d_off[f] + h * a_n;
            for (int u = lane; u < a_n; u += 32) acc += q_s[base + u] * k_j[base + u];
          } else {
            const T tr = tau_e[2 * n], ti = tau_e[2 * n + 1];
            const int base = d_off[f] + 2 * h * a_n;
            for (int u = lane; u < a_n; u += 32) {
              const T kr = k_j[base + 2 * u], ki = k_j[base + 2 * u + 1];
              acc += q_s[base + 2 * u] * (tr * kr - ti * ki) + q_s[base + 2 * u + 1] * (tr * ki + ti * kr);
            }
          }
        }
        acc = warp_sum(acc);
        if (lane == 0) logits[t * a.H + h] = a.scale * acc + bias;
      }
    }
    __syncthreads();
    for (int h = warp; h < a.H; h += n_warps) {
      T m = neg_inf<T>();
      for (int t = lane; t < deg; t += 32) {
        const T lw = logits[t * a.H + h];
        if (a.inside[e0 + t] && lw > m) m = lw;  // masked edges never set the shift
      }
      m = warp_max(m);
      T sum = T(0);
      for (int t = lane; t < deg; t += 32) {
        const T u = a.inside[e0 + t] ? gm_exp(logits[t * a.H + h] - m) : T(0);
        logits[t * a.H + h] = u;
        sum += u;
      }
      sum = warp_sum(sum);
      for (int t = lane; t < deg; t += 32) a.alpha[(e0 + t) * a.H + h] = logits[t * a.H + h] / sum;
    }
  }
}


// Scores + softmax with the lanes of a warp split into H head groups (H a power of two): PARTS warps per target,
// a group of L = 32 / H lanes owns a head and each lane the copies u = s, s + L, ... of every frequency (at most
// R per frequency).  Per edge every lane reads its own columns of k_j (the groups together read the whole row once),
// the group reduces with log2(L) xor-shuffles, and all H logits of the edge appear at once.  The raw logits go to
// alpha, the row is then normalised in place by the same warps (masked edges never enter the shift or the sum).
// NF: the number of descriptor rows when known at compile time (3 or 4 frequencies: the usual head types), 0 = up to MAX_F
//
// PARTS warps share a target, four edges of it in turn each.  Two where the launch is about as long as its longest target's chain
// of edges (about 1 us for four), one where there are edges enough to hide it: then every warp of a pair only repeats the other's
// q_i and waits for it.  us with one / two, float32: 128 x 256, radius 3 pi / 128, 4 heads of 8 x (m <= 3) (3 899 edges per edge of the
// longest target) 584 / 509; 64 x 128, radius 4 pi / 64 (2 126) 338 / 187; 128 x 256, radius 4 pi / 128 (4 931) equal; 2 562 points of even degree 200, 4 of
// 8 x (m <= 2), 130 / 79; 10 242 points, degree 12 24 / 30, degree 200 334 / 323; 120 000, degree 12 289 / 383.  Eight heads' groups of four lanes take
// longer over an edge: 10 242 points, degree 40 100 / 91 and 203 / 187, degree 200 534 / 468, but degree 21 56 / 57 and (4 x (m <= 1)) 32 / 36, 40 962 202 / 232.
// 288 timings: 1.1 % above the better of the two in the mean, one frequency pair of 2 562 points with eight heads 34 % (11 us).
//
// What bounds it: the issue of what surrounds the gathers.  With every slot of a lane looked up and branched around in the walk the
// first of these took 740 us, with the kind of a slot known and lanes without a copy reading nothing 511 (two edges in flight 683,
// two with their sources read ahead 614); 99 x 198, radius 2.5 pi / 99: 8 heads of 8 x (m <= 2) 494 -> 278, of 16 x (m <= 2) 2 014 -> 546,
// 120 x 200, radius 3 pi / 120, 8 heads of 4 x (m <= 1) 447 -> 262.  CTAs of 8 or 16 warps on neighbouring targets: 583, 566.
int score_parts(int64_t n_nodes, int64_t n_edges, int64_t deg_max, int H) {
  return n_edges <= 4096 * deg_max || (H == 8 && n_edges >= 32 * n_nodes) ? 2 : 1;
}

// The logits of a target's edges turn, turn + turns, ... and their maximum, in the descriptor's order and number by number.  Not
// inlined: in the kernel's body it cost the usual walk 17 % (513 -> 602 us).
template <typename T>
__device__ __noinline__ T logits_in_any_order(const SoftmaxArgs<T>* args, int64_t i, int turn, int turns, int h, int s, int L, unsigned group_mask) {
  const SoftmaxArgs<T>& a = *args;
  const T* q_i = a.q + i * a.D;
  T m = neg_inf<T>();
  for (int64_t e = a.row_ptr[i] + turn; e < a.row_ptr[i + 1]; e += turns) {
    const T *k_j = a.k + a.source[e] * a.D, *tau = a.transport + e * a.orders * 2;
    T sum = T(0);
    for (int f = 0; f < a.F; ++f) {
      const int n = (int)a.desc[f * DESC], a_n = (int)a.desc[f * DESC + 1], off = (int)a.desc[f * DESC + 2];
      for (int u = s; u < a_n; u += L) {
        const int c = off + (n == 0 ? 1 : 2) * (h * a_n + u);
        if (n == 0) sum += q_i[c] * k_j[c];
        else sum += q_i[c] * (tau[2 * n] * k_j[c] - tau[2 * n + 1] * k_j[c + 1]) + q_i[c + 1] * (tau[2 * n] * k_j[c + 1] + tau[2 * n + 1] * k_j[c]);
      }
    }
    for (int o = L >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(group_mask, sum, o);
    const T lw = a.scale * sum + a.bias[e];
    if (a.inside[e] && lw > m) m = lw;
    if (s == 0) a.alpha[e * a.H + h] = lw;
  }
  return m;
}

template <typename T, int R, int NF, int PARTS, bool SHARED>
__global__ void __launch_bounds__(128) softmax_forward_grouped_kernel(const __grid_constant__ SoftmaxArgs<T> a) {
  constexpr int FN = NF ? NF : MAX_F, TARGETS = 4 / PARTS;
  __shared__ T max_s[TARGETS][PARTS][MAX_H], sum_s[TARGETS][PARTS][MAX_H];
  const int lane = threadIdx.x & 31, part = (threadIdx.x >> 5) % PARTS, mine = (threadIdx.x >> 5) / PARTS;
  const int64_t x = (int64_t)blockIdx.x * TARGETS + mine;
  const bool present = x < a.n_nodes;
  const int64_t i = present ? from_both_ends(x, a.n_nodes) : 0;
  // narrow heads leave lanes free: a.shares groups of H heads' lanes take the target's edges in turn
  const int shares = SHARED ? a.shares : 1, full = 32 / a.H, L = full / shares;
  const int share = SHARED ? lane / (a.H * L) : 0, h = SHARED ? lane / L % a.H : lane / L, s = lane % L;
  const unsigned group_mask = SHARED ? ((1u << (a.H * L)) - 1u) << (share * a.H * L) : 0xffffffffu;
  int col[FN][R], order[FN];
  uintptr_t bits = bits_of(a.k) | bits_of(a.transport) | (uintptr_t)a.D * sizeof(T);
  bool sorted = true;  // NF: frequency 0 can only be the first
  T qr[FN][R], qi[FN][R];
#pragma unroll
  for (int f = 0; f < FN; ++f) {
    order[f] = -1;
#pragma unroll
    for (int r = 0; r < R; ++r) { col[f][r] = -1; qr[f][r] = qi[f][r] = T(0); }
    if (NF || f < a.F) {
      const int n = (int)a.desc[f * DESC], a_n = (int)a.desc[f * DESC + 1], off = (int)a.desc[f * DESC + 2];
      order[f] = n;
      if (n != 0) bits |= (uintptr_t)off * sizeof(T);
      else if (NF && f > 0) sorted = false;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int u = s + L * r;
        if (u < a_n) {
          col[f][r] = off + (n == 0 ? 1 : 2) * (h * a_n + u);
          qr[f][r] = a.q[i * a.D + col[f][r]];
          if (n != 0) qi[f][r] = a.q[i * a.D + col[f][r] + 1];
        }
      }
    }
  }
  const int64_t e0 = a.row_ptr[i], e1 = present ? a.row_ptr[i + 1] : e0;
  const int degree = (int)(e1 - e0);
  const int64_t* source = a.source + e0;
  const T *transport = a.transport + e0 * a.orders * 2, *bias = a.bias + e0;
  const uint8_t* inside = a.inside + e0;
  T* const alpha = a.alpha + e0 * a.H + h;
  T m = neg_inf<T>();
  constexpr int U = 4;  // edges in flight: their gathers of k_j are issued together (8: 0.96 ms against 0.88)
  auto walk = [&](auto is_vec) {  // VEC: every (re, im) and phase is read as a pair
    constexpr bool VEC = decltype(is_vec)::value;
    // this lane's share of <q_i, tau k_j> for one edge
    auto dot = [&](int t, unsigned j) -> T {
      const T *k_j = a.k + (size_t)j * (unsigned)a.D, *tau = transport + (size_t)(unsigned)t * (2u * a.orders);
      T sum = T(0);
#pragma unroll
      for (int f = 0; f < FN; ++f) {
        if (!NF && order[f] < 0) continue;
        if ((!NF || f == 0) && order[f] == 0) {
#pragma unroll
          for (int r = 0; r < R; ++r) sum += qr[f][r] * (col[f][r] >= 0 ? k_j[col[f][r]] : T(0));
          continue;
        }
        T tr = T(0), ti = T(0);
        if (col[f][0] >= 0) load_pair<VEC>(tau + 2 * order[f], tr, ti);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          T kr = T(0), ki = T(0);
          if (col[f][r] >= 0) load_pair<VEC>(k_j + col[f][r], kr, ki);
          sum += qr[f][r] * (tr * kr - ti * ki) + qi[f][r] * (tr * ki + ti * kr);
        }
      }
      return sum;
    };
    auto edges = [&](int t, auto count, auto from) {
      constexpr int N = decltype(count)::value;
      T sum[N];
#pragma unroll
      for (int u = 0; u < N; ++u) sum[u] = dot(t + u, from(u));
      for (int o = L >> 1; o > 0; o >>= 1) {
#pragma unroll
        for (int u = 0; u < N; ++u) sum[u] += __shfl_xor_sync(group_mask, sum[u], o);
      }
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const T lw = a.scale * sum[u] + bias[t + u];
        if (inside[t + u] && lw > m) m = lw;
        if (s == 0) alpha[(size_t)(unsigned)(t + u) * (unsigned)a.H] = lw;
      }
    };
    for_edges<U, false>(part * shares + share, PARTS * shares, degree, source, edges);
  };
  if (!sorted) m = present ? logits_in_any_order(&a, i, part * shares + share, PARTS * shares, h, s, L, group_mask) : m;
  else if (whole_pairs<T>(bits)) walk(std::true_type());
  else walk(std::false_type());
  for (int o = a.H * L; SHARED && o < 32; o <<= 1) {
    const T other = __shfl_xor_sync(0xffffffffu, m, o);
    m = other > m ? other : m;
  }
  if constexpr (PARTS > 1) {
    if (s == 0) max_s[mine][part][h] = m;
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PARTS; ++p) m = max_s[mine][p][h] > m ? max_s[mine][p][h] : m;
  } else {
    __syncwarp();
  }
  // normalise: a head's lanes stride the row's edges.  The sum is that of two halves (every other `full` edges),
  // so that one warp gets the bits of two: a chunk of an edge set may be given to one, the whole set to two
  const int place = s + L * share;
  auto head_sum = [&](T v) {
    for (int o = full >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, SHARED && o >= L ? o / L * (a.H * L) : o);
    return v;
  };
  auto weigh = [&](int t) {
    const T u = inside[t] ? gm_exp(alpha[(size_t)(unsigned)t * (unsigned)a.H] - m) : T(0);
    alpha[(size_t)(unsigned)t * (unsigned)a.H] = u;
    return u;
  };
  T sum = T(0);
  if constexpr (PARTS > 1) {
    static_assert(PARTS == 2, "as many halves as there are");
    for (int t = place + full * part; t < degree; t += full * PARTS) sum += weigh(t);
    sum = head_sum(sum);
    if (place == 0) sum_s[mine][part][h] = sum;
    __syncthreads();
    sum = sum_s[mine][0][h] + sum_s[mine][1][h];
  } else {
    T other = T(0);
    for (int t = place; t < degree; t += 2 * full) {
      sum += weigh(t);
      if (t + full < degree) other += weigh(t + full);
    }
    sum = head_sum(sum) + head_sum(other);
  }
  for (int t = place + full * part; t < degree; t += full * PARTS) alpha[(size_t)(unsigned)t * (unsigned)a.H] /= sum;
}

// ------------------------------------------------------------------ depthwise conv

template <typename T>
struct ConvArgs {
  const T *v, *rc, *cc, *transport, *angular, *rho, *weights, *g;
  const int64_t *desc, *row_ptr, *source;
  T *out, *dv, *drc, *dcc;
  int64_t n_nodes;
  int D, F, orders, A0, W;
};

template <typename T>
__device__ __forceinline__ T rho_power(T rho, int n) {  // (r / c)^{2n} by repeated multiplication from 1 (n >= 1)
  const T two = rho * rho, four = two * rho * rho;
  T s = n == 1 ? two : four;
  for (int i = 2; i < n; ++i) s = s * rho * rho;
  return s;
}

// One work item of the depthwise conv = one copy of one frequency: a scalar column, or a (re, im) column pair.
struct ConvItem {
  int col;    // flat column (of the real part)
  int order;  // frequency n
  int coef;   // index into a row of rc (n = 0) / of cc: A at coef, B at coef + 2 mult (n > 0)
  int mult;
};

// A warp's lanes on up to 32 items: as many groups of lanes as there is room for (4 lanes at least), which take a node's edges in
// turn.
struct Lanes {
  int width, item, group, groups;
  __device__ __forceinline__ Lanes(int lane, int n) {
    width = n > 16 ? 32 : n > 8 ? 16 : n > 4 ? 8 : 4;
    item = lane & (width - 1);
    group = lane / width;
    groups = 32 / width;
  }
  template <typename T> __device__ __forceinline__ T sum(T v) const {  // over the groups
    for (int o = width; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
};
// p[0] += x, p[1] += y.  A float pair on an 8-byte boundary (ALIGNED: known to be on one) is one vector reduction: half as many
// operations for the L2 units.  128 x 256, radius 3 pi / 128, 4 heads of 8 x (m <= 3), float32: 1 098 -> 897 us for the scores' backward.
// (The depthwise backward lost by it, 1 045 -> 1 190, while every access tested its address; now it gains, 745 -> 712.)
template <bool VECTOR, bool ALIGNED = false, typename T>
__device__ __forceinline__ void add_pair(T* p, T x, T y) {
  if constexpr (VECTOR && std::is_same<T, float>::value) {
    if (ALIGNED || (reinterpret_cast<uintptr_t>(p) & 7) == 0) {
      asm volatile("red.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(p), "f"(x), "f"(y));
      return;
    }
  }
  atomicAdd(p, x);
  atomicAdd(p + 1, y);
}

// One (head, frequency, copy) of the scores' backward: a scalar column or a (re, im) column pair of one head
struct ScoreItem {
  int col, order, head, pad;
};

// Backward of scores + softmax: a warp per target node.  The lanes first reduce sum_e alpha dalpha per head, then
// every lane owns one item and walks the node's edges, four edges' gathers in flight; dk is accumulated atomically.
// VECTOR: pairs of it by one reduction; VEC: every pair is read and written as one.
template <bool VECTOR, bool VEC, bool AHEAD, typename T>
__device__ __forceinline__ void softmax_backward_node(const SoftmaxArgs<T>& a, const ScoreItem* items_s, int n_items, int n_real, int64_t i) {
  const int lane = threadIdx.x & 31;
  constexpr int U = 4;
  const int64_t e0 = a.row_ptr[i];
  const int degree = (int)(a.row_ptr[i + 1] - e0);
  const T *alpha = a.alpha_in + e0 * a.H, *dalpha = a.dalpha + e0 * a.H, *transport = a.transport + e0 * a.orders * 2;
  const int64_t* source = a.source + e0;
  T total_of_lane = T(0);  // lane h < H ends up with sum_e alpha[e, h] dalpha[e, h]
  for (int h = 0; h < a.H; ++h) {
    T total = T(0);
    for (int t = lane; t < degree; t += 32) total += alpha[(size_t)t * a.H + h] * dalpha[(size_t)t * a.H + h];
    total = warp_sum(total);
    if (lane == h) total_of_lane = total;
  }
  for (int t0 = 0; t0 < n_items;) {
    // a block of 32 items never mixes scalar and complex items
    const int t1 = t0 < n_real ? min(t0 + 32, n_real) : min(t0 + 32, n_items);
    const Lanes lanes(lane, t1 - t0);
    const bool active = t0 + lanes.item < t1;
    const ScoreItem it = items_s[active ? t0 + lanes.item : t0];
    const T total = __shfl_sync(0xffffffffu, total_of_lane, it.head);
    const T *al_at = alpha + it.head, *da_at = dalpha + it.head, *k_at = a.k + it.col;
    T* dk_at = a.dk + it.col;
    if (t0 < n_real) {
      const T q_c = a.q[i * a.D + it.col];
      T dq = T(0);
      if (active)
        for_edges<U, AHEAD>(lanes.group, lanes.groups, degree, source, [&](int t, auto count, auto from) {
          constexpr int N = decltype(count)::value;
          size_t j[N];
          T al[N], da[N], kc[N];
#pragma unroll
          for (int u = 0; u < N; ++u) {
            j[u] = (size_t)from(u) * (unsigned)a.D;
            al[u] = al_at[(size_t)(unsigned)(t + u) * (unsigned)a.H];
            da[u] = da_at[(size_t)(unsigned)(t + u) * (unsigned)a.H];
            kc[u] = k_at[j[u]];
          }
#pragma unroll
          for (int u = 0; u < N; ++u) {
            const T ds = a.scale * al[u] * (da[u] - total);
            dq += ds * kc[u];
            atomicAdd(dk_at + j[u], ds * q_c);
          }
        });
      dq = lanes.sum(dq);
      if (active && lanes.group == 0) a.dq[i * a.D + it.col] = dq;
    } else {
      T q_r, q_i;
      load_pair<VEC>(a.q + i * a.D + it.col, q_r, q_i);
      T dq_r = T(0), dq_i = T(0);
      const T* tau_at = transport + it.order * 2;
      const unsigned tau_step = 2 * a.orders;
      if (active)
        for_edges<U, AHEAD>(lanes.group, lanes.groups, degree, source, [&](int t, auto count, auto from) {
          constexpr int N = decltype(count)::value;
          size_t j[N];
          T al[N], da[N], tr[N], ti[N], kr[N], ki[N];
#pragma unroll
          for (int u = 0; u < N; ++u) {
            j[u] = (size_t)from(u) * (unsigned)a.D;
            al[u] = al_at[(size_t)(unsigned)(t + u) * (unsigned)a.H];
            da[u] = da_at[(size_t)(unsigned)(t + u) * (unsigned)a.H];
            load_pair<VEC>(tau_at + (size_t)(unsigned)(t + u) * tau_step, tr[u], ti[u]);
            load_pair<VEC>(k_at + j[u], kr[u], ki[u]);
          }
#pragma unroll
          for (int u = 0; u < N; ++u) {
            const T ds = a.scale * al[u] * (da[u] - total);
            dq_r += ds * (tr[u] * kr[u] - ti[u] * ki[u]);  // (tau k)
            dq_i += ds * (tr[u] * ki[u] + ti[u] * kr[u]);
            add_pair<VECTOR>(dk_at + j[u], ds * (tr[u] * q_r + ti[u] * q_i), ds * (tr[u] * q_i - ti[u] * q_r));  // conj(tau) q
          }
        });
      dq_r = lanes.sum(dq_r);
      dq_i = lanes.sum(dq_i);
      if (active && lanes.group == 0) store_pair<VEC>(a.dq + i * a.D + it.col, dq_r, dq_i);
    }
    t0 = t1;
  }
}

template <typename T, bool VECTOR, bool AHEAD>
__global__ void __launch_bounds__(128) softmax_backward_kernel(const __grid_constant__ SoftmaxArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ScoreItem* items_s = reinterpret_cast<ScoreItem*>(smem_raw);
  int n_items = 0, n_real = 0;
  uintptr_t bits = bits_of(a.q) | bits_of(a.k) | bits_of(a.transport) | bits_of(a.dq) | (uintptr_t)a.D * sizeof(T);
  auto list = [&](int f, int at) {  // the items of row f from `at` on; their number
    const int n = (int)a.desc[f * DESC], a_n = (int)a.desc[f * DESC + 1], off = (int)a.desc[f * DESC + 2], dim = (int)a.desc[f * DESC + 4];
    for (int x = threadIdx.x; x < a.H * a_n; x += blockDim.x) items_s[at + x] = ScoreItem{off + dim * x, n, x / a_n, 0};
    if (n != 0) bits |= (uintptr_t)off * sizeof(T);
    return a.H * a_n;
  };
  bool behind = false;  // scalar items behind others
  for (int f = 0; f < a.F; ++f) {
    const int count = list(f, n_items);
    if (a.desc[f * DESC] == 0) {
      behind = behind || n_real != n_items;
      n_real += count;
    }
    n_items += count;
  }
  if (behind) {  // the walk wants them in front (two passes over the descriptor for everyone: 6 us of 780)
    __syncthreads();
    int scalar = 0, other = n_real;
    for (int f = 0; f < a.F; ++f) {
      int& at = a.desc[f * DESC] == 0 ? scalar : other;
      at += list(f, at);
    }
  }
  __syncthreads();
  const bool vec = whole_pairs<T>(bits);
  const int warps = blockDim.x >> 5;
  for (int64_t x = (int64_t)blockIdx.x * warps + (threadIdx.x >> 5); x < a.n_nodes; x += (int64_t)gridDim.x * warps) {
    const int64_t i = from_both_ends(x, a.n_nodes);
    if (vec) softmax_backward_node<VECTOR, true, AHEAD>(a, items_s, n_items, n_real, i);
    else softmax_backward_node<VECTOR, false, AHEAD>(a, items_s, n_items, n_real, i);
  }
}

// The items of the (single-head) descriptor, in column order, into shared memory; returns their number.
__device__ __forceinline__ int build_conv_items(const int64_t* desc, int F, ConvItem* items_s) {
  int total = 0;
  for (int f = 0; f < F; ++f) {
    const int64_t* row = desc + f * DESC;
    const int n = (int)row[0], a_n = (int)row[1], off = (int)row[2], coff = (int)row[3], dim = (int)row[4];
    for (int x = threadIdx.x; x < a_n; x += blockDim.x)
      items_s[total + x] = ConvItem{off + dim * x, n, n == 0 ? x : coff + 2 * x, a_n};
    total += a_n;
  }
  return total;
}

// Depthwise conv, forward: a warp per target node, a lane per item (scalar items and complex items in separate
// passes, so a pass never diverges); the node's edges are walked four at a time, with the four edges' loads issued before their
// arithmetic and the next four's sources read meanwhile.  What bounds it: the latency of the gathers and issue.  128 x 256, radius
// 3 pi / 128, 16 x (m <= 2), float32, forward and backward: 675 + 940 us with every access testing its address, 504 with sources read
// ahead and 110 registers, 428 with six CTAs to an SM (five 443; seven 420, but they spill) + 676 with seven; lane groups on narrow
// fields: 4 x (m <= 1), radius 2.5 pi / 128, 380 + 503 -> 98 + 118.
constexpr int CONV_UNROLL = 4, CONV_BACKWARD_UNROLL = 3;  // (backward: 710 us with four and five CTAs to an SM, 676 with three and seven)

template <bool VEC, typename T>
__device__ __forceinline__ void conv_forward_node(const ConvArgs<T>& a, const ConvItem* items_s, int n_items, int n_real, int64_t i) {
  const int lane = threadIdx.x & 31;
  const int64_t e0 = a.row_ptr[i];
  const int degree = (int)(a.row_ptr[i + 1] - e0);
  const int64_t* source = a.source + e0;
  const T* weights = a.weights + e0;
  for (int t0 = 0; t0 < n_real; t0 += 32) {
    const Lanes lanes(lane, n_real - t0);
    const bool active = t0 + lanes.item < n_real;
    const ConvItem it = items_s[active ? t0 + lanes.item : t0];
    const T *r_at = a.rc + e0 * a.A0 + it.coef, *v_at = a.v + it.col;
    T y = T(0);
    if (active)
      for_edges<CONV_UNROLL, true>(lanes.group, lanes.groups, degree, source, [&](int t, auto count, auto from) {
        constexpr int N = decltype(count)::value;
        T w[N], r[N], x[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
          w[u] = weights[t + u];
          r[u] = r_at[(size_t)(unsigned)(t + u) * (unsigned)a.A0];
          x[u] = v_at[(size_t)from(u) * (unsigned)a.D];
        }
#pragma unroll
        for (int u = 0; u < N; ++u) y += w[u] * (r[u] * x[u]);
      });
    y = lanes.sum(y);
    if (active && lanes.group == 0) a.out[i * a.D + it.col] = y;
  }
  for (int t0 = n_real; t0 < n_items; t0 += 32) {
    const Lanes lanes(lane, n_items - t0);
    const bool active = t0 + lanes.item < n_items;
    const ConvItem it = items_s[active ? t0 + lanes.item : t0];
    const int n = it.order;
    const T *rho_at = a.rho + e0, *v_at = a.v + it.col, *co_at = a.cc + e0 * a.W + it.coef;
    const T *tau_at = a.transport + (e0 * a.orders + n) * 2, *ang_at = a.angular + (e0 * a.orders + 2 * n) * 2;
    const unsigned phase_step = 2 * a.orders;
    const int behind = 2 * it.mult;
    T yr = T(0), yi = T(0);
    if (active)
      for_edges<CONV_UNROLL, true>(lanes.group, lanes.groups, degree, source, [&](int t, auto count, auto from) {
        constexpr int N = decltype(count)::value;
        T w[N], rho[N], tr[N], ti[N], vr[N], vi[N], Ar[N], Ai[N], Br[N], Bi[N], ar[N], ai[N];
#pragma unroll
        for (int u = 0; u < N; ++u) {
          const unsigned x = t + u;
          w[u] = weights[x];
          rho[u] = rho_at[x];
          load_pair<VEC>(v_at + (size_t)from(u) * (unsigned)a.D, vr[u], vi[u]);
          load_pair<VEC>(tau_at + (size_t)x * phase_step, tr[u], ti[u]);
          load_pair<VEC>(ang_at + (size_t)x * phase_step, ar[u], ai[u]);
          const T* co = co_at + (size_t)x * (unsigned)a.W;
          load_pair<VEC>(co, Ar[u], Ai[u]);
          load_pair<VEC>(co + behind, Br[u], Bi[u]);
        }
#pragma unroll
        for (int u = 0; u < N; ++u) {
          const T zr = tr[u] * vr[u] - ti[u] * vi[u], zi = tr[u] * vi[u] + ti[u] * vr[u];  // z = tau v
          const T p = rho_power(rho[u], n);
          const T wr = p * ar[u], wi = p * ai[u];
          // m = A z + w (B conj z)
          const T bzr = Br[u] * zr + Bi[u] * zi, bzi = Bi[u] * zr - Br[u] * zi;
          const T mr = (Ar[u] * zr - Ai[u] * zi) + (wr * bzr - wi * bzi);
          const T mi = (Ar[u] * zi + Ai[u] * zr) + (wr * bzi + wi * bzr);
          yr += w[u] * mr;
          yi += w[u] * mi;
        }
      });
    yr = lanes.sum(yr);
    yi = lanes.sum(yi);
    if (active && lanes.group == 0) store_pair<VEC>(a.out + i * a.D + it.col, yr, yi);
  }
}

// Backward: same walk and grouping; the edge-owned coefficient gradients are written once, dv is accumulated atomically.
template <bool VEC, typename T>
__device__ __forceinline__ void conv_backward_node(const ConvArgs<T>& a, const ConvItem* items_s, int n_items, int n_real, int64_t i) {
  const int lane = threadIdx.x & 31;
  const int64_t e0 = a.row_ptr[i];
  const int degree = (int)(a.row_ptr[i + 1] - e0);
  const int64_t* source = a.source + e0;
  const T* weights = a.weights + e0;
  for (int t0 = 0; t0 < n_real; t0 += 32) {
    const Lanes lanes(lane, n_real - t0);
    if (t0 + lanes.item >= n_real) continue;
    const ConvItem it = items_s[t0 + lanes.item];
    const T dy = a.g[i * a.D + it.col];
    const T *r_at = a.rc + e0 * a.A0 + it.coef, *v_at = a.v + it.col;
    T *dr_at = a.drc + e0 * a.A0 + it.coef, *dv_at = a.dv + it.col;
    for_edges<CONV_BACKWARD_UNROLL, true>(lanes.group, lanes.groups, degree, source, [&](int t, auto count, auto from) {
      constexpr int N = decltype(count)::value;
      T w[N], r[N], x[N];
      size_t j[N];
#pragma unroll
      for (int u = 0; u < N; ++u) {
        j[u] = (size_t)from(u) * (unsigned)a.D;
        w[u] = weights[t + u];
        r[u] = r_at[(size_t)(unsigned)(t + u) * (unsigned)a.A0];
        x[u] = v_at[j[u]];
      }
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const T dm = w[u] * dy;
        dr_at[(size_t)(unsigned)(t + u) * (unsigned)a.A0] = dm * x[u];
        atomicAdd(dv_at + j[u], dm * r[u]);
      }
    });
  }
  for (int t0 = n_real; t0 < n_items; t0 += 32) {
    const Lanes lanes(lane, n_items - t0);
    if (t0 + lanes.item >= n_items) continue;
    const ConvItem it = items_s[t0 + lanes.item];
    const int n = it.order;
    T dyr, dyi;
    load_pair<VEC>(a.g + i * a.D + it.col, dyr, dyi);
    const T *rho_at = a.rho + e0, *v_at = a.v + it.col, *co_at = a.cc + e0 * a.W + it.coef;
    const T *tau_at = a.transport + (e0 * a.orders + n) * 2, *ang_at = a.angular + (e0 * a.orders + 2 * n) * 2;
    T *dco_at = a.dcc + e0 * a.W + it.coef, *dv_at = a.dv + it.col;
    const unsigned phase_step = 2 * a.orders;
    const int behind = 2 * it.mult;
    for_edges<CONV_BACKWARD_UNROLL, true>(lanes.group, lanes.groups, degree, source, [&](int t, auto count, auto from) {
      constexpr int N = decltype(count)::value;
      T w[N], rho[N], tr[N], ti[N], vr[N], vi[N], Ar[N], Ai[N], Br[N], Bi[N], ar[N], ai[N];
      size_t j[N];
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const unsigned x = t + u;
        j[u] = (size_t)from(u) * (unsigned)a.D;
        w[u] = weights[x];
        rho[u] = rho_at[x];
        load_pair<VEC>(v_at + j[u], vr[u], vi[u]);
        load_pair<VEC>(tau_at + (size_t)x * phase_step, tr[u], ti[u]);
        load_pair<VEC>(ang_at + (size_t)x * phase_step, ar[u], ai[u]);
        const T* co = co_at + (size_t)x * (unsigned)a.W;
        load_pair<VEC>(co, Ar[u], Ai[u]);
        load_pair<VEC>(co + behind, Br[u], Bi[u]);
      }
#pragma unroll
      for (int u = 0; u < N; ++u) {
        const T zr = tr[u] * vr[u] - ti[u] * vi[u], zi = tr[u] * vi[u] + ti[u] * vr[u];
        const T p = rho_power(rho[u], n);
        const T wr = p * ar[u], wi = p * ai[u];
        const T dmr = w[u] * dyr, dmi = w[u] * dyi;
        // dA = dm conj(z); dB = (dm conj(w)) z
        const T dAr = dmr * zr + dmi * zi, dAi = dmi * zr - dmr * zi;
        const T cr = dmr * wr + dmi * wi, ci2 = dmi * wr - dmr * wi;
        const T dBr = cr * zr - ci2 * zi, dBi = cr * zi + ci2 * zr;
        T* dco = dco_at + (size_t)(unsigned)(t + u) * (unsigned)a.W;
        store_pair<VEC>(dco, dAr, dAi);
        store_pair<VEC>(dco + behind, dBr, dBi);
        // dz = conj(A) dm + w (B conj(dm)); dv = conj(tau) dz
        const T bdr = Br[u] * dmr + Bi[u] * dmi, bdi = Bi[u] * dmr - Br[u] * dmi;
        const T dzr = (Ar[u] * dmr + Ai[u] * dmi) + (wr * bdr - wi * bdi);
        const T dzi = (Ar[u] * dmi - Ai[u] * dmr) + (wr * bdi + wi * bdr);
        add_pair<VEC, VEC>(dv_at + j[u], tr[u] * dzr + ti[u] * dzi, tr[u] * dzi - ti[u] * dzr);
      }
    });
  }
}

template <typename T, bool BACKWARD>
__global__ void __launch_bounds__(128, sizeof(T) == 8 ? 4 : BACKWARD ? 7 : 6) conv_kernel(ConvArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ConvItem* items_s = reinterpret_cast<ConvItem*>(smem_raw);
  const int n_items = build_conv_items(a.desc, a.F, items_s);
  uintptr_t bits = bits_of(a.v) | bits_of(a.cc) | bits_of(a.transport) | bits_of(a.angular) | bits_of(a.out) | bits_of(a.g) | bits_of(a.dcc) | bits_of(a.dv) |
                   (uintptr_t)(a.D | a.W) * sizeof(T);
  for (int f = 0; f < a.F; ++f)
    if (a.desc[f * DESC] != 0) bits |= (uintptr_t)(a.desc[f * DESC + 2] | a.desc[f * DESC + 3]) * sizeof(T);
  __syncthreads();
  const bool vec = whole_pairs<T>(bits);
  int n_real = 0;  // items are in column order: the scalar block (frequency 0) first
  while (n_real < n_items && items_s[n_real].order == 0) ++n_real;
  const int warps = blockDim.x >> 5;
  for (int64_t x = (int64_t)blockIdx.x * warps + (threadIdx.x >> 5); x < a.n_nodes; x += (int64_t)gridDim.x * warps) {
    const int64_t i = from_both_ends(x, a.n_nodes);
    if constexpr (BACKWARD) {
      if (vec) conv_backward_node<true>(a, items_s, n_items, n_real, i);
      else conv_backward_node<false>(a, items_s, n_items, n_real, i);
    } else {
      if (vec) conv_forward_node<true>(a, items_s, n_items, n_real, i);
      else conv_forward_node<false>(a, items_s, n_items, n_real, i);
    }
  }
}

constexpr int CONV_THREADS = 128;  // 4 target nodes per CTA

int conv_grid(int64_t n_nodes) {  // CTAs stride the nodes, so that the item table is built once for several: up to
  // 64 per SM (16, all resident at once, leave the polar rows' nodes to few of them: depthwise 682 + 1 033 us against
  // 675 + 989; nodes of even degree: the same, 40 962 of degree 20 221 / 219)
  const int64_t want = (n_nodes + CONV_THREADS / 32 - 1) / (CONV_THREADS / 32);
  const int64_t cap = (int64_t)sm_count() * 64;
  return (int)(want < cap ? (want < 1 ? 1 : want) : cap);
}

int grid_for(int64_t n_nodes) { return (int)(n_nodes < (int64_t)1 << 30 ? n_nodes : (int64_t)1 << 30); }

template <typename T>
int softmax_forward_t(SoftmaxArgs<T> a, int64_t n_edges, int64_t deg_max, int max_mult, cudaStream_t stream) {
  // head-group kernel when the heads split a warp evenly and every lane owns at most 4 copies per frequency
  if ((a.H == 1 || a.H == 2 || a.H == 4 || a.H == 8) && max_mult > 0 && max_mult <= 4 * (32 / a.H)) {
    const int per_lane = (max_mult + 32 / a.H - 1) / (32 / a.H);
    a.shares = 1;
    // (with fewer edges most groups have none: of 5 edges each 1.13 to 1.19 of the time without groups for one frequency, 8 0.82 to 0.88)
    if (n_edges >= 7 * a.n_nodes)
      while (2 * a.shares * max_mult <= 32 / a.H) a.shares *= 2;
    auto go = [&](auto parts) {
      constexpr int P = decltype(parts)::value;
      const unsigned blocks = (unsigned)((a.n_nodes * P + 3) / 4);
      auto run = [&](auto kernel) { kernel<<<blocks, 128, 0, stream>>>(a); };
      auto frequencies = [&](auto nf) {
        constexpr int NF = decltype(nf)::value;
        if (a.shares > 1) run(softmax_forward_grouped_kernel<T, 1, NF, P, true>);
        else if (per_lane <= 1) run(softmax_forward_grouped_kernel<T, 1, NF, P, false>);
        else if (per_lane <= 2) run(softmax_forward_grouped_kernel<T, 2, NF, P, false>);
        else run(softmax_forward_grouped_kernel<T, 4, NF, P, false>);
      };
      if (a.F == 2) frequencies(std::integral_constant<int, 2>());
      else if (a.F == 3) frequencies(std::integral_constant<int, 3>());
      else if (a.F == 4) frequencies(std::integral_constant<int, 4>());
      else frequencies(std::integral_constant<int, 0>());
      return launch_status("gm_softmax_forward");
    };
    return score_parts(a.n_nodes, n_edges, deg_max, a.H) == 2 ? go(std::integral_constant<int, 2>()) : go(std::integral_constant<int, 1>());
  }
  // Logits in shared memory when the largest neighbourhood fits ~96 KiB; else kept in alpha.
  const size_t budget = 96 * 1024;
  size_t want = (size_t)deg_max * a.H;
  if ((want + a.D) * sizeof(T) > budget) want = 0;
  a.slots = (int)want;
  const size_t smem = (a.D + want) * sizeof(T);
  int status = allow_smem(softmax_forward_kernel<T>, smem, "gm_softmax_forward");
  if (status != GM_OK) return status;
  softmax_forward_kernel<T><<<grid_for(a.n_nodes), SM_THREADS, smem, stream>>>(a);
  return launch_status("gm_softmax_forward");
}

template <typename T>
int softmax_backward_t(SoftmaxArgs<T> a, int64_t n_edges, int64_t deg_max, cudaStream_t stream) {
  // dk by pairs where targets have many edges, on average or some of them: with few the vector reductions only hold the next
  // target's loads back.  us by numbers / by pairs: 163 842 points of even degree 12 492 / 552, 40 962 of degree 12 146 / 157, 10 242 of degree 21
  // 69 / 67, of degree 100 261 / 232; 64 x 128, radius 2 pi / 64 (mean 38, at most 257) 220 / 200; 128 x 256, radius 3 pi / 128 1 051 / 829.
  // Uneven only where the longest targets' chains are not lost among many short ones: the same with deg_max 8 x the degree at both ends,
  // as uneven / as even, mean over twelve types against the time before either: 40 000 nodes of 5 edges 1.22 / 0.94, of 16 0.89 / 0.73, 14 000 of 8 0.99 /
  // 0.87, of 24 0.67 / 0.67, of 40 0.59 / 0.63, 3 000 of 3 0.99 / 0.81, of 8 0.64 / 0.66; but 128 x 256, radius pi / 128 (mean 12, at most 257) 178 / 273 us.
  const bool few = a.n_nodes <= 12288, uneven = deg_max * a.n_nodes >= (n_edges >= (few ? 6 : 20) * a.n_nodes ? 4 : 12) * n_edges;
  const bool pairs = n_edges >= 24 * a.n_nodes || uneven;
  auto go = [&](auto kernel) { kernel<<<conv_grid(a.n_nodes), CONV_THREADS, a.D * sizeof(ScoreItem), stream>>>(a); };
  // Sources read ahead where the chains of gathers show: some targets' long ones, or few targets.  us without / with: 120 x 240, radius
  // 2.5 pi / 120, 4 heads of 5 x (m <= 3) 505 / 389, 99 x 198, radius 2.5 pi / 99, 8 of 5 x (m <= 2) 502 / 346, 8 of 16 x (m <= 2) 1 372 / 980, 128 x 256,
  // radius 3 pi / 128, 4 of 8 x (m <= 3) 822 / 775; points of even degree 40, 30 000, 4 of 8 x (m <= 2) 303 / 319, of 8 x (m <= 1) 207 / 229,
  // 3 000 85 / 82.  (A group of lanes per head and one walk for all frequencies: 765 and 286 on the lattices of 4 heads of 8 x (m <= 3), but
  // 1 158 for the 16 copies and 502 for the five, and 1 425 against 957 where 20 000 points have 40 edges each, 8 of 16 x (m <= 3).)
  const bool ahead = uneven || (few && (sizeof(T) == 4 || n_edges >= 16 * a.n_nodes));  // (float64, 3 000 of 5 edges each: 6 % slower ahead)
  if (pairs && ahead) go(softmax_backward_kernel<T, true, true>);
  else if (pairs) go(softmax_backward_kernel<T, true, false>);
  else if (ahead) go(softmax_backward_kernel<T, false, true>);
  else go(softmax_backward_kernel<T, false, false>);
  return launch_status("gm_softmax_backward");
}

int check_softmax(const void* q, const void* k, const void* transport, const void* bias, const uint8_t* inside,
                  const int64_t* desc, const int64_t* row_ptr, const int64_t* source, int64_t n_nodes, int64_t n_edges,
                  int D, int F, int orders, int H, int dtype) {
  GM_REQUIRE(n_nodes >= 0 && n_edges >= 0, GM_ERR_ARGUMENT, "gm_softmax: negative size");
  GM_REQUIRE(D >= 1, GM_ERR_ARGUMENT, "gm_softmax: D must be positive");
  GM_REQUIRE(H >= 1 && H <= MAX_H, GM_ERR_ARGUMENT, "gm_softmax: at most %d heads", MAX_H);
  GM_REQUIRE(F >= 0 && F <= MAX_F, GM_ERR_ARGUMENT, "gm_softmax: desc must be int64 (F <= %d, %d)", MAX_F, DESC);
  GM_REQUIRE(orders >= 1, GM_ERR_ARGUMENT, "gm_softmax: transport must be (n_edges, orders, 2)");
  GM_REQUIRE(dtype == GM_F32 || dtype == GM_F64, GM_ERR_UNSUPPORTED, "gm_softmax: dtype must be float32 or float64");
  if (n_nodes == 0) return GM_OK;
  GM_REQUIRE(q && k && desc && row_ptr, GM_ERR_ARGUMENT, "gm_softmax: null pointer");
  GM_REQUIRE(n_edges == 0 || (transport && bias && inside && source), GM_ERR_ARGUMENT, "gm_softmax: null edge table");
  return GM_OK;
}

}  // namespace
}  // namespace gmb

using namespace gmb;

extern "C" int gm_softmax_forward(const void* q, const void* k, const void* transport, const void* bias,
                                  const uint8_t* inside, const int64_t* desc, const int64_t* row_ptr,
                                  const int64_t* source, int64_t n_nodes, int64_t n_edges, int D, int F, int orders,
                                  int H, double scale, int64_t deg_max, int max_mult, int dtype, void* alpha, void* stream) {
  int status = check_softmax(q, k, transport, bias, inside, desc, row_ptr, source, n_nodes, n_edges, D, F, orders, H, dtype);
  if (status != GM_OK || n_nodes == 0 || n_edges == 0) return status;
  GM_REQUIRE(alpha, GM_ERR_ARGUMENT, "gm_softmax_forward: null alpha");
  GM_REQUIRE(deg_max >= 1, GM_ERR_ARGUMENT, "gm_softmax_forward: deg_max must be positive");
  auto run = [&](auto tag) {
    using T = decltype(tag);
    SoftmaxArgs<T> a{};
    a.q = (const T*)q; a.k = (const T*)k; a.transport = (const T*)transport; a.bias = (const T*)bias;
    a.inside = inside; a.desc = desc; a.row_ptr = row_ptr; a.source = source; a.alpha = (T*)alpha;
    a.n_nodes = n_nodes; a.D = D; a.F = F; a.orders = orders; a.H = H; a.scale = (T)scale;
    return softmax_forward_t<T>(a, n_edges, deg_max, max_mult, (cudaStream_t)stream);
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}

extern "C" int gm_softmax_backward(const void* dalpha, const void* q, const void* k, const void* transport,
                                   const void* bias, const uint8_t* inside, const int64_t* desc, const int64_t* row_ptr,
                                   const int64_t* source, const void* alpha, int64_t n_nodes, int64_t n_edges, int D,
                                   int F, int orders, int H, double scale, int64_t deg_max, int dtype, void* dq,
                                   void* dk, void* stream) {
  int status = check_softmax(q, k, transport, bias, inside, desc, row_ptr, source, n_nodes, n_edges, D, F, orders, H, dtype);
  if (status != GM_OK || n_nodes == 0) return status;
  GM_REQUIRE(dq && dk, GM_ERR_ARGUMENT, "gm_softmax_backward: null output");
  GM_REQUIRE(n_edges == 0 || (alpha && dalpha), GM_ERR_ARGUMENT, "gm_softmax_backward: null alpha / dalpha");
  auto run = [&](auto tag) {
    using T = decltype(tag);
    SoftmaxArgs<T> a{};
    a.q = (const T*)q; a.k = (const T*)k; a.transport = (const T*)transport; a.bias = (const T*)bias;
    a.inside = inside; a.desc = desc; a.row_ptr = row_ptr; a.source = source;
    a.alpha_in = (const T*)alpha; a.dalpha = (const T*)dalpha; a.dq = (T*)dq; a.dk = (T*)dk;
    a.n_nodes = n_nodes; a.D = D; a.F = F; a.orders = orders; a.H = H; a.scale = (T)scale;
    return softmax_backward_t<T>(a, n_edges, deg_max, (cudaStream_t)stream);
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}

namespace {

int check_conv(const void* v, const void* rc, const void* cc, const void* transport, const void* angular, const void* rho,
               const void* weights, const int64_t* desc, const int64_t* row_ptr, const int64_t* source, int64_t n_nodes,
               int64_t n_edges, int D, int F, int orders, int A0, int W, int dtype) {
  GM_REQUIRE(n_nodes >= 0 && n_edges >= 0, GM_ERR_ARGUMENT, "gm_conv: negative size");
  GM_REQUIRE(D >= 1, GM_ERR_ARGUMENT, "gm_conv: D must be positive");
  GM_REQUIRE(F >= 0 && F <= MAX_F, GM_ERR_ARGUMENT, "gm_conv: desc must be int64 (F <= %d, %d)", MAX_F, DESC);
  GM_REQUIRE(A0 >= 0 && W >= 0 && orders >= 1, GM_ERR_ARGUMENT, "gm_conv: bad widths");
  GM_REQUIRE(dtype == GM_F32 || dtype == GM_F64, GM_ERR_UNSUPPORTED, "gm_conv: dtype must be float32 or float64");
  if (n_nodes == 0) return GM_OK;
  GM_REQUIRE(v && desc && row_ptr, GM_ERR_ARGUMENT, "gm_conv: null pointer");
  if (n_edges > 0) {
    GM_REQUIRE(transport && angular && rho && weights && source, GM_ERR_ARGUMENT, "gm_conv: null edge table");
    GM_REQUIRE(A0 == 0 || rc, GM_ERR_ARGUMENT, "gm_conv: rc must hold (1, n_edges, a_0) entries");
    GM_REQUIRE(W == 0 || cc, GM_ERR_ARGUMENT, "gm_conv: cc must hold (1, n_edges, W) entries");
  }
  return GM_OK;
}

template <typename T>
ConvArgs<T> conv_args(const void* v, const void* rc, const void* cc, const void* transport, const void* angular,
                      const void* rho, const void* weights, const int64_t* desc, const int64_t* row_ptr,
                      const int64_t* source, int64_t n_nodes, int D, int F, int orders, int A0, int W) {
  ConvArgs<T> a{};
  a.v = (const T*)v; a.rc = (const T*)rc; a.cc = (const T*)cc; a.transport = (const T*)transport;
  a.angular = (const T*)angular; a.rho = (const T*)rho; a.weights = (const T*)weights;
  a.desc = desc; a.row_ptr = row_ptr; a.source = source;
  a.n_nodes = n_nodes; a.D = D; a.F = F; a.orders = orders; a.A0 = A0; a.W = W;
  return a;
}

}  // namespace

extern "C" int gm_conv_forward(const void* v, const void* rc, const void* cc, const void* transport, const void* angular,
                               const void* rho, const void* weights, const int64_t* desc, const int64_t* row_ptr,
                               const int64_t* source, int64_t n_nodes, int64_t n_edges, int D, int F, int orders, int A0,
                               int W, int dtype, void* out, void* stream) {
  int status = check_conv(v, rc, cc, transport, angular, rho, weights, desc, row_ptr, source, n_nodes, n_edges, D, F, orders, A0, W, dtype);
  if (status != GM_OK || n_nodes == 0) return status;
  GM_REQUIRE(out, GM_ERR_ARGUMENT, "gm_conv_forward: null out");
  auto run = [&](auto tag) {
    using T = decltype(tag);
    auto a = conv_args<T>(v, rc, cc, transport, angular, rho, weights, desc, row_ptr, source, n_nodes, D, F, orders, A0, W);
    a.out = (T*)out;
    conv_kernel<T, false><<<conv_grid(n_nodes), CONV_THREADS, D * sizeof(ConvItem), (cudaStream_t)stream>>>(a);
    return launch_status("gm_conv_forward");
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}

extern "C" int gm_conv_backward(const void* g, const void* v, const void* rc, const void* cc, const void* transport,
                                const void* angular, const void* rho, const void* weights, const int64_t* desc,
                                const int64_t* row_ptr, const int64_t* source, int64_t n_nodes, int64_t n_edges, int D,
                                int F, int orders, int A0, int W, int dtype, void* dv, void* drc, void* dcc, void* stream) {
  int status = check_conv(v, rc, cc, transport, angular, rho, weights, desc, row_ptr, source, n_nodes, n_edges, D, F, orders, A0, W, dtype);
  if (status != GM_OK || n_nodes == 0 || n_edges == 0) return status;
  GM_REQUIRE(g && dv, GM_ERR_ARGUMENT, "gm_conv_backward: null g / dv");
  GM_REQUIRE((A0 == 0 || drc) && (W == 0 || dcc), GM_ERR_ARGUMENT, "gm_conv_backward: null coefficient gradient");
  auto run = [&](auto tag) {
    using T = decltype(tag);
    auto a = conv_args<T>(v, rc, cc, transport, angular, rho, weights, desc, row_ptr, source, n_nodes, D, F, orders, A0, W);
    a.g = (const T*)g; a.dv = (T*)dv; a.drc = (T*)drc; a.dcc = (T*)dcc;
    conv_kernel<T, true><<<conv_grid(n_nodes), CONV_THREADS, D * sizeof(ConvItem), (cudaStream_t)stream>>>(a);
    return launch_status("gm_conv_backward");
  };
  return dtype == GM_F32 ? run(float()) : run(double());
}
