// Device helpers shared by the PCG kernels of the tile path (solver.cu) and
// its one-launch form (pcg_grid.cu): reductions in a fixed order, contact
// rows and the scalar recurrences.
#pragma once
#include <cfloat>

#include "kernels.cuh"

namespace hobak {

// Fixed-order sum over the CTA; result valid in thread 0.  NT multiple of 32.
// The whole tree runs in R (FP32 for the inner solve of the mixed path) and
// only the CTA's total is widened to FP64: a conversion per warp costs a
// 16-cycle issue on GB300's 2-lane FP64 pipe even when one lane uses it.
template <int NT, typename R>
__device__ __forceinline__ double block_sum(R v, double* sh) {
  R* shr = reinterpret_cast<R*>(sh);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x / 32, l = threadIdx.x % 32;
  if (l == 0) shr[w] = v;
  __syncthreads();
  double s = 0;
  if (threadIdx.x == 0) {
    R t = R(0);
#pragma unroll
    for (int i = 0; i < NT / 32; i++) t += shr[i];
    s = double(t);
  }
  __syncthreads();
  return s;
}

// Three sums in one pass (one pair of barriers), each in the order of
// block_sum; results valid in thread 0.  `sh` holds 3 * NT / 32 doubles.
template <int NT, typename R>
__device__ __forceinline__ void block_sum3(R a, R b, R c, double* sh, double (&out)[3]) {
  R* shr = reinterpret_cast<R*>(sh);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  const int w = threadIdx.x / 32, l = threadIdx.x % 32;
  if (l == 0) {
    shr[w] = a;
    shr[NT / 32 + w] = b;
    shr[2 * (NT / 32) + w] = c;
  }
  __syncthreads();
  out[0] = out[1] = out[2] = 0.0;
  if (threadIdx.x == 0) {
    R ta = R(0), tb = R(0), tc = R(0);
#pragma unroll
    for (int i = 0; i < NT / 32; i++) {
      ta += shr[i];
      tb += shr[NT / 32 + i];
      tc += shr[2 * (NT / 32) + i];
    }
    out[0] = double(ta);
    out[1] = double(tb);
    out[2] = double(tc);
  }
  __syncthreads();
}

// After thread 0 wrote the CTA's partial(s): true in the CTA that finishes
// the scene's reduction (ticket == ntiles - 1).  Only thread 0 published
// anything the last CTA reads, so only it fences before taking its ticket.
// The ticket is reset for reuse.
__device__ __forceinline__ bool last_tile(unsigned* ticket, int ntiles, int* flag) {
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned t = atomicAdd(ticket, 1u);
    *flag = (t == (unsigned)(ntiles - 1));
    if (*flag) *ticket = 0u;
  }
  __syncthreads();
  const bool last = *flag != 0;
  if (last) __threadfence();
  return last;
}

// Sum partial[(tile0 + i) * kPartials + comp] over i < n in a fixed order.
template <int NT>
__device__ __forceinline__ double sum_partials(const double* partial, int tile0, int n, int comp, double* sh) {
  double s = 0;
  for (int i = threadIdx.x; i < n; i += NT) s += __ldcg(&partial[(size_t)(tile0 + i) * kPartials + comp]);
  return block_sum<NT>(s, sh);
}

// Order of the PCG's three dot products, the same on every path so that all
// give the same bits.  An FP64 add costs 19 cycles of the SM's pipe per warp
// instruction however few of its lanes work, and 64 cycles of latency, so the
// trees below fill their lanes, and sums run in short chains on several warps.
//   FP32  tile: a tree per warp, the warps in order (block_sum3); group:
//         kGroupVerts / TV consecutive tiles of the scene, added pairwise in
//         FP64; scene: lane l adds groups l, l + 32, ..., then a warp tree
//   FP64  tile: its 3 TV row products, a tree over every 32, the trees in
//         order; scene: lane l of 3 TV adds tiles l, l + 3 TV, ..., then as a tile
constexpr int kGroupVerts = 512;

__device__ __forceinline__ double warp_tree(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums of groups g0 .. g0 + 7 (those below n) of 32 values each, get(g, l)
// value l of group g, by the pairs of an xor-shuffle tree (16, 8, 4, 2, 1), to
// out[g].  One warp, which halves its number of values per lane with every
// exchange: 9 adds where eight shuffle trees issue 40.
template <typename Get>
__device__ __forceinline__ void tree32_warp(int g0, int n, Get get, double* out) {
  const int lane = threadIdx.x % 32, l = lane & 15, hi = lane >> 4;
  const bool b3 = lane & 8, b2 = lane & 4;
  double a[4];  // lanes 0..15: group g0 + 2 j, lanes 16..31: g0 + 2 j + 1
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int g = g0 + 2 * j + hi;
    a[j] = g < n ? get(g, l) + get(g, l + 16) : 0.0;
  }
  double c[2];
#pragma unroll
  for (int m = 0; m < 2; m++)
    c[m] = (b3 ? a[2 * m + 1] : a[2 * m]) + __shfl_xor_sync(0xffffffffu, b3 ? a[2 * m] : a[2 * m + 1], 8);
  double d = (b2 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, b2 ? c[0] : c[1], 4);
  d += __shfl_xor_sync(0xffffffffu, d, 2);
  d += __shfl_xor_sync(0xffffffffu, d, 1);
  const int g = g0 + 4 * (b2 ? 1 : 0) + 2 * (b3 ? 1 : 0) + hi;
  if ((lane & 3) == 0 && g < n) out[g] = d;
}
// ... of all n groups by the CTA's warps
template <typename Get>
__device__ __forceinline__ void tree32(int n, Get get, double* out) {
#pragma unroll 1
  for (int g0 = 8 * (threadIdx.x / 32); g0 < n; g0 += 8 * (blockDim.x / 32)) tree32_warp(g0, n, get, out);
}

// Sum of n values in order, each loaded ahead of the add before it.
__device__ __forceinline__ double chain(const double* v, int n) {
  double t = v[0], next = n > 1 ? v[1] : 0.0;
#pragma unroll 1
  for (int i = 1; i < n; i++) {
    const double x = next;
    if (i + 1 < n) next = v[i + 1];
    t += x;
  }
  return t;
}

// FP64: the trees of a scene's three sums over its n tiles' partials,
// tile(c, i), to out[trees * c + ...]; trees = scene_trees(n): those with a tile
// in their lanes (the others are zero).
template <int TV>
__device__ __forceinline__ int scene_trees(int n) {
  return n < 3 * TV ? (n + 31) / 32 : 3 * TV / 32;
}
// lanes: 9 TV doubles of shared memory.  All threads of the CTA.
template <int TV, typename Tile>
__device__ __forceinline__ void scene_tree32(int n, Tile tile, double* lanes, double* out) {
  const int trees = scene_trees<TV>(n), width = 32 * trees;
#pragma unroll 1
  for (int k = threadIdx.x; k < 3 * width; k += blockDim.x) {
    const int c = k >= 2 * width ? 2 : k >= width ? 1 : 0, l = k - c * width;
    double s = l < n ? tile(c, l) : 0.0;
#pragma unroll 1
    for (int i = l + 3 * TV; i < n; i += 3 * TV) s += tile(c, i);
    lanes[k] = s;
  }
  __syncthreads();
  tree32(3 * trees, [&](int g, int l) { return lanes[32 * g + l]; }, out);
}

// The sum of a group's tiles, get(i) its i-th (0 past the scene's last tile).
template <int TV, typename Get>
__device__ __forceinline__ double group_sum(Get get) {
  double a = (get(0) + get(1)) + (get(2) + get(3));
  if (kGroupVerts / TV == 4) return a;
  return a + ((get(4) + get(5)) + (get(6) + get(7)));
}

// A scene's sum by one warp: group(g) for its n groups.
template <typename Group>
__device__ __forceinline__ double scene_sum(int n, Group group) {
  double s = 0.0;
#pragma unroll 1
  for (int g = threadIdx.x % 32; g < n; g += 32) s += group(g);
  return warp_tree(s);
}

// FP32: the three scene sums from the tiles' partials, [component][stride], in
// scene_sum's order.  True in the CTA that ends them, with the sums in thread 0.
// The iteration waits for them, so the last CTA of a scene adds all groups only up
// to kOneCta of them.  Past that they lie in segments of 32: the last CTA of a
// segment forms its groups' sums, a lane each, and the last of the segments adds
// those (one more ticket: 1.7 us where one CTA is soon done).  Steps of 400
// iterations, one CTA / segments: tiles of 128 (three warps), 59,319 vertices (116
// groups) 6.85 / 7.44 ms; tiles of 64 (two warps) 9.1 / 7.7 ms, 17,576 (35 groups)
// 5.1 / 5.7 ms.  With one CTA and a lane's groups one after the other k_spmv of 52^3
// took 23.3 us (18.7 as here), of 72^3 (760 groups) 65 (55; tiles of 64 83 and 59).
// tickets: one per tile, zero (a segment takes its first tile's).
template <int NT, int TV>
__device__ __forceinline__ bool scene_sums(const double* partial, double* groupSums, int stride, unsigned* tickets,
                                           unsigned* sceneTicket, const SceneParams& sp, int tile, int* flag,
                                           double* sh, double (&out)[3]) {
  constexpr int kG = kGroupVerts / TV, kWarps = NT / 32;
  constexpr int kOneCta = TV == 128 ? 512 : 64;
  const int tile0 = sp.tile0, n = sp.ntiles, ng = (n + kG - 1) / kG;
  const bool one = ng <= kOneCta;
  const int g0 = one ? 0 : (tile - tile0) / (32 * kG) * 32, g1 = one ? ng : min(ng, g0 + 32);
  // a warp's component, and with two warps the first one's second: both in flight
  const int c = threadIdx.x / 32, lane = threadIdx.x % 32;
  const bool mine = c < 3, two = kWarps < 3 && c + kWarps < 3;
  if (!last_tile(one ? sceneTicket : &tickets[tile0 + g0 * kG], min(n, g1 * kG) - g0 * kG, flag)) return false;
  auto group = [&](int comp, int g) {
    const double* q = partial + (size_t)comp * stride + tile0;
    return group_sum<TV>([&](int i) { return g * kG + i < n ? __ldcg(&q[g * kG + i]) : 0.0; });
  };
  double a = 0.0, b = 0.0;
  if (one) {
    if (mine)
#pragma unroll 4
      for (int g = lane; g < ng; g += 32) {
        a += group(c, g);
        if (two) b += group(c + kWarps, g);
      }
  } else {
    double* sums = groupSums + (size_t)c * stride + tile0;
    if (mine) a = group(c, g0 + lane);
    if (two) b = group(c + kWarps, g0 + lane);
    if (mine) sums[g0 + lane] = a;
    if (two) sums[(size_t)kWarps * stride + g0 + lane] = b;
    __syncthreads();  // last_tile's fence by thread 0 covers the writers
    if (!last_tile(sceneTicket, (ng + 31) / 32, flag)) return false;
    a = b = 0.0;
    if (mine)
#pragma unroll 8
      for (int g = lane; g < ng; g += 32) {
        a += __ldcg(&sums[g]);
        if (two) b += __ldcg(&sums[(size_t)kWarps * stride + g]);
      }
  }
  a = warp_tree(a);
  if (kWarps < 3) b = warp_tree(b);
  if (mine && lane == 0) sh[c] = a;
  if (two && lane == 0) sh[c + kWarps] = b;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 3; k++) out[k] = sh[k];
  return true;
}

__device__ __forceinline__ bool finite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// a / b, correctly rounded, from y = 1 / b correctly rounded (0: not given): a
// quotient off by at most a few ulps and Markstein's correction ("Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990), a
// chain of three FMAs (200 cycles in one thread) where the division takes
// ~630.  Outside the range where the residual is exact, the division.
__device__ __forceinline__ double divide(double a, double b, double y) {
  const auto plain = [](double x) {
    const int e = (__double2hiint(x) >> 20) & 0x7ff;
    return e > 523 && e < 1523;
  };
  if (!(plain(a) && plain(b) && plain(y))) return a / b;
  const double q = a * y;
  return fma(fma(-q, b, a), y, q);
}

// A scene's iteration step (one thread), from
// rho = |r|^2, gamma = (r, u) and delta = (w, u): after an update, stop when
// |r|^2 < threshold (ConjugateGradient.h:75-78), on a non-finite value, or at
// the iteration limit; otherwise beta and alpha for this iteration's update,
// which the iteration count then includes.  Returns true when it stops.
// gammaInv, alphaInv: 1 / st.gamma and 1 / st.alpha where the caller has them.
template <typename T>
__device__ __forceinline__ bool pcg_decide(SolveState& st, double rho, double gamma, double delta,
                                           double gammaInv = 0.0, double alphaInv = 0.0) {
  if (st.iters > 0) {
    st.rr = rho;
    bool stop = false;
    if (rho < st.innerThreshold) {
      stop = true;
    } else if (!finite(rho) || !finite(gamma) || !finite(st.alpha)) {
      stop = true;
      st.converged = -1;
      st.outerDone = 1;
    } else if (st.totalIters >= st.maxit) {
      stop = true;
    }
    if (stop) {
      st.done = 1;
      if (sizeof(T) == sizeof(double) && st.converged >= 0) {
        // FP64 path: the recursive residual is the solver's verdict (Eigen)
        st.rr64 = rho;
        st.converged = rho < st.threshold ? 1 : 0;
        st.outerDone = 1;
      }
      return true;
    }
  }
  st.delta = delta;
  if (st.iters == 0) {
    st.beta = 0.0;
    st.alpha = gamma / delta;
  } else {
    const double beta = divide(gamma, st.gamma, gammaInv);  // st.gamma: the previous iteration's (r, u)
    st.beta = beta;
    st.alpha = gamma / (delta - divide(beta * gamma, st.alpha, alphaInv));
  }
  st.gammaOld = st.gamma;
  st.gamma = gamma;
  if (sizeof(T) == sizeof(float)) {
    st.alphaF = float(st.alpha);
    st.betaF = float(st.beta);
  }
  st.iters += 1;
  st.totalIters += 1;
  return false;
}

// u of a vertex as the one-launch PCG shares it, four wide: in FP32 with the
// iteration it belongs to in the fourth word, written at once, so that a
// reader knows by the value itself whether it is the one it needs.
__device__ __forceinline__ void publish_u(float* u4, int w, const float (&x)[3], int iteration) {
  const unsigned long long lo = (unsigned long long)__float_as_uint(x[1]) << 32 | __float_as_uint(x[0]);
  const unsigned long long hi = (unsigned long long)(unsigned)iteration << 32 | __float_as_uint(x[2]);
  asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(u4 + 4 * (size_t)w),
               "l"(lo), "l"(hi)
               : "memory");
}
__device__ __forceinline__ void publish_u(double* u4, int w, const double (&x)[3], int) {
  __stcg(reinterpret_cast<double2*>(u4) + 2 * (size_t)w, make_double2(x[0], x[1]));
  __stcg(u4 + 4 * (size_t)w + 2, x[2]);
}

// Words of the one-launch PCGs: a value and the tag it belongs to, written and
// read at once.
__device__ __forceinline__ void st_word(ulonglong2* p, double value, unsigned long long tag) {
  asm volatile(
      "{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(p),
      "l"(__double_as_longlong(value)), "l"(tag)
      : "memory");
}
__device__ __forceinline__ void ld_word(const ulonglong2* p, double& value, unsigned long long& tag) {
  unsigned long long bits;
  asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
               : "=l"(bits), "=l"(tag)
               : "l"(p)
               : "memory");
  value = __longlong_as_double((long long)bits);
}

// N words whose tags must all be `tag`: use(k) says which of them, at(k) where.
// All are loaded at once, and those not there yet again at once, so a wait costs
// the latency of the last one and not of each.  Clears ok when one is not there
// after `limit` polls.
template <int N, typename Use, typename At>
__device__ __forceinline__ void ld_words(Use use, At at, unsigned long long tag, int limit, double (&value)[N], bool& ok) {
  unsigned long long got[N];
#pragma unroll
  for (int k = 0; k < N; k++)
    if (use(k)) ld_word(at(k), value[k], got[k]);
#pragma unroll 1
  for (int n = 0; ok; n++) {
    bool missing = false;
#pragma unroll
    for (int k = 0; k < N; k++)
      if (use(k) && got[k] != tag) missing = true;
    if (!missing) break;
    if (n >= limit) ok = false;
#pragma unroll
    for (int k = 0; k < N; k++)
      if (use(k) && got[k] != tag) ld_word(at(k), value[k], got[k]);
  }
}

// a . b of two 3-vectors, as the compiler contracts a0 b0 + a1 b1 + a2 b2
template <typename T>
__device__ __forceinline__ T dot3v(T a0, T a1, T a2, T b0, T b1, T b2) {
  return a0 * b0 + a1 * b1 + a2 * b2;
}

// Contact: w H_coll x at a vertex (w = collision_lhs_scale), H_coll = sum over
// its collision tets of (c c^T) (x) G (free rows only; x vanishes on pinned
// rows, which keeps the columns masked too).  FP64 throughout: the contact
// blocks are not part of the (possibly FP32) assembled LHS.  One incidence:
// t = G sum_q c_q x_q, and the weight c_a of the vertex's own row; load(id, x)
// reads the vector at a vertex.
template <typename T, typename Load>
__device__ __forceinline__ double collision_incidence(const DeviceCollisions& c, int k, Load load, double (&t)[3]) {
  const int e = c.incList[k], p = e >> 2;
  const int4 ct = c.pairTet[p];
  const double* C = c.pairC + 4 * (size_t)p;
  const double* G = c.pairG + 9 * (size_t)p;
  const int id[4] = {ct.x, ct.y, ct.z, ct.w};
  T x[4][3];
#pragma unroll
  for (int q = 0; q < 4; q++) load(id[q], x[q]);
  double z[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int j = 0; j < 3; j++) z[j] += C[q] * double(x[q][j]);
#pragma unroll
  for (int i = 0; i < 3; i++) t[i] = G[i] * z[0] + G[i + 3] * z[1] + G[i + 6] * z[2];
  return C[e & 3];
}

// A vertex's rows, its incidences in order.
template <typename T, typename Load>
__device__ __forceinline__ void collision_rows(const DeviceBatch& b, int u, Load load, double (&out)[3]) {
  const DeviceCollisions& c = b.coll;
  const int k0 = c.incCount[u], k1 = c.incCount[u + 1];
  out[0] = out[1] = out[2] = 0.0;
  if (k0 == k1) return;
#pragma unroll 1
  for (int k = k0; k < k1; k++) {
    double t[3];
    const double w = collision_incidence<T>(c, k, load, t);
#pragma unroll
    for (int i = 0; i < 3; i++) out[i] = fma(w, t[i], out[i]);
  }
  const double scale = collision_lhs_scale(b, b.vertexScene[u]);
#pragma unroll
  for (int i = 0; i < 3; i++) out[i] = __dmul_rn(out[i], scale);
}

}  // namespace hobak
