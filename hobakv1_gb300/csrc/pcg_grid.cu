// The tile path's inner PCG in one cooperative launch.
//
// solver.cu runs an iteration as two grid-wide kernels (SpMV, update).  For a
// batch whose tiles fit the GPU at once that spends most of an iteration on
// the kernels' edges: launch, a cold walk tile -> row -> column -> u, the
// matrix again from L2, two reductions' tails.  Here one launch runs every
// iteration of the solve: a CTA per SM owns up to 512 vertices (whole tiles of
// one scene) for the whole solve, one per thread.  A vertex's u, p, s, d, r
// stay in registers; the first blocks of its matrix row and their columns in
// shared memory (as many as fit, the same count for every row), in FP32 the
// next six in registers; the rest of the row comes from L2.  Per iteration the CTAs of a scene meet twice:
//   * the partial sums of the three dot products go out as 16-byte words
//     {value, iteration}, |r|^2 and (r, u) before the SpMV, (w, u) after it, written and polled with
//     single-copy-atomic 128-bit accesses, so a reader needs no flag and no
//     fence; every CTA adds them in the same order and takes the same decision;
//   * after the update the new u: in FP32 the same way, each vertex's u carries
//     its iteration; a CTA reads its halo (the other CTAs' vertices in its
//     rows' columns, listed once) into shared memory, each vertex once and
//     not up to 15 times, and a load repeats until the iteration fits; in FP64 (two words a
//     vertex) a CTA releases a flag, and a CTA waits for the flags of the CTAs
//     its rows' columns lie in (with contact: all of the scene's).
// The partials' exchange also orders u's reuse: a CTA overwrites its u only
// after every CTA of the scene has published the partials of the SpMV that
// read it.  Partials alternate between two buffers for the same reason.
// Row, tile and scene sums are formed as in solver.cu (pcg_common.cuh), so
// both give the same bits and a scene's result does not depend on the batch.
//
// What bounds it: in FP64 the SM's FP64 pipe, 19 cycles per warp instruction
// (16 warps x 135 products of 512 vertices' rows are 39,000 of an iteration's
// 64,000 cycles); in FP32 latency: the row sums from shared memory are 4,600 of
// 16,200 cycles, the halo 1,700, the partials' exchange 2,100, the scalars
// 3,600.  The phases between barriers run once an iteration on few warps, so
// loops there are kept rolled: 108 KB of code cost 4,000 cycles more an
// iteration in instruction fetches than 53 KB.  68,921 vertices, us an
// iteration: FP64 45.8 -> 31.3 (365 iterations: step 19.9 -> 13.7 ms), FP32
// 17.0 -> 7.9 (383: 7.2 -> 3.8 ms); two cubes in contact, 31,250 vertices,
// FP64 56 -> 25; 1,331 vertices FP64 23 -> 15.
//
// Every wait is bounded; a wait that runs out ends the CTA's part, and the
// scene's solve is marked failed.  All CTAs are resident (cooperative launch,
// at most one per SM), so no CTA waits for one that cannot run.
#include <algorithm>

#include "pcg_common.cuh"

namespace hobak {

namespace {

constexpr int kGridThreads = 512;      // vertices of a CTA, at most (128 registers each)
constexpr int kGridSmemMax = 224 * 1024;
constexpr int kMaxCtas = kGridCtas;
constexpr int kHaloMax = 3072;         // halo vertices of a CTA, at most (48 KB of shared memory)

__device__ __forceinline__ int ld_flag(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_flag(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The u of a vertex for iteration `it`, from L2: other SMs write it.
struct Gather32 {
  unsigned long long lo, hi;
  __device__ __forceinline__ void load(const float* u4, int w) {
    asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }"
                 : "=l"(lo), "=l"(hi)
                 : "l"(u4 + 4 * (size_t)w)
                 : "memory");
  }
  // repeats the load of vertex() until it fits; clears ok when it does not
  template <typename Vertex>
  __device__ __forceinline__ void get(const float* u4, Vertex vertex, int it, int limit, float (&x)[3], bool& ok) {
#pragma unroll 1
    for (int n = 0; (int)(hi >> 32) != it && ok; n++) {
      if (n >= limit) ok = false;
      load(u4, vertex());
    }
    x[0] = __uint_as_float((unsigned)lo);
    x[1] = __uint_as_float((unsigned)(lo >> 32));
    x[2] = __uint_as_float((unsigned)hi);
  }
};
struct Gather64 {  // the caller has waited for the owner's flag
  double2 a;
  double z;
  __device__ __forceinline__ void load(const double* u4, int w) {
    a = __ldcg(reinterpret_cast<const double2*>(u4) + 2 * (size_t)w);
    z = __ldcg(u4 + 4 * (size_t)w + 2);
  }
  template <typename Vertex>
  __device__ __forceinline__ void get(const double*, Vertex, int, int, double (&x)[3], bool&) {
    x[0] = a.x, x[1] = a.y, x[2] = z;
  }
};
template <typename T>
struct GatherOf {
  using type = Gather64;
};
template <>
struct GatherOf<float> {
  using type = Gather32;
};

// One block times x into the row sums, in solver.cu's order: FP32 one nested
// chain per row; FP64 two chains per row, even and odd blocks.
template <typename T>
struct RowSums {
  T a[sizeof(T) == 4 ? 3 : 6];
  __device__ __forceinline__ RowSums() {
#pragma unroll
    for (T& v : a) v = T(0);
  }
  __device__ __forceinline__ void add(const T (&m)[9], const T (&x)[3], bool odd) {
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int i = 0; i < 3; i++) a[i] = fma(m[3 * i], x[0], fma(m[3 * i + 1], x[1], fma(m[3 * i + 2], x[2], a[i])));
    } else {
#pragma unroll
      for (int i = 0; i < 3; i++) {
        T& c = odd ? a[3 + i] : a[i];
        c = fma(m[3 * i], x[0], c);
        c = fma(m[3 * i + 1], x[1], c);
        c = fma(m[3 * i + 2], x[2], c);
      }
    }
  }
  __device__ __forceinline__ void total(T (&w)[3]) const {
#pragma unroll
    for (int i = 0; i < 3; i++)
      if constexpr (sizeof(T) == 4) w[i] = a[i];
      else w[i] = a[i] + a[3 + i];
  }
};

// ctas: per CTA its scene and the scene's tile it starts at.  tpc: tiles per
// CTA.  rows: blocks of every row kept in shared memory (even in FP64).
// scratch: doubles of the exchange area.
template <int TV, typename T>
__global__ void __launch_bounds__(kGridThreads, 1)
    k_pcg_grid(DeviceBatch b, PcgVecs<T> v, const int2* __restrict__ ctas, int tpc, int rows, int scratch, int halo) {
  constexpr bool kF32 = sizeof(T) == sizeof(float);
  constexpr int kTail = 6;  // FP32: row blocks past the shared ones, in registers
  constexpr int kQ = 2;     // FP64: blocks per trip
  constexpr int kG = kGroupVerts / TV;
  using Gather = typename GatherOf<T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SolveState ss;
  __shared__ T warpSum[3][kGridThreads / 32];
  __shared__ double sums[3], recip[2];              // recip: of the last gamma and alpha
  __shared__ double trees[9 * kGridThreads / 32];  // FP64: sums of 32 rows or tiles
  __shared__ unsigned nbrBits[kMaxCtas / 32];
  __shared__ int nbr[kMaxCtas];
  __shared__ int nNbr, stop;
  __shared__ T sAlpha, sBeta;

  const int tid = threadIdx.x, NT = blockDim.x;
  const int2 cta = ctas[blockIdx.x];
  const int s = cta.x;
  const SceneParams& sp = b.scenes[s];
  SolveState& st = b.solve[s];
  if (st.done) return;  // converged at its start, parked or failed (every CTA of the scene alike)
  const int ntiles = sp.ntiles, v0 = sp.v0;
  const int slot = cta.y + tid / TV;  // the thread's tile of the scene
  const int u = slot < ntiles ? b.tileV0[sp.tile0 + slot] + tid % TV : v0;
  const bool valid = slot < ntiles && u < b.tileV1[sp.tile0 + slot];
  const int own = valid ? u : v0;  // a vertex that any gather may read

  double* area = reinterpret_cast<double*>(smem);
  float4* us = reinterpret_cast<float4*>(area + scratch);  // FP32: u of the CTA's and of its halo's vertices
  T* mat = reinterpret_cast<T*>(us + (kF32 ? NT + halo : 0));
  int* col = reinterpret_cast<int*>(mat + (size_t)9 * rows * NT);  // both [entry][thread]

  if (tid == 0) {
    ss = st;
    nNbr = 0;
    stop = 0;
  }
  if (tid < kMaxCtas / 32) nbrBits[tid] = 0u;
  __syncthreads();

  // ---- the row's blocks and columns; the vertex's vectors (p = s = d = 0) ----
  const int nCta = (ntiles + tpc - 1) / tpc, ctaVerts = tpc * TV;
  T* u4 = v.p;  // p and s live in registers here: their buffers hold the shared u
  int len = 0;
  size_t lb = 0, cb = 0;
  const int* cols = kF32 ? b.clusterGather : b.colS;  // FP32: indices into us
  const int self = kF32 ? tid : own;
  T un[3], p[3], sv[3], d[3], r[3];
#pragma unroll
  for (int i = 0; i < 3; i++) un[i] = p[i] = sv[i] = d[i] = r[i] = T(0);
  if (valid) {
    const T* rsrc = kF32 ? v.r : reinterpret_cast<const T*>(b.r64);
    len = b.rowptr[u + 1] - b.rowptr[u];
    lb = lhs_slot(b, u, 0);
    cb = col_slot(b, u, 0);
    if (!kF32)
#pragma unroll 1
      for (int j = 0; j < len; j++) {
        const int c = (__ldg(&b.colS[cb + kSlice * j]) - v0) / ctaVerts;
        if (!((nbrBits[c / 32] >> (c % 32)) & 1u)) atomicOr(&nbrBits[c / 32], 1u << (c % 32));
      }
#pragma unroll
    for (int i = 0; i < 3; i++) {
      un[i] = v.u[3 * u + i];
      r[i] = rsrc[3 * u + i];
    }
  }
#pragma unroll 1
  for (int j = 0; j < rows; j++) {  // zeros past the row's end
    col[(size_t)j * NT + tid] = j < len ? __ldg(&cols[cb + kSlice * j]) : self;
#pragma unroll
    for (int e = 0; e < 9; e++)
      mat[((size_t)9 * j + e) * NT + tid] = j < len ? __ldg(&v.lhs[lb + (size_t)kSlotVals * j + kSlice * e]) : T(0);
  }
  int tailCol[kTail];
  T tail[kF32 ? kTail : 1][9];  // FP32: the row's next blocks stay in registers
  if constexpr (kF32)
#pragma unroll
    for (int q = 0; q < kTail; q++) {
      tailCol[q] = rows + q < len ? __ldg(&cols[cb + kSlice * (rows + q)]) : self;
#pragma unroll
      for (int e = 0; e < 9; e++)
        tail[q][e] = rows + q < len ? __ldg(&v.lhs[lb + (size_t)kSlotVals * (rows + q) + kSlice * e]) : T(0);
    }
  __syncthreads();
  if (!kF32)
#pragma unroll 1
    for (int c = tid; c < nCta; c += NT)
      if ((b.collOn || ((nbrBits[c / 32] >> (c % 32)) & 1u)) && c != cta.y / tpc) nbr[atomicAdd(&nNbr, 1)] = c;
  // the CTA's contact incidences (CSR by vertex, its vertices are consecutive)
  int inc0 = 0, inc1 = 0, my0 = 0, my1 = 0;
  double collScale = 0.0;
  if (b.collOn) {
    const int last = min(ntiles, cta.y + tpc) - 1;
    inc0 = b.coll.incCount[b.tileV0[sp.tile0 + cta.y]];
    inc1 = b.coll.incCount[b.tileV1[sp.tile0 + last]];
    if (valid && b.freeMask[u]) {
      my0 = b.coll.incCount[u];
      my1 = b.coll.incCount[u + 1];
    }
    if (inc1 > inc0) collScale = collision_lhs_scale(b, s);
  }
  const int lenMax = __reduce_max_sync(0xffffffffu, len);
  __syncthreads();
  int* flags = b.gridFlags + sp.tile0;  // a CTA's flag: that of its first tile
  const int* haloList = halo_list(b, s, b.tileV0[sp.tile0 + cta.y]);
  const int nHalo = kF32 ? b.gridHaloCount[sp.tile0 + cta.y] : 0;
  if constexpr (kF32) us[tid] = make_float4(un[0], un[1], un[2], 0.f);
  const bool whole = kF32 && tpc == kG;  // partials: one per group, else one per tile
  const int nGroups = (ntiles + kG - 1) / kG, nParts = whole ? nGroups : ntiles;
  constexpr int kTrees = 3 * TV / 32;  // FP64: trees of a tile's rows
  auto words = [&](int it) {
    return reinterpret_cast<ulonglong2*>(b.gridPartials) + 3 * ((it & 1) * (size_t)b.gridTilesCap + sp.tile0);
  };
  // FP32: warp sums (one value each in warpSum[c]) -> tile or group sums of
  // component c0 .. c0 + n - 1, published for iteration it
  auto publish32 = [&](int c0, int n, int it) {
    auto tile = [&](int t, int c) {  // block_sum3's order over the tile's warps
      T a = T(0);
#pragma unroll
      for (int i = 0; i < TV / 32; i++) a += warpSum[c][t * (TV / 32) + i];
      return double(a);
    };
    if (whole && tid < n)
      st_word(words(it) + 3 * (cta.y / kG) + c0 + tid, group_sum<TV>([&](int t) { return tile(t, c0 + tid); }), it);
    else if (!whole && tid < n * tpc && cta.y + tid % tpc < ntiles)
      st_word(words(it) + 3 * (cta.y + tid % tpc) + c0 + tid / tpc, tile(tid % tpc, c0 + tid / tpc), it);
  };
  // FP64: row products in area[c][tile][row] -> the same
  auto publish64 = [&](int c0, int n, int it) {
    double* t = trees + c0 * tpc * kTrees;
    tree32(n * tpc * kTrees, [&](int g, int l) { return area[3 * c0 * NT + 32 * g + l]; }, t);
    __syncthreads();
    if (tid < n * tpc && cta.y + tid % tpc < ntiles)
      st_word(words(it) + 3 * (cta.y + tid % tpc) + c0 + tid / tpc, chain(t + tid * kTrees, kTrees), it);
  };
  // |r|^2 and (r, u) of iteration it, known as soon as its u is: ahead of the SpMV
  auto publish_ru = [&](int it) {
    if constexpr (kF32) {
      T t0 = T(0), t1 = T(0);
      if (valid) {
        t1 = dot3v(r[0], r[1], r[2], un[0], un[1], un[2]);
        t0 = dot3v(r[0], r[1], r[2], r[0], r[1], r[2]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        t0 += __shfl_xor_sync(0xffffffffu, t0, o);
        t1 += __shfl_xor_sync(0xffffffffu, t1, o);
      }
      if (tid % 32 == 0) {
        warpSum[0][tid / 32] = t0;
        warpSum[1][tid / 32] = t1;
      }
      __syncthreads();
      publish32(0, 2, it);
    } else {
#pragma unroll
      for (int i = 0; i < 3; i++) {
        area[3 * tid + i] = valid ? r[i] * r[i] : 0.0;
        area[3 * NT + 3 * tid + i] = valid ? r[i] * un[i] : 0.0;
      }
      __syncthreads();
      publish64(0, 2, it);
    }
  };
  bool ok = true;  // this thread's waits
  int failed = 0;  // some thread's wait ran out (the same in all threads)
  T alpha = T(0);

#pragma unroll 1
  for (int it = 1;; it++) {
    publish_ru(it);
    auto reciprocals = [&] {
      if (it > 1 && tid >= NT - 2) recip[NT - 1 - tid] = 1.0 / (tid == NT - 1 ? ss.gamma : ss.alpha);
    };
    RowSums<T> acc;
    if constexpr (kF32) {
      // the halo's u to shared memory, four loads in flight
#pragma unroll 1
      for (int i0 = tid; i0 < nHalo; i0 += 4 * NT) {
        Gather g[4];
        int w[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (i0 + k * NT < nHalo) g[k].load(u4, w[k] = __ldg(&haloList[i0 + k * NT]));
#pragma unroll
        for (int k = 0; k < 4; k++) {
          if (i0 + k * NT >= nHalo) break;
          T x[3];
          g[k].get(u4, [&] { return w[k]; }, it, b.waitPolls, x, ok);
          us[NT + i0 + k * NT] = make_float4(x[0], x[1], x[2], 0.f);
        }
      }
      reciprocals();
      if ((failed = __syncthreads_or(!ok))) break;
      auto vec = [&](int c, float (&x)[3]) {
        const float4 t = us[c];
        x[0] = t.x, x[1] = t.y, x[2] = t.z;
      };
      const int nsm = min(lenMax, rows);
#pragma unroll 3
      for (int j = 0; j < nsm; j++) {
        T x[3], m[9];
        vec(col[(size_t)j * NT + tid], x);
#pragma unroll
        for (int e = 0; e < 9; e++) m[e] = mat[((size_t)9 * j + e) * NT + tid];
        acc.add(m, x, false);
      }
      if (lenMax > rows) {
#pragma unroll
        for (int q = 0; q < kTail; q++) {
          T x[3];
          vec(tailCol[q], x);
          acc.add(tail[q], x, false);
        }
#pragma unroll 1
        for (int j = rows + kTail; j < len; j++) {  // rows longer than the mesh's usual
          T m[9], x[3];
#pragma unroll
          for (int e = 0; e < 9; e++) m[e] = __ldg(&v.lhs[lb + (size_t)kSlotVals * j + kSlice * e]);
          vec(__ldg(&cols[cb + kSlice * j]), x);
          acc.add(m, x, false);
        }
      }
    } else {
      reciprocals();
#pragma unroll 1
      for (int i = tid; i < nNbr; i += NT) {
        const int* f = flags + nbr[i] * tpc;
        int n = 0;
#pragma unroll 1
        while (ld_flag(f) < it && ok)
          if (n++ >= b.waitPolls) ok = false;
      }
      if ((failed = __syncthreads_or(!ok))) break;
      // Two blocks per trip (the chains of even and odd blocks), the next
      // trip's u ahead of this trip's products.  FP64-pipe bound: the bounds
      // are the warp's, so that no product is issued for nobody.
      Gather g[kQ];
      auto gather = [&](int j) {
#pragma unroll
        for (int q = 0; q < kQ; q++) {
          const int w = j + q < rows  ? col[(size_t)(j + q) * NT + tid]
                        : j + q < len ? __ldg(&b.colS[cb + kSlice * (j + q)])
                                      : own;
          g[q].load(u4, w);
        }
      };
      gather(0);
#pragma unroll 1
      for (int j = 0; j < lenMax; j += kQ) {
        T m[kQ][9], x[kQ][3];
        if (j < rows) {
#pragma unroll
          for (int q = 0; q < kQ; q++)
#pragma unroll
            for (int e = 0; e < 9; e++) m[q][e] = mat[((size_t)9 * (j + q) + e) * NT + tid];
        } else {
#pragma unroll
          for (int q = 0; q < kQ; q++)
#pragma unroll
            for (int e = 0; e < 9; e++)
              m[q][e] = j + q < len ? __ldg(&v.lhs[lb + (size_t)kSlotVals * (j + q) + kSlice * e]) : T(0);
        }
#pragma unroll
        for (int q = 0; q < kQ; q++) g[q].get(u4, [] { return 0; }, it, b.waitPolls, x[q], ok);
        if (j + kQ < lenMax) gather(j + kQ);
        acc.add(m[0], x[0], false);
        if (j + 1 < lenMax) acc.add(m[1], x[1], true);
      }
    }
    T w[3];
    acc.total(w);
    if (inc1 > inc0) {
      // contact: an incidence per thread, then every vertex adds its own in order
      double cr[3] = {0.0, 0.0, 0.0};
      const int chunk = min(NT, scratch / 4);
#pragma unroll 1
      for (int base = inc0; base < inc1; base += chunk) {
        if (tid < chunk && base + tid < inc1) {
          double t[3];
          area[4 * tid + 3] = collision_incidence<T>(
              b.coll, base + tid,
              [&](int id, T (&x)[3]) {
                Gather g;
                g.load(u4, id);
                g.get(u4, [&] { return id; }, it, b.waitPolls, x, ok);
              },
              t);
#pragma unroll
          for (int i = 0; i < 3; i++) area[4 * tid + i] = t[i];
        }
        __syncthreads();
#pragma unroll 1
        for (int k = max(my0, base); k < min(my1, base + chunk); k++)
#pragma unroll
          for (int i = 0; i < 3; i++) cr[i] = fma(area[4 * (k - base) + 3], area[4 * (k - base) + i], cr[i]);
        __syncthreads();
      }
      if (my1 > my0)
#pragma unroll
        for (int i = 0; i < 3; i++) w[i] += T(__dmul_rn(cr[i], collScale));
    }
    // ---- (w, u): tile sums, exchanged ----
    if constexpr (kF32) {
      T t2 = valid ? dot3v(w[0], w[1], w[2], un[0], un[1], un[2]) : T(0);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t2 += __shfl_xor_sync(0xffffffffu, t2, o);
      if (tid % 32 == 0) warpSum[2][tid / 32] = t2;
      if ((failed = __syncthreads_or(!ok))) break;
      publish32(2, 1, it);
    } else {
#pragma unroll
      for (int i = 0; i < 3; i++) area[6 * NT + 3 * tid + i] = valid ? w[i] * un[i] : 0.0;
      __syncthreads();
      publish64(2, 1, it);
    }
    if (it > 1)  // the last update's d, in the exchange's shadow
#pragma unroll
      for (int i = 0; i < 3; i++) d[i] = d[i] + alpha * p[i];
    const ulonglong2* in = words(it);
#pragma unroll 1
    for (int i0 = tid; i0 < 3 * nParts; i0 += 4 * NT) {
      double value[4];
      ld_words<4>([&](int k) { return i0 + k * NT < 3 * nParts; }, [&](int k) { return in + i0 + k * NT; },
                  (unsigned long long)it, b.waitPolls, value, ok);
#pragma unroll
      for (int k = 0; k < 4; k++) {
        const int i = i0 + k * NT;
        if (i < 3 * nParts) area[(i % 3) * nParts + i / 3] = value[k];
      }
    }
    failed = __syncthreads_or(!ok);
    const int nTrees = scene_trees<TV>(ntiles);
    if constexpr (kF32) {
#pragma unroll 1
      for (int c = tid / 32; c < 3; c += NT / 32) {
        const double* q = area + c * nParts;
        const double t = whole ? scene_sum(nGroups, [&](int g) { return q[g]; }) : scene_sum(nGroups, [&](int g) {
          return group_sum<TV>([&](int i) { return g * kG + i < ntiles ? q[g * kG + i] : 0.0; });
        });
        if (tid % 32 == 0) sums[c] = t;
      }
    } else {
      scene_tree32<TV>(ntiles, [&](int c, int i) { return area[c * nParts + i]; }, area + 3 * nParts, trees);
    }
    T M[9];
    if (kF32 && valid)
#pragma unroll
      for (int e = 0; e < 9; e++) M[e] = v.minv[minv_slot(u) + kSlice * e];
    __syncthreads();
    if (!kF32 && tid < 3) {
      sums[tid] = chain(trees + tid * nTrees, nTrees);
      __syncwarp(7u);
    }
    if (tid == 0) {
      stop = pcg_decide<T>(ss, sums[0], sums[1], sums[2], recip[0], recip[1]) ? 1 : 0;
      if constexpr (kF32) {
        sAlpha = ss.alphaF;
        sBeta = ss.betaF;
      } else {
        sAlpha = ss.alpha;
        sBeta = ss.beta;
      }
    }
    __syncthreads();
    if (stop || failed) break;
    // ---- p = u + beta p, s = w + beta s, d += alpha p, r -= alpha s, u = Minv r ----
    alpha = sAlpha;
    const T beta = sBeta;
    if (valid) {
      if (!kF32)  // (18 registers: not held across the scalars)
#pragma unroll
        for (int e = 0; e < 9; e++) M[e] = v.minv[minv_slot(u) + kSlice * e];
#pragma unroll
      for (int i = 0; i < 3; i++) {
        p[i] = un[i] + beta * p[i];
        sv[i] = w[i] + beta * sv[i];
        r[i] = r[i] - alpha * sv[i];
      }
#pragma unroll
      for (int i = 0; i < 3; i++) un[i] = M[3 * i] * r[0] + M[3 * i + 1] * r[1] + M[3 * i + 2] * r[2];
      publish_u(u4, u, un, it + 1);
      if constexpr (kF32) us[tid] = make_float4(un[0], un[1], un[2], 0.f);
    }
    if (!kF32) {
      __syncthreads();
      if (tid == 0) st_flag(flags + cta.y, it + 1);  // after the barrier: covers the whole CTA's u
    }
  }
  if (valid)
#pragma unroll
    for (int i = 0; i < 3; i++) v.d[3 * u + i] = d[i];
  // A CTA whose wait ran out publishes nothing more, so the scene's first CTA
  // runs out too, unless this iteration was the last.
  if (tid == 0 && cta.y == 0) {
    if (failed) {
      ss.converged = kSolveTimedOut;
      ss.waitFailures += 1;
      ss.outerDone = 1;
    }
    ss.done = 1;
    st = ss;
  }
}

template <int TV, typename T>
cudaError_t launch_tv(const DeviceBatch& b, const PcgVecs<T>& v, const GridPlan& g, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)g.ctas);
  cfg.blockDim = dim3((unsigned)(g.tpc * TV));
  cfg.dynamicSmemBytes = g.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_pcg_grid<TV, T>, b, v, g.list, g.tpc, g.rows, g.scratch, g.halo);
}

}  // namespace

// The line between the one launch and the loop: whether the tiles are resident
// at once, one CTA of at most 512 threads (128 registers each) per SM; below it
// the launch was the faster at every size of cube measured (343 to 68,921 vertices,
// 1.3 to 2.1 times an iteration).
// Not so in FP64 where rows are uneven: a warp's 32 rows take the longest one's
// time on the FP64 pipe, in the loop (a thread per scalar row) only 11 do, and the
// loop spreads any scene over all SMs.  Random Delaunay meshes, rows of 16 blocks
// and the longest of 32 on average 25, 5,500 to 77,000 vertices: the launch is the
// faster with 192 to 384 vertices a CTA on at least 70% of the SMs, 128 on 80% (us an
// iteration of launch / loop: 18,000 vertices 30.6 / 32.5, 32,000 38.6 / 45.7, 50,000
// 49.4 / 60.8) and the slower outside (5,500 26.6 / 20.6; 7,500 with 64 vertices a
// CTA 25.5 / 20.2; 15,000 with 128 on 78%, tiles of 64, 29.6 / 27.1; 20,000 on 52%
// 37.1 / 33.4; 70,000 with 512 69.5 / 59.8).  uneven: rows
// past those of a cube (15) and a quarter of the slices' places empty (cubes 2-6%,
// these meshes 55%).
// Tiles per CTA so that the tiles of the given scenes (their tile counts) take
// at most one CTA per SM, the fewest that does (an SM's FP64 pipe and L2 port
// are what an iteration runs at); none: they do not fit, and solver.cu's loop
// runs them.
GridPlan plan_grid_pcg(const int* tiles, int n, int tileV, bool mixed, bool uneven, int sms) {
  GridPlan g{};
  int most = 0;
  for (int s = 0; s < n; s++) most = std::max(most, tiles[s]);
  if (most == 0) return g;
  for (int tpc = 1; tpc * tileV <= kGridThreads; tpc++) {
    long long ctas = 0;
    for (int s = 0; s < n; s++) ctas += (tiles[s] + tpc - 1) / tpc;
    if (ctas > std::min(sms, kMaxCtas)) continue;
    const int verts = tpc * tileV;
    if (!mixed && uneven && (verts < 128 || verts > 384 || 10 * ctas < (verts == 128 ? 8 : 7) * sms))
      return g;
    g.ctas = (int)ctas;
    g.tpc = tpc;
    // the partials of a scene (in FP64 beside its tree's lanes); in FP64 the row
    // products, nine a thread
    g.scratch = mixed ? 3 * std::max(most, verts) : std::max(9 * verts, 3 * most + 9 * tileV);
    g.scratch += g.scratch % 2;
    return g;
  }
  return g;
}

// Shared memory: the exchange area, in FP32 the u of the CTA's vertices and of
// its halo, and of every row as many blocks and columns as still fit.
void plan_grid_smem(GridPlan& g, int tileV, int longestRow, bool mixed) {
  if (g.halo > kHaloMax) {
    g = GridPlan{};
    return;
  }
  const size_t threads = (size_t)g.tpc * tileV;
  const size_t fixed = sizeof(double) * g.scratch + (mixed ? sizeof(float4) * (threads + g.halo) : 0);
  const size_t row = threads * (9 * (mixed ? sizeof(float) : sizeof(double)) + sizeof(int));
  const int fit = (int)((kGridSmemMax - fixed) / row);
  // FP64 takes two blocks a trip
  g.rows = mixed ? std::min(longestRow, fit) : std::min(longestRow + longestRow % 2, fit / 2 * 2);
  g.smem = fixed + row * g.rows;
}

// A CTA's halo: the vertices of other CTAs in its rows' columns, ascending (a
// bit per vertex of the scene, then ranks), and every column's index in the
// shared u: the thread of an own vertex, or past the threads the halo's rank.
// A list longer than its room (four times the threads, kHaloMax) leaves
// the batch to solver.cu's loop.
constexpr int kHaloWords = 152 * kGridThreads / 32 + 8 * kMaxCtas;
__global__ void __launch_bounds__(kGridThreads) k_grid_halo(DeviceBatch b, const int2* __restrict__ ctas, int tpc,
                                                            int* largest) {
  __shared__ unsigned bits[kHaloWords];
  __shared__ int rank[kHaloWords];
  __shared__ int warpTot[kGridThreads / 32];
  const int tid = threadIdx.x, NT = blockDim.x;
  const int2 cta = ctas[blockIdx.x];
  const SceneParams& sp = b.scenes[cta.x];
  const int v0 = sp.v0, words = (sp.nv + 31) / 32;
  const int a = b.tileV0[sp.tile0 + cta.y], z = b.tileV1[sp.tile0 + min(sp.ntiles, cta.y + tpc) - 1];
  if (words > kHaloWords) return;  // (a scene of a plan has at most one CTA's vertices per SM)
  for (int i = tid; i < words; i += NT) bits[i] = 0u;
  __syncthreads();
  const int u = a + tid;
  const int len = u < z ? b.rowptr[u + 1] - b.rowptr[u] : 0;
  const size_t cb = u < z ? col_slot(b, u, 0) : 0;
  for (int j = 0; j < len; j++) {
    const int w = b.colS[cb + kSlice * j];
    if (w < a || w >= z) atomicOr(&bits[(w - v0) / 32], 1u << ((w - v0) % 32));
  }
  __syncthreads();
  // exclusive ranks of the words: each thread a run of them, then the runs
  const int per = (words + NT - 1) / NT, i0 = min(words, tid * per), i1 = min(words, i0 + per);
  int mine = 0;
  for (int i = i0; i < i1; i++) mine += __popc(bits[i]);
  int x = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (tid % 32 >= o) x += y;
  }
  if (tid % 32 == 31) warpTot[tid / 32] = x;
  __syncthreads();
  int at = x - mine;
  for (int i = 0; i < tid / 32; i++) at += warpTot[i];
  const int cap = min(kHaloMax, 4 * NT);
  int* list = halo_list(b, cta.x, a);
  for (int i = i0; i < i1; i++) {
    rank[i] = at;
    for (unsigned m = bits[i]; m; m &= m - 1, at++)
      if (at < cap) list[at] = v0 + 32 * i + __ffs(m) - 1;
  }
  if (tid == NT - 1) {
    b.gridHaloCount[sp.tile0 + cta.y] = at;
    atomicMax(largest, at <= cap ? at : kHaloMax + 1);
  }
  __syncthreads();
  for (int j = 0; j < len; j++) {
    const int w = b.colS[cb + kSlice * j], l = w - v0;
    int c = w - a;
    if (w < a || w >= z) {
      const int r = rank[l / 32] + __popc(bits[l / 32] & ((1u << (l % 32)) - 1u));
      c = NT + r;
    }
    b.clusterGather[cb + kSlice * j] = c;
  }
}

void launch_grid_halo(const DeviceBatch& b, const GridPlan& g, int* largest, cudaStream_t s) {
  k_grid_halo<<<g.ctas, g.tpc * b.tileV, 0, s>>>(b, g.list, g.tpc, largest);
}

// Dynamic shared-memory opt-in (once per device, outside capture).
int configure_grid_pcg() {
  static OncePerDevice once;
  return once_on_this_device(once, [] {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_pcg_grid<64, float>, attr, kGridSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_pcg_grid<128, float>, attr, kGridSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_pcg_grid<64, double>, attr, kGridSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_pcg_grid<128, double>, attr, kGridSmemMax);
    return (int)e;
  });
}

template <typename T>
int launch_grid_pcg(const DeviceBatch& b, const PcgVecs<T>& v, const GridPlan& g, cudaStream_t s) {
  return (int)(b.tileV == 64 ? launch_tv<64, T>(b, v, g, s) : launch_tv<128, T>(b, v, g, s));
}
template int launch_grid_pcg<double>(const DeviceBatch&, const PcgVecs<double>&, const GridPlan&, cudaStream_t);
template int launch_grid_pcg<float>(const DeviceBatch&, const PcgVecs<float>&, const GridPlan&, cudaStream_t);

}  // namespace hobak
