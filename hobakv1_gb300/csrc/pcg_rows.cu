// The FP64 one-launch PCG of small scenes, a thread per scalar row.
//
// pcg_grid.cu gives a CTA at least a tile, 64 or 128 vertices, one per thread:
// a scene of a few thousand vertices then runs on a few SMs, each warp's 135
// products a row block chain through an FP64 pipe that takes 19 cycles for
// each.  Where 32 vertices per SM hold all tile-path scenes of the batch
// (4,864 vertices), a CTA here takes 32 vertices with three threads each: its
// three warps run on three of the SM's sub-partitions (45 products each, 64
// cycles apart), and the 32 rows of a warp are exactly one tree of the tile
// sums' order, so no sum needs shared memory.  The matrix rows are all in shared
// memory.  Both exchanges are pcg_grid.cu's tagged 16-byte words, u one word per
// row; partials carry the solve's number beside the iteration, so no solve has
// to clear them.  Sums and scalars are formed as in solver.cu, with the same bits.
//
// What bounds it: latency (two exchanges through L2, the FP64 chains of the tile
// and scene sums and of the scalars).  1,331 vertices: 31,000 -> 17,000 cycles
// an iteration, 10^3 drop-in solve 399 -> 305 us; 343 vertices 260 -> 214 us.
// Waiting for a thread's words together and not one by one: 2,197 vertices, three
// Newmark iterations 1,120 -> 990 us, 3,375 vertices 493 -> 466 us.
#include <algorithm>

#include "pcg_common.cuh"

namespace hobak {

namespace {

constexpr int kRowVerts = 32;                // vertices of a CTA
constexpr int kRowThreads = 3 * kRowVerts;
constexpr int kRowCtas = kGridCtas;
constexpr int kRowSmemMax = 200 * 1024;
constexpr int kBatch = 4;                    // blocks whose u is in flight
constexpr int kWords = 8;                    // partials a thread polls at a time

// ctas: per CTA its scene and its index in the scene.
template <int TV>
__global__ void __launch_bounds__(kRowThreads, 1)
    k_pcg_rows(DeviceBatch b, PcgVecs<double> v, const int2* __restrict__ ctas, int rows) {
  constexpr int kTrees = 3 * TV / 32;  // of a tile
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ SolveState ss;
  __shared__ double part[3][3 * kRowCtas];             // [component][tree of the scene]
  __shared__ double tiles[3][kRowCtas * kRowVerts / 64];  // [component][tile]
  __shared__ double inc[kRowThreads][4];               // contact incidences
  __shared__ double sums[3], recip[2], newR[kRowThreads];
  __shared__ int stop;

  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int2 cta = ctas[blockIdx.x];
  const int s = cta.x;
  const SceneParams& sp = b.scenes[s];
  SolveState& st = b.solve[s];
  if (st.done) return;  // converged at its start, parked or failed (every CTA of the scene alike)
  const int v0 = sp.v0, n = sp.nv, ntiles = sp.ntiles;
  const int nCta = (n + kRowVerts - 1) / kRowVerts, nTrees = 3 * nCta;
  const int lv = tid / 3, i = tid - 3 * lv;
  const int u = v0 + kRowVerts * cta.y + lv;
  const bool valid = u < v0 + n;
  const int own = valid ? u : v0;
  const size_t row = 3 * (size_t)u + i;

  double* mat = reinterpret_cast<double*>(smem);                              // [3 j + c][thread]
  int* col = reinterpret_cast<int*>(mat + (size_t)3 * rows * kRowThreads);    // [j][vertex]
  int len = 0;
  double un = 0.0, r = 0.0, p = 0.0, sv = 0.0, d = 0.0, M[3] = {0.0, 0.0, 0.0};
  size_t lb = 0, cb = 0;
  if (valid) {
    len = b.rowptr[u + 1] - b.rowptr[u];
    lb = lhs_slot(b, u, 0) + kSlice * 3 * i;
    cb = col_slot(b, u, 0);
    un = v.u[row];
    r = b.r64[row];
#pragma unroll
    for (int c = 0; c < 3; c++) M[c] = v.minv[minv_slot(u) + kSlice * (3 * i + c)];
  }
#pragma unroll 1
  for (int j = 0; j < rows; j++) {  // zeros past the row's end
    if (i == 0) col[j * kRowVerts + lv] = j < len ? __ldg(&b.colS[cb + kSlice * j]) : own;
#pragma unroll
    for (int c = 0; c < 3; c++)
      mat[(size_t)(3 * j + c) * kRowThreads + tid] =
          j < len ? __ldg(&v.lhs[lb + (size_t)kSlotVals * j + kSlice * c]) : 0.0;
  }
  if (tid == 0) {
    ss = st;
    stop = 0;
  }
  int inc0 = 0, inc1 = 0, my0 = 0, my1 = 0;
  double collScale = 0.0;
  if (b.collOn) {  // the CTA's contact incidences (CSR by vertex)
    const int first = v0 + kRowVerts * cta.y;
    inc0 = b.coll.incCount[first];
    inc1 = b.coll.incCount[min(v0 + n, first + kRowVerts)];
    if (valid && b.freeMask[u]) {
      my0 = b.coll.incCount[u];
      my1 = b.coll.incCount[u + 1];
    }
    if (inc1 > inc0) collScale = collision_lhs_scale(b, s);
  }
  const int lenMax = __reduce_max_sync(0xffffffffu, len);
  __syncthreads();
  const unsigned long long solve = (unsigned long long)(unsigned)ss.epoch << 32;
  ulonglong2* uw = reinterpret_cast<ulonglong2*>(v.p);  // u: a word per row
  ulonglong2* mine = b.gridRowWords + 9 * (size_t)blockIdx.x;
  const ulonglong2* scene = b.gridRowWords + 9 * (size_t)(blockIdx.x - cta.y);
  constexpr size_t kParity = 9 * (size_t)kRowCtas;
  bool ok = true;  // this thread's waits
  int failed = 0;  // some thread's wait ran out (the same in all threads)

#pragma unroll 1
  for (int it = 1;; it++) {
    const unsigned long long tag = solve | (unsigned)it;
    const size_t par = (it & 1) * kParity;
    // ---- |r|^2 and (r, u): the warp's rows are one tree of its tile ----
    {
      const double rl = warp_tree(valid ? r * r : 0.0), gl = warp_tree(valid ? r * un : 0.0);
      if (lane == 0) {
        st_word(mine + par + 3 * warp, rl, tag);
        st_word(mine + par + 3 * warp + 1, gl, tag);
      }
    }
    if (it > 1 && tid >= kRowThreads - 2)
      recip[kRowThreads - 1 - tid] = 1.0 / (tid == kRowThreads - 1 ? ss.gamma : ss.alpha);
    // ---- w = A u: the chains of even and odd blocks ----
    double a0 = 0.0, a1 = 0.0;
#pragma unroll 1
    for (int j0 = 0; j0 < lenMax; j0 += kBatch) {
      double x[3 * kBatch];
      int w[kBatch];
#pragma unroll
      for (int q = 0; q < kBatch; q++) w[q] = j0 + q < rows ? col[(j0 + q) * kRowVerts + lv] : own;
      ld_words<3 * kBatch>([&](int) { return true; }, [&](int k) { return uw + 3 * (size_t)w[k / 3] + k % 3; },
                           (unsigned long long)it, b.waitPolls, x, ok);
#pragma unroll
      for (int q = 0; q < kBatch; q++)
        if (j0 + q < lenMax) {
          double& a = q & 1 ? a1 : a0;
#pragma unroll
          for (int c = 0; c < 3; c++)
            a = fma(mat[(size_t)(3 * (j0 + q) + c) * kRowThreads + tid], x[3 * q + c], a);
        }
    }
    double w = a0 + a1;
    if (inc1 > inc0) {
      double cr = 0.0;
#pragma unroll 1
      for (int base = inc0; base < inc1; base += kRowThreads) {
        if (base + tid < inc1) {
          double t[3];
          inc[tid][3] = collision_incidence<double>(
              b.coll, base + tid,
              [&](int id, double (&x)[3]) {
                ld_words<3>([&](int) { return true; }, [&](int c) { return uw + 3 * (size_t)id + c; },
                            (unsigned long long)it, b.waitPolls, x, ok);
              },
              t);
#pragma unroll
          for (int c = 0; c < 3; c++) inc[tid][c] = t[c];
        }
        __syncthreads();
#pragma unroll 1
        for (int k = max(my0, base); k < min(my1, base + kRowThreads); k++)
          cr = fma(inc[k - base][3], inc[k - base][i], cr);
        __syncthreads();
      }
      if (my1 > my0) w += __dmul_rn(cr, collScale);
    }
    // ---- (w, u), then everybody's partials ----
    {
      const double dl = warp_tree(valid ? w * un : 0.0);
      if (lane == 0) st_word(mine + par + 3 * warp + 2, dl, tag);
    }
    if (it > 1) d = d + ss.alpha * p;  // the last update's d, in the exchange's shadow
#pragma unroll 1
    for (int k0 = tid; k0 < 3 * nTrees; k0 += kWords * kRowThreads) {
      double value[kWords];
      ld_words<kWords>([&](int k) { return k0 + k * kRowThreads < 3 * nTrees; },
                       [&](int k) { return scene + par + k0 + k * kRowThreads; }, tag, b.waitPolls, value, ok);
#pragma unroll
      for (int k = 0; k < kWords; k++) {
        const int q = k0 + k * kRowThreads;
        if (q < 3 * nTrees) part[q % 3][q / 3] = value[k];
      }
    }
    if ((failed = __syncthreads_or(!ok))) break;
    // tile sums in order of their trees (the trees past the scene's end are zero)
#pragma unroll 1
    for (int k = tid; k < 3 * ntiles; k += kRowThreads) {
      const int c = k % 3, t = k / 3;
      tiles[c][t] = chain(part[c] + kTrees * t, min(kTrees, nTrees - kTrees * t));
    }
    __syncthreads();
    {
      // lanes of the scene's sum: a tile each (at most 76 tiles, 3 TV lanes)
      double t = warp_tree(lane < ntiles ? tiles[warp][lane] : 0.0);
#pragma unroll 1
      for (int l = 32; l < ntiles; l += 32) t += warp_tree(l + lane < ntiles ? tiles[warp][l + lane] : 0.0);
      if (lane == 0) sums[warp] = t;
    }
    __syncthreads();
    if (tid == 0) stop = pcg_decide<double>(ss, sums[0], sums[1], sums[2], recip[0], recip[1]) ? 1 : 0;
    __syncthreads();
    if (stop) break;
    // ---- p = u + beta p, s = w + beta s, r -= alpha s, u = Minv r (d: above) ----
    const double alpha = ss.alpha, beta = ss.beta;
    p = un + beta * p;
    sv = w + beta * sv;
    r = r - alpha * sv;
    newR[tid] = r;
    __syncthreads();
    un = M[0] * newR[3 * lv] + M[1] * newR[3 * lv + 1] + M[2] * newR[3 * lv + 2];
    if (valid) st_word(uw + row, un, (unsigned long long)(it + 1));
  }
  if (valid) v.d[row] = d;
  // a CTA whose wait ran out publishes nothing more, so the first one runs out too
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

template <int TV>
cudaError_t launch_tv(const DeviceBatch& b, const PcgVecs<double>& v, const GridPlan& g, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)g.ctas);
  cfg.blockDim = dim3(kRowThreads);
  cfg.dynamicSmemBytes = g.smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_pcg_rows<TV>, b, v, g.list, g.rows);
}

}  // namespace

size_t grid_row_words() { return 2 * 9 * (size_t)kRowCtas; }

// The plan for scenes of nv[s] vertices (0: not on the tile path); none where
// they take more than one CTA of 32 vertices per SM.
GridPlan plan_rows_pcg(const int* nv, int n, int longestRow, int sms) {
  GridPlan g{};
  long long ctas = 0;
  for (int s = 0; s < n; s++) ctas += (nv[s] + kRowVerts - 1) / kRowVerts;
  const size_t smem = (size_t)longestRow * (3 * kRowThreads * sizeof(double) + kRowVerts * sizeof(int));
  if (ctas == 0 || ctas > std::min(sms, kRowCtas) || smem > kRowSmemMax) return g;
  g.ctas = (int)ctas;
  g.rowVerts = kRowVerts;
  g.rows = longestRow;
  g.smem = smem;
  return g;
}

// Dynamic shared-memory opt-in (once per device, outside capture).
int configure_rows_pcg() {
  static OncePerDevice once;
  return once_on_this_device(once, [] {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_pcg_rows<64>, attr, kRowSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_pcg_rows<128>, attr, kRowSmemMax);
    return (int)e;
  });
}

int launch_rows_pcg(const DeviceBatch& b, const PcgVecs<double>& v, const GridPlan& g, cudaStream_t s) {
  return (int)(b.tileV == 64 ? launch_tv<64>(b, v, g, s) : launch_tv<128>(b, v, g, s));
}

}  // namespace hobak
