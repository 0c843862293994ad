// Conjugate gradients as one resident kernel: the whole solve in a single
// cooperative launch, one CTA an SM, each owning a block of rows that is
// compact in space.
//
// What bounds the three-kernel iteration (fm_poisson.cu) is not bytes but the
// chain of three launches, each with a reduction over the grid, and a matrix
// product whose gathers go through L2: 31.6 us an iteration at 64^3 tets
// (274,625 rows; its 41 MB of matrix sit in L2) and 18.9 us at 20,944 rows.
// Here a CTA keeps the direction of its rows and of the columns they touch
// (its halo) in shared memory, so the product gathers from there with 16-bit
// local columns (10 instead of 12 bytes an entry), and as much of its matrix
// block as fits stays there too; two exchanges over the grid remain in an
// iteration.  Each halo copy of the direction is updated with the same
// arithmetic as its owner's, from the preconditioned residual z that the
// owners write out, so z is all that crosses CTAs.  (residual_z and
// next_direction fix the roundings: left to the compiler, an owner's
// D^-1 r + beta p may round beta p where a copy's z + beta p rounds z, and the
// copies drift from their owners.)
//
// An exchange: every CTA writes its two partial sums into a table and adds
// one to an arrival counter (release, which covers its z), one thread polls
// the counter (acquire) until all have arrived, and the first warp of every
// CTA adds the table in the same order, so all take the same decisions and
// the sums have a fixed order.  2.1 us over 148 CTAs; polling the other CTAs'
// table entries directly, without the counter, took 5.9 us (148 x 148 polls
// of lines that are being written).  The table is double buffered: a CTA that
// writes for exchange k + 2 has seen all arrive at k + 1, hence all have read
// k.  The launch is cooperative (all CTAs are resident), the poll loop is
// bounded (CgResident::polls), and a CTA that gives up returns with a time-out
// in the control word, which no other CTA's verdict replaces.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace {

// Rows a CTA: up to kResOne rows one CTA (no exchange: 3.2 against 5.2 us an
// iteration at 729 rows), else at least kResRows (256 or 512 a CTA: 7.0 / 8.8
// against 6.8 us at 21,952 rows).
constexpr int kResOne = 1024, kResRows = 128;
// Threads: 1024 once a CTA has more than kResWide rows (12.2 against 13.0 us
// at 64^3 tets, 46 against 57 us at 96^3), else 512 (6.8 against 7.3 us at
// 21,952 rows).
constexpr int kResWide = 1024;
// Loads a thread has in flight: matrix entries, and rows of the vector loops.
constexpr int res_batch(int threads) { return threads == 1024 ? 8 : 16; }
constexpr int kResRowsAhead = 4;
constexpr uint32_t kResPolls = 1u << 22;  // default limit of an exchange's wait: a few seconds

// Device view.  CTA c owns rows row0[c] .. row0[c+1] of the reordered system.
// Its local columns: first its own rows, then halo[halo0[c] ..] (row numbers).
// Its rows are cut into slices of 32, a lane a row, entry k of slice s at
// (slice_at[s] + k) * 32 + lane, padded to the slice's longest row.
struct CgResident {
  int32_t ctas, threads;
  int32_t rows_max, local_max, halo_max;  // largest CTA's
  int32_t vectors;                        // vectors in shared memory beside p: 0, 2 (q, r) or 4 (and x, D^-1)
  int32_t cache;                          // matrix entries kept in shared memory (a multiple of 32)
  const int32_t *row0, *halo0, *halo, *slice0, *slice_at;
  const double* val;
  const uint16_t* col;
  double2* partials;   // [2][ctas]
  unsigned long long* arrived;
  uint32_t polls;                         // an exchange's wait gives up after this many (kResPolls)
  double* seen;                           // null, or where the last direction goes: the rows', then the halos' copies
  size_t smem;
};

__device__ __forceinline__ void warp_sum(double& v0, double& v1) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v0 += __shfl_xor_sync(0xffffffffu, v0, o);
    v1 += __shfl_xor_sync(0xffffffffu, v1, o);
  }
}

// Adds v0 and v1 over all CTAs (see above).  arrive: this CTA's sums are in;
// wait: the totals, the same in every thread, false when the exchange did not
// complete.  Work that needs neither goes between.  sh: 2 x (warps + 1)
// doubles.
template <int THREADS>
__device__ __forceinline__ void grid_arrive(const CgResident& R, uint64_t number, double v0, double v1, double* sh) {
  constexpr int W = THREADS / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  warp_sum(v0, v1);
  if (lane == 0) {
    sh[warp] = v0;
    sh[W + warp] = v1;
  }
  __syncthreads();
  if (warp == 0) {
    v0 = lane < W ? sh[lane] : 0.0;
    v1 = lane < W ? sh[W + lane] : 0.0;
    warp_sum(v0, v1);
    if (lane == 0) {
      if (R.ctas > 1) {
        R.partials[(number & 1) * R.ctas + blockIdx.x] = make_double2(v0, v1);
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(R.arrived) : "memory");
      } else {
        sh[2 * W] = v0;
        sh[2 * W + 1] = v1;
      }
    }
  }
}
template <int THREADS>
__device__ __forceinline__ bool grid_wait(const CgResident& R, uint64_t number, double& v0, double& v1, double* sh,
                                          int* failed) {
  constexpr int W = THREADS / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp == 0 && R.ctas > 1) {
    if (lane == 0) {
      const uint64_t all = number * (uint64_t)R.ctas;
      uint64_t n = 0;
      for (uint32_t polls = 0; n < all && polls < R.polls; ++polls)
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(n) : "l"(R.arrived) : "memory");
      if (n < all) *failed = 1;
    }
    __syncwarp();
    v0 = v1 = 0.0;
    for (int i = lane; i < R.ctas; i += 32) {
      const double2 t = __ldcg(R.partials + (number & 1) * R.ctas + i);
      v0 += t.x;
      v1 += t.y;
    }
    warp_sum(v0, v1);
    if (lane == 0) {
      sh[2 * W] = v0;
      sh[2 * W + 1] = v1;
    }
  }
  __syncthreads();
  v0 = sh[2 * W];
  v1 = sh[2 * W + 1];
  return *failed == 0;
}

// Entries of one slice in order, this lane's row: val / col point at entry 0
// of the lane, w entries.
template <int BATCH>
__device__ __forceinline__ double slice_row(const double* val, const uint16_t* col, int w, const double* p) {
  double s = 0.0;
  for (int k = 0; k < w; k += BATCH) {
    double v[BATCH];
    int j[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      const bool in = k + u < w;
      v[u] = in ? val[(k + u) * 32] : 0.0;
      j[u] = in ? col[(k + u) * 32] : 0;
    }
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
      if (k + u < w) s += v[u] * p[j[u]];
  }
  return s;
}

// f(load, use) over i = tid, tid + THREADS, ... < n in groups: the group's
// loads are issued before its first use (the compiler cannot move a load
// over another element's store by itself).
template <int THREADS, class LOAD, class USE>
__device__ __forceinline__ void ahead(int n, LOAD load, USE use) {
  for (int i0 = threadIdx.x; i0 < n; i0 += kResRowsAhead * THREADS) {
    double v[kResRowsAhead];
#pragma unroll
    for (int u = 0; u < kResRowsAhead; ++u)
      if (i0 + u * THREADS < n) v[u] = load(i0 + u * THREADS);
#pragma unroll
    for (int u = 0; u < kResRowsAhead; ++u)
      if (i0 + u * THREADS < n) use(i0 + u * THREADS, v[u]);
  }
}

__device__ __forceinline__ double residual_z(double dinv, double r) { return __dmul_rn(dinv, r); }
__device__ __forceinline__ double next_direction(double z, double beta, double p) { return __fma_rn(beta, p, z); }

// VECTORS: how many of q, r, x, D^-1 (in this order) live in shared memory
// beside p: 4, 2 or 0 (known at compile time, so that their accesses are
// plain shared-memory ones).
template <int THREADS, int VECTORS>
__global__ void __launch_bounds__(THREADS, 1) cg_resident_kernel(Cg c, CgResident R) {
  extern __shared__ __align__(16) double sm[];
  __shared__ double sh[2 * (THREADS / 32 + 1)];
  __shared__ int failed;
  const int cta = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t r0 = R.row0[cta];
  const int rows = (int)(R.row0[cta + 1] - r0);
  const int nh = R.halo0[cta + 1] - R.halo0[cta];
  const int s0 = R.slice0[cta], ns = R.slice0[cta + 1] - s0;
  double* p = sm;  // own rows, then the halo
  double* own = p + R.local_max;
  double* q = VECTORS >= 2 ? own : c.q + r0;
  double* r = VECTORS >= 2 ? own + R.rows_max : c.r + r0;
  double* x = VECTORS >= 4 ? own + 2 * R.rows_max : c.x + r0;
  double* dinv = VECTORS >= 4 ? own + 3 * R.rows_max : const_cast<double*>(c.dinv) + r0;
  double* cval = own + VECTORS * R.rows_max;
  int32_t* halo = reinterpret_cast<int32_t*>(cval + R.cache);
  uint16_t* ccol = reinterpret_cast<uint16_t*>(halo + R.halo_max);
  if (tid == 0) failed = 0;
  // the first slices that fit stay in shared memory
  const int64_t e0 = (int64_t)R.slice_at[s0] * 32;
  int cached = 0;
  while (cached < ns && ((int64_t)R.slice_at[s0 + cached + 1] * 32 - e0) <= R.cache) ++cached;
  const int64_t ce = (int64_t)R.slice_at[s0 + cached] * 32 - e0;
  for (int64_t i = tid; i < ce; i += THREADS) {
    cval[i] = R.val[e0 + i];
    ccol[i] = R.col[e0 + i];
  }
  for (int i = tid; i < nh; i += THREADS) halo[i] = R.halo[R.halo0[cta] + i];
  // x = x0, r = b, z = D^-1 r
  double rz = 0.0, rr = 0.0;
  for (int i = tid; i < rows; i += THREADS) {
    const double ri = c.b[r0 + i], di = c.dinv[r0 + i], zi = residual_z(di, ri);
    x[i] = c.xinit[r0 + i];
    r[i] = ri;
    if (VECTORS >= 4) dinv[i] = di;
    c.z[r0 + i] = zi;
    rz += ri * zi;
    rr += ri * ri;
  }
  uint64_t number = 0;
  grid_arrive<THREADS>(R, ++number, rz, rr, sh);
  bool ok = grid_wait<THREADS>(R, number, rz, rr, sh, &failed);
  const double stop = c.scal[6];
  const int max_it = c.ctl[3];
  int it = 0, error = 0;
  double beta = 0.0;
  bool done = !ok || rr <= stop || max_it <= 0;
  while (!done) {
    // p = z + beta p, own rows and halo
    if (it == 0) {
      for (int i = tid; i < rows; i += THREADS) p[i] = residual_z(dinv[i], r[i]);
      for (int i = tid; i < nh; i += THREADS) p[rows + i] = __ldcg(c.z + halo[i]);
    } else {
      ahead<THREADS>(
          nh, [&](int i) { return __ldcg(c.z + halo[i]); },
          [&](int i, double z) { p[rows + i] = next_direction(z, beta, p[rows + i]); });
      if constexpr (VECTORS >= 4) {
        for (int i = tid; i < rows; i += THREADS) p[i] = next_direction(residual_z(dinv[i], r[i]), beta, p[i]);
      } else {
        ahead<THREADS>(
            rows, [&](int i) { return dinv[i]; },
            [&](int i, double d) { p[i] = next_direction(residual_z(d, r[i]), beta, p[i]); });
      }
    }
    __syncthreads();
    double pq = 0.0, unused;
    for (int s = warp; s < ns; s += THREADS / 32) {
      const int64_t at = (int64_t)R.slice_at[s0 + s] * 32;
      const int w = R.slice_at[s0 + s + 1] - R.slice_at[s0 + s];
      const int row = s * 32 + lane;
      const double a = s < cached ? slice_row<res_batch(THREADS)>(cval + (at - e0) + lane, ccol + (at - e0) + lane, w, p)
                                  : slice_row<res_batch(THREADS)>(R.val + at + lane, R.col + at + lane, w, p);
      if (row < rows) {
        q[row] = a;
        pq += p[row] * a;
      }
    }
    grid_arrive<THREADS>(R, ++number, pq, 0.0, sh);
    ok = grid_wait<THREADS>(R, number, pq, unused, sh, &failed);
    if (!ok) break;
    if (!(pq > 0.0) || !isfinite(pq)) {
      error = 1;  // breakdown: K not positive definite on p, or a NaN
      break;
    }
    const double alpha = rz / pq;
    double nrz = 0.0;
    rr = 0.0;
    auto update = [&](int i, double d) {
      const double ri = r[i] - alpha * q[i];
      const double zi = residual_z(d, ri);
      r[i] = ri;
      c.z[r0 + i] = zi;
      nrz += ri * zi;
      rr += ri * ri;
    };
    if constexpr (VECTORS >= 4) {
      for (int i = tid; i < rows; i += THREADS) {
        x[i] += alpha * p[i];
        update(i, dinv[i]);
      }
      grid_arrive<THREADS>(R, ++number, nrz, rr, sh);
    } else {
      ahead<THREADS>(rows, [&](int i) { return dinv[i]; }, update);
      grid_arrive<THREADS>(R, ++number, nrz, rr, sh);
      // x while the others arrive
      ahead<THREADS>(
          rows, [&](int i) { return x[i]; }, [&](int i, double xi) { x[i] = xi + alpha * p[i]; });
    }
    ok = grid_wait<THREADS>(R, number, nrz, rr, sh, &failed);
    if (!ok) break;
    ++it;
    if (!isfinite(rr)) {
      error = 1;
      break;
    }
    done = rr <= stop || it >= max_it;
    beta = nrz / rz;
    rz = nrz;
  }
  if (VECTORS >= 4)
    for (int i = tid; i < rows; i += THREADS) c.x[r0 + i] = x[i];
  if (R.seen && it > 0) {
    for (int i = tid; i < rows; i += THREADS) R.seen[r0 + i] = p[i];
    for (int i = tid; i < nh; i += THREADS) R.seen[c.n + R.halo0[cta] + i] = p[rows + i];
  }
  if (!ok && tid == 0) c.ctl[2] = 2;
  if (ok && cta == 0 && tid == 0) {
    c.scal[4] = rr;
    c.ctl[0] = 1;
    c.ctl[1] = it;
    if (error) atomicMax(c.ctl + 2, 1);  // a time-out (2) of another CTA stays
  }
}

using ResidentKernel = void (*)(Cg, CgResident);
inline ResidentKernel resident_kernel(int threads, int vectors) {
  if (vectors == 2) return cg_resident_kernel<1024, 2>;
  if (vectors == 0) return cg_resident_kernel<1024, 0>;
  return threads == 1024 ? cg_resident_kernel<1024, 4> : cg_resident_kernel<512, 4>;
}

// ---- host side ----
// The reordered system of the resident kernel.
struct ResidentHost {
  bool fits = false;
  CgResident R{};
  fm::hvec<int32_t> row_of;   // row of each node
  fm::hvec<int64_t> node_of;  // node of each row
  std::vector<int32_t> row0, halo0, slice0, slice_at;
  fm::hvec<int32_t> halo;
  fm::hvec<double> val;
  fm::hvec<uint16_t> col;
};

// Cuts the system (rowp: the rows' offsets; row(v): the columns and values of
// node v's row) into the CTAs' blocks.  Rows go by the
// Morton order of their nodes, so a block is compact and its halo small;
// within a block the longest rows come first, so a slice's rows are alike.
// fits is false when some CTA's direction would not fit shared memory (above
// about 20,000 rows an SM): the caller then keeps the three-kernel iteration.
template <class ROW>
void build_resident(const double* coords, int64_t N, const std::vector<int32_t>& rowp, ROW row, int sms,
                    size_t smem_limit, ResidentHost& H) {
  CgResident& R = H.R;
  const int G = N <= kResOne ? 1 : (int)std::min<int64_t>(sms, N / kResRows);
  if ((size_t)(N / G) * 8 > smem_limit) return;
  R.ctas = G;
  R.threads = N / G > kResWide ? 1024 : 512;
  fm::morton_order_nodes(coords, N, H.node_of);
  H.row_of.resize(N);
  H.row0.resize(G + 1);
  for (int g = 0; g <= G; ++g) H.row0[g] = (int32_t)(N * g / G);
  auto len = [&](int64_t v) { return rowp[v + 1] - rowp[v]; };
  std::vector<std::vector<int32_t>> hal(G);
  std::vector<std::vector<int32_t>> width(G);
  // the blocks on the host threads, some 4,000 rows a thread at least (below,
  // starting a thread costs more than its work)
  auto over = [&](auto&& f) {
    fm::parallel_blocks(
        G, [&](int64_t b, int64_t e, int) { for (int64_t g = b; g < e; ++g) f((int)g); }, 4096 * G / N + 1);
  };
  over([&](int g) {
    std::stable_sort(H.node_of.begin() + H.row0[g], H.node_of.begin() + H.row0[g + 1],
                     [&](int64_t a, int64_t b) { return len(a) > len(b); });
    for (int64_t i = H.row0[g]; i < H.row0[g + 1]; ++i) H.row_of[H.node_of[i]] = (int32_t)i;
  });
  // each block's halo (its columns outside it, through a small open-addressing
  // map) and its entries' local columns; once a block does not fit, the others
  // are not formed
  std::vector<std::vector<uint16_t>> local(G);
  std::atomic<bool> over_limit{false};
  over([&](int g) {
    if (over_limit) return;
    const int32_t a = H.row0[g], b = H.row0[g + 1];
    std::vector<int32_t>& h = hal[g];
    std::vector<int32_t> key(1024, -1), id(1024);
    uint32_t mask = 1023;
    auto slot = [&](int32_t w) {
      uint32_t q = ((uint32_t)w * 2654435761u) >> 7 & mask;
      while (key[q] != w && key[q] >= 0) q = (q + 1) & mask;
      return q;
    };
    int64_t entries = 0;
    for (int32_t i = a; i < b; ++i) entries += len(H.node_of[i]);
    std::vector<uint16_t>& lc = local[g];
    lc.resize(entries);
    // halo columns by their first occurrence, then in order
    uint16_t* out = lc.data();
    for (int32_t i = a; i < b; ++i) {
      const int64_t v = H.node_of[i];
      const int n = len(v);
      if ((i - a) % 32 == 0) width[g].push_back(n);
      const int32_t* col = row(v).first;
      for (int32_t k = 0; k < n; ++k) {
        const int32_t w = H.row_of[col[k]];
        if (w >= a && w < b) {
          *out++ = (uint16_t)(w - a);
          continue;
        }
        uint32_t q = slot(w);
        if (key[q] < 0) {
          const size_t m = h.size() + 1;  // the direction and the halo's row numbers
          if (b - a + m > 65536 || (b - a + m) * 8 + m * 4 > smem_limit) {
            over_limit = true;
            return;
          }
          if (2 * (h.size() + 1) > mask) {
            mask = 2 * mask + 1;
            key.assign(mask + 1, -1);
            id.resize(mask + 1);
            for (size_t j = 0; j < h.size(); ++j) {
              const uint32_t r = slot(h[j]);
              key[r] = h[j];
              id[r] = (int32_t)j;
            }
            q = slot(w);
          }
          key[q] = w;
          id[q] = (int32_t)h.size();
          h.push_back(w);
        }
        *out++ = (uint16_t)(b - a + id[q]);
      }
    }
    std::vector<uint16_t> rank(h.size());
    std::vector<int32_t> first(h);
    std::sort(h.begin(), h.end());
    for (size_t i = 0; i < h.size(); ++i) id[slot(h[i])] = (int32_t)i;
    for (size_t j = 0; j < first.size(); ++j) rank[j] = (uint16_t)(b - a + id[slot(first[j])]);
    for (uint16_t& c : lc)
      if (c >= b - a) c = rank[c - (b - a)];
  });
  if (over_limit) return;
  H.halo0.assign(G + 1, 0);
  H.slice0.assign(G + 1, 0);
  int64_t hsum = 0;
  for (int g = 0; g < G; ++g) {
    const int rows = H.row0[g + 1] - H.row0[g], nh = (int)hal[g].size();
    hsum += nh;
    if (rows + nh > 65536 || hsum >= INT32_MAX) return;
    R.rows_max = std::max(R.rows_max, rows);
    R.halo_max = std::max(R.halo_max, nh);
    R.local_max = std::max(R.local_max, rows + nh);
    H.halo0[g + 1] = (int32_t)hsum;
    H.slice0[g + 1] = H.slice0[g] + (int32_t)width[g].size();
  }
  R.halo_max = (R.halo_max + 1) & ~1;
  const size_t fixed = (size_t)R.local_max * 8 + (size_t)R.halo_max * 4 + 64;
  if (fixed > smem_limit) return;
  size_t left = smem_limit - fixed;
  const size_t vec = (size_t)R.rows_max * 8;
  R.vectors = 4 * vec <= left ? 4 : 2 * vec <= left ? 2 : 0;
  if (R.vectors < 4) R.threads = 1024;  // the only form built
  left -= R.vectors * vec;
  H.slice_at.assign(H.slice0[G] + 1, 0);
  int64_t at = 0, block = 0;
  for (int g = 0; g < G; ++g) {
    const int64_t first = at;
    for (size_t s = 0; s < width[g].size(); ++s) {
      H.slice_at[H.slice0[g] + s] = (int32_t)at;
      at += width[g][s];
    }
    block = std::max(block, (at - first) * 32);
    if (at >= INT32_MAX / 32) return;
  }
  H.slice_at[H.slice0[G]] = (int32_t)at;
  R.cache = (int32_t)std::min<int64_t>(block, (int64_t)(left / 10) & ~31ll);
  R.smem = fixed + R.vectors * vec + (size_t)R.cache * 10;
  H.halo.resize(hsum);
  H.val.resize((size_t)at * 32);
  H.col.resize((size_t)at * 32);
  over([&](int g) {
    const int32_t a = H.row0[g], b = H.row0[g + 1];
    const std::vector<int32_t>& h = hal[g];
    std::copy(h.begin(), h.end(), H.halo.begin() + H.halo0[g]);
    const uint16_t* lc = local[g].data();
    for (int32_t s = H.slice0[g]; s < H.slice0[g + 1]; ++s) {
      const int64_t e0 = (int64_t)H.slice_at[s] * 32;
      const int w = H.slice_at[s + 1] - H.slice_at[s];
      for (int l = 0; l < 32; ++l) {
        const int32_t i = a + (s - H.slice0[g]) * 32 + l;
        const int64_t v = i < b ? H.node_of[i] : -1;
        const int n = i < b ? len(v) : 0;
        const double* v0 = i < b ? row(v).second : nullptr;
        for (int k = 0; k < w; ++k) {
          H.val[e0 + k * 32 + l] = k < n ? v0[k] : 0.0;
          H.col[e0 + k * 32 + l] = k < n ? lc[k] : (uint16_t)0;
        }
        lc += n;
      }
    }
  });
  H.fits = true;
}

}  // namespace

