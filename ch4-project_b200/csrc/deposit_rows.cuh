// Two-way momentum deposit by lattice rows (included by particles.cuh inside namespace ch4).
//
// src/lagrange_feedback.c:11-256: the particle loop adds fac * fp * vol of every particle to
// the 8 cells of its stencil.  Here every particle is listed under the row segment its home cell
// lies in -- at most ROW_SEG cells of one (y, z) row -- and one warp owns one segment of a lattice
// row: it merges the lists of the four home rows around it in particle-index order and adds
// every particle to the two cells it has in the row, in shared memory.  Each cell thus sums its
// particles in the reference's order whatever the schedule, and no array runs over the home
// cells.
//
// The lists are built by counting: a particle draws its place in its list from a counter (the
// sub-step that has just moved it does), a pass over the lists gives each its range, a pass over
// the particles fills them in, and a last one puts every list in particle-index order -- the
// order of the draws is the schedule's, the lists and sums are not.
//
// Rows longer than ROW_SEG are cut into segments of ROW_CUT cells.  A segment's last cell also takes
// from the next segment's first home cell; the particles of that home are listed a second time, in
// an edge list of their own, so that no warp reads the next segment's whole list for them.  us a step
// FP32, by home cells / rows with the next segment's list merged whole / with edge lists and 256
// cells a segment / 128: 512x128x64 with 0.06 particles a cell 442 / 495 / 404 / 384, with 0.25 776 /
// 1,265 / 829 / 720, with 0.008 351 / 290 / 288 / 294; 300x128x96 (256 + 44 cells left half of the
// warps with most of the work) with 0.11 476 / 605 / 499 / 412.
//
// Why rows: at the workloads' 0.04 depositing particles per cell nearly every home cell is
// empty, and a list per home cell (a range of 8 bytes each, cleared, filled, read and scanned
// every step) moved more bytes than the particles; a row of 256 cells has some 10 particles a
// list.  Measured, us a step, home cells -> rows: 250,000 particles in 160^3 FP32 505 -> 431,
// 15,000 in 60x50x70 FP64 164 -> 109 (re-sort every 16 steps and only of the planes that differ
// included); the lists by radix sort -> by counting: 390 -> 347 and 85 -> 53, 800,000 in 240^3
// 1,155 -> 1,073 (four launches of the sort and the copy of the records into its order gone).
#pragma once

constexpr int ROW_SEG = 256;    // cells of a row that one warp owns, at most
constexpr int ROW_CUT_SHIFT = 7, ROW_CUT = 1 << ROW_CUT_SHIFT;  // cells of a segment of a longer row
constexpr int ROW_CHUNK = 64;   // merged entries in shared memory at a time
constexpr int ROW_WARPS = 4;    // warps per block
constexpr int ROW_REC = 10;     // doubles of a record: fac*fp (3), dxm dxp dym dyp dzm dzp, hx (as int)

// the segments of a row of NX cells: all of `len` cells but for the last; the last home cell (hx =
// NX) belongs to the last segment
inline RowSegs row_segs(int NX) {
  if (NX <= ROW_SEG) return {1, NX, 31};
  return {(NX + ROW_CUT - 1) / ROW_CUT, ROW_CUT, ROW_CUT_SHIFT};
}
// lists of one home row: its segments', then the edge lists of the first home cells of segments
// 1 .. (home len s is the first of segment s)
__host__ __device__ __forceinline__ unsigned int row_lists(const RowSegs& g) { return 2u * (unsigned)g.n - 1u; }
inline unsigned int row_bins(const RowSegs& g, int NY, int NZ) {
  return row_lists(g) * (unsigned)(NY + 1) * (unsigned)(NZ + 1);
}
__host__ __device__ __forceinline__ int row_seg(int hx, const RowSegs& g) {
  const int s = hx >> g.shift;
  return s < g.n ? s : g.n - 1;
}
// the list of a home cell, and its edge list or -1
__host__ __device__ __forceinline__ int row_bin(int hx, int hy, int hz, const RowSegs& g, int NY) {
  return (int)(((unsigned)hz * (unsigned)(NY + 1) + (unsigned)hy) * row_lists(g)) + row_seg(hx, g);
}
__host__ __device__ __forceinline__ int row_edge_bin(int hx, int hy, int hz, const RowSegs& g, int NY) {
  const int s = row_seg(hx, g);
  if (s == 0 || hx != s * g.len) return -1;
  return (int)(((unsigned)hz * (unsigned)(NY + 1) + (unsigned)hy) * row_lists(g)) + g.n + s - 1;
}
// places of a particle: one, and with edge lists a second
__host__ __device__ __forceinline__ int row_places(const RowSegs& g) { return g.n > 1 ? 2 : 1; }

// The longest list with which the deposit still goes by rows, and (row_resume) the one with which
// it returns to them.  One warp walks a row's merged entries one after the other, while by home cells
// every cell has a thread of its own, so rows lose once lists are long, whether the particles are
// dense or gathered in a few rows.  us a step by home cells / by rows, FP32, by mean list (with
// particles spread evenly the longest of a lattice is some four deviations more: 97 for 64, 135 for 96):
//   64^3 24: 174 / 90, 64: 216 / 194, 80: 239 / 233, 128: 281 / 364;  128^3 64: 655 / 633, 96: 834 /
//   901;  160^3 16: 506 / 426, 64: 1,021 / 1,010, 96: 1,304 / 1,422;  60x50x70 FP64 32: 203 / 126,
//   64: 236 / 209, 96: 262 / 291.  Rows cut into segments, 512x128x64 32: 777 / 719, 48: 991 / 968;
//   300x128x96 55: 957 / 967.
//   Gathered in 160^3: 170,000 between two planes (longest some 600) 407 / 630, a million 763 /
//   2,805; in 64 clusters (some 200) 548 / 494, the one case seen that the limit costs; in 256
//   (some 60) 416 / 344.
__host__ __device__ __forceinline__ int row_limit(const RowSegs& g) { return g.n == 1 ? 120 : 80; }
__host__ __device__ __forceinline__ int row_resume(const RowSegs& g) { return row_limit(g) * 3 / 4; }

#ifdef __CUDACC__

// Deposit record and place in its list of one particle (src/lagrange_feedback.c:34-118).  The
// last sub-step of a step calls it with the state it has in registers; a and D (acceleration
// and Du/Dt) are read from the state where `have` is not set.
template <typename A>
__device__ __forceinline__ void deposit_rows_emit(const PartParams<A>& P, int ip, double x, double y, double z,
                                                  double beta, bool have, const double* a, const double* D) {
  const double* pf = P.pf;
  const long long np = P.np;
#define F(name) pf[CH4_PF(name) * np + ip]
  Stencil t;
  double px, py, pz;
  const bool inside = wrapped_position(P, x, y, z, px, py, pz);
  make_stencil(px, py, pz, t);
  const double fac = pf[PF_VOL * np + ip];
  const bool live = inside && (fac > 0.0) && beta != 0.0;
  const int hx = t.im + 1, hy = t.jm + 1, hz = t.km + 1;
  if (P.segs.n > 1) {
    const int edge = live ? row_edge_bin(hx, hy, hz, P.segs, P.NY) : -1;
    P.row_place[np + ip] = make_int2(edge, edge < 0 ? 0 : atomicAdd(P.row_count + edge, 1));
  }
  if (!live) {
    P.row_place[ip] = make_int2(-1, 0);
    return;
  }
  const int bin = row_bin(hx, hy, hz, P.segs, P.NY);
  P.row_place[ip] = make_int2(bin, atomicAdd(P.row_count + bin, 1));
  const double dr = pf[PF_DR * np + ip];
  double aa[3], DD[3];
  if (have) {
#pragma unroll
    for (int q = 0; q < 3; q++) aa[q] = a[q], DD[q] = D[q];
  } else {
    aa[0] = F(ax), aa[1] = F(ay), aa[2] = F(az);
    DD[0] = F(Dt_ux), DD[1] = F(Dt_uy), DD[2] = F(Dt_uz);
  }
#undef F
  // gravity_vector of src/lagrange_feedback.c:95-103 (y points down)
  const double g[3] = {P.gravity ? P.g[0] : 0.0, P.gravity ? -P.g[1] : 0.0, P.gravity ? P.g[2] : 0.0};
  double f[3];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    if (P.twoway_stau) f[q] = fac * ((DD[q] - g[q]) * (1 - dr));  // src/lagrange_feedback.c:106-110
    else f[q] = fac * (DD[q] - g[q] + dr * (g[q] - aa[q]));
  }
  double2* r = reinterpret_cast<double2*>(P.rec + (long long)ip * ROW_REC);
  r[0] = make_double2(f[0], f[1]);
  r[1] = make_double2(f[2], t.dxm);
  r[2] = make_double2(t.dxp, t.dym);
  r[3] = make_double2(t.dyp, t.dzm);
  r[4] = make_double2(t.dzp, __hiloint2double(0, hx));
}

// the same from the state (a resumed run's first deposit; random re-entry, which moves
// particles after the sub-step)
template <typename A>
__global__ void deposit_rows_prepare_kernel(const PartParams<A> P) {
  grid_chain();
  const int ip = blockIdx.x * blockDim.x + threadIdx.x;
  if (ip >= P.np) return;
  const long long np = P.np;
  deposit_rows_emit(P, ip, P.pf[CH4_PF(x) * np + ip], P.pf[CH4_PF(y) * np + ip], P.pf[CH4_PF(z) * np + ip],
                    P.pf[CH4_PF(beta_coeff) * np + ip], false, (const double*)nullptr, (const double*)nullptr);
}

// the range of every list (bins of a warp together, at a place drawn from *cursor), the counters
// cleared for the next sub-step; the longest list beyond `limit` to *longest
static __global__ void row_ranges_kernel(int* count, unsigned int nb, int2* list, int* cursor, int limit, int* longest) {
  grid_chain();
  const unsigned int b = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int c = b < nb ? count[b] : 0;
  int sum = c;  // inclusive prefix
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, sum, d);
    if ((int)lane >= d) sum += v;
  }
  const int most = __reduce_max_sync(0xffffffffu, c);
  if (lane == 0 && most > limit) atomicMax(longest, most);
  int base = 0;
  if (lane == 31 && sum > 0) base = atomicAdd(cursor, sum);
  base = __shfl_sync(0xffffffffu, base, 31) + sum - c;
  if (b < nb) {
    list[b] = make_int2(base, base + c);
    if (c) count[b] = 0;
  }
}

// the particles into their lists, as {index, slot}
static __global__ void row_fill_kernel(const int2* place, int places, const int2* list, const int* pid, int np,
                                       int2* entry, int* cursor) {
  grid_chain();
  const int ip = blockIdx.x * blockDim.x + threadIdx.x;
  if (ip == 0) *cursor = 0;  // for the next deposit
  if (ip >= np) return;
  for (int k = 0; k < places; k++) {
    const int2 p = place[(long long)k * np + ip];
    if (p.x >= 0) entry[list[p.x].x + p.y] = make_int2(pid[ip], ip);
  }
}

// every list in particle-index order, a warp per list: up to 32 entries ranked in registers, more
// by a bitonic merge sort in place (for any length: an exchange with a partner beyond the end is
// left out, as such a partner would be larger)
static __global__ void row_order_kernel(const int2* list, unsigned int nb, int2* entry) {
  grid_chain();
  const unsigned int b = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (b >= nb) return;
  const int2 l = list[b];
  const int n = l.y - l.x;
  if (n < 2) return;
  int2* const e = entry + l.x;
  if (n <= 32) {
    const int2 v = (int)lane < n ? e[lane] : make_int2(0x7fffffff, 0);
    int rank = 0;
    for (int q = 0; q < n; q++) rank += __shfl_sync(0xffffffffu, v.x, q) < v.x ? 1 : 0;
    if ((int)lane < n) e[rank] = v;
    return;
  }
  for (long long k = 2; k < 2LL * n; k <<= 1) {  // runs of k from runs of k / 2
    for (long long j = k >> 1; j > 0; j >>= 1) {
      // the first exchange of a merge mirrors the second run, the others are at distance j
      for (long long i = lane; i < n; i += 32) {
        const long long q = j == k >> 1 ? (i | (k - 1)) - (i & (k - 1)) : i ^ j;
        if (q > i && q < n) {
          const int2 a = e[i], c = e[q];
          if (a.x > c.x) e[i] = c, e[q] = a;
        }
      }
      __syncwarp();
    }
  }
}

// shared memory of one warp: the contributions by merged position (component c of corner di
// at 2 c + di), the row's sums (three rows of `cells`), indices and cells of the merged entries
__host__ __device__ __forceinline__ int row_cells(const RowSegs& g) { return g.len + 1; }  // and a spare one
__host__ __device__ __forceinline__ int row_shared(const RowSegs& g) {
  return ROW_CHUNK * 6 * 8 + 3 * row_cells(g) * 8 + ROW_CHUNK * 3 * 4;
}

// what a record of list l adds to the two cells it has in the row of n cells: component c of
// corner di at o[2 c + di], its cell (the one of corner 1 comes before) at at[di]; a cell outside
// the row is `spare`, which is never read
__device__ __forceinline__ void row_entry(const double2* r, int l, int x0, int n, int spare, double* o, int* at) {
  const double wy = (l & 1) ? r[3].x : r[2].y;         // dyp : dym
  const double wz = ((l >> 1) & 1) ? r[4].x : r[3].y;  // dzp : dzm
  const double v0 = r[1].y * wy * wz, v1 = r[2].x * wy * wz;
  o[0] = r[0].x * v0;
  o[1] = r[0].x * v1;
  o[2] = r[0].y * v0;
  o[3] = r[0].y * v1;
  o[4] = r[1].x * v0;
  o[5] = r[1].x * v1;
  const unsigned int c0 = (unsigned)(__double2loint(r[4].y) - x0), c1 = c0 - 1u;
  at[0] = c0 < (unsigned)n ? (int)c0 : spare;
  at[1] = c1 < (unsigned)n ? (int)c1 : spare;
}

// the merged entries in particle order: lane 2 c + di adds component c to the corner di
__device__ __forceinline__ void row_accumulate(int merged, int lane, int cells, const double* con, const int* s_at,
                                               double* acc) {
  if (lane < 6) {
    double* const mine = acc + (lane >> 1) * cells;
    const int* at = s_at + (lane & 1);
    const double* v = con + lane;
#pragma unroll 4
    for (int e = 0; e < merged; e++) {
      mine[at[2 * e]] += v[6 * e];
      __syncwarp(0x3f);
    }
  }
  __syncwarp();
}

// nl: lists of a warp, 4, or 8 where rows are cut
template <typename A, int nl>
__global__ void __launch_bounds__(32 * ROW_WARPS) deposit_rows_kernel(const PartParams<A> P) {
  grid_chain();
  extern __shared__ double row_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, cells = row_cells(P.segs);
  double* const con = row_smem + warp * (row_shared(P.segs) / 8);
  double* const acc = con + ROW_CHUNK * 6;
  int* const s_pid = reinterpret_cast<int*>(acc + 3 * cells);
  int* const s_at = s_pid + ROW_CHUNK;
  const int ns = nl == 4 ? 1 : P.segs.n;
  const unsigned int w = blockIdx.x * ROW_WARPS + warp;  // of plane k's ns * NY
  const int j = (int)(nl == 4 ? w : w / (unsigned)ns), seg = (int)w - j * ns, k = blockIdx.y;
  if (j >= P.NY) return;  // whole warps: no block barrier below
  const int x0 = seg * P.segs.len, n = min(P.segs.len, P.NX - x0);
  A* out = P.dep + ((long long)k * P.NY + j) * P.NX + x0;
  // lane l < 4: the home row (y + (l & 1), z + (l >> 1)) of this segment; 4 <= l < 8: the same
  // rows' edge list, of the next segment's first home cell
  int beg = 0, end = 0;
  if (lane < nl && (lane < 4 || seg + 1 < ns)) {
    const unsigned int b = ((unsigned)(k + ((lane >> 1) & 1)) * (unsigned)(P.NY + 1) + (unsigned)(j + (lane & 1))) *
                               row_lists(P.segs) + (unsigned)(lane < 4 ? seg : ns + seg);
    const int2 range = P.row_list[b];
    beg = range.x;
    end = range.y;
  }
  constexpr unsigned ALL = 0xffffffffu;
  if (__any_sync(ALL, beg < end)) {
    for (int c = lane; c < n; c += 32) acc[c] = acc[cells + c] = acc[2 * cells + c] = 0.0;
    const int all = __reduce_add_sync(ALL, end - beg);
    if (all <= 32) {
      // one entry per lane, ranked by comparing it with every other
      int off = end - beg;
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) {
        const int v = __shfl_up_sync(ALL, off, d);
        if (lane >= d && lane < 8) off += v;
      }
      off -= end - beg;
      int l = 0;
      for (int q = 1; q < nl; q++)  // the last list that begins at or before this lane
        if (__shfl_sync(ALL, off, q) <= lane) l = q;
      const int pos = __shfl_sync(ALL, beg, l) - __shfl_sync(ALL, off, l) + lane;
      const bool on = lane < all;
      const int2 who = on ? P.row_entry[pos] : make_int2(0x7fffffff, 0);
      const double2* r = reinterpret_cast<const double2*>(P.rec + (long long)who.y * ROW_REC);
      double2 e[5];
#pragma unroll
      for (int q = 0; q < 5; q++) e[q] = r[q];
      const int pid = who.x;
      int rank = 0;
      for (int q = 0; q < all; q++) rank += __shfl_sync(ALL, pid, q) < pid ? 1 : 0;
      if (on) row_entry(e, l, x0, n, cells - 1, con + 6 * rank, s_at + 2 * rank);
      __syncwarp();
      row_accumulate(all, lane, cells, con, s_at, acc);
      beg = end;
    }
    // chunks of the merge: up to cap entries of each list; with entries left behind, only those
    // up to the smallest index T that ends a cut list are merged now
    while (__any_sync(ALL, beg < end)) {
      const int left = __reduce_add_sync(ALL, end - beg);
      // (an edge list holds the particles of one home cell, the others those of a segment's)
      const int cap = left <= ROW_CHUNK ? ROW_CHUNK : nl == 4 ? ROW_CHUNK / 4 : lane < 4 ? ROW_CHUNK / 4 - 2 : 2;
      const int cnt = min(end - beg, cap);
      int off = cnt;  // inclusive prefix over the lists, then exclusive
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) {
        const int v = __shfl_up_sync(ALL, off, d);
        if (lane >= d && lane < 8) off += v;
      }
      const int total = __shfl_sync(ALL, off, 7);
      off -= cnt;
      for (int e = lane; e < ROW_CHUNK; e += 32) {
        const bool on = e < total;
        int l = 0;
        for (int q = 1; q < nl; q++)  // the last list that begins at or before e
          if (__shfl_sync(ALL, off, q) <= e) l = q;
        const int base = __shfl_sync(ALL, beg, l) - __shfl_sync(ALL, off, l);
        if (on) s_pid[e] = P.row_entry[base + e].x;
      }
      __syncwarp();
      const bool cut = lane < 8 && end - beg > cnt;
      const int T = __reduce_min_sync(ALL, cut ? s_pid[off + cnt - 1] : 0x7fffffff);
      for (int e = lane; e < ROW_CHUNK; e += 32) {
        const int pid = e < total ? s_pid[e] : 0x7fffffff;
        const bool on = e < total && pid <= T;
        int rank = 0, l = 0;
        for (int q = 0; q < nl; q++) {  // entries of list q below this one (its own: its position)
          const int a = __shfl_sync(ALL, off, q), c = __shfl_sync(ALL, cnt, q);
          if (a <= e) l = q;
          if (!on) continue;
          int lo = 0, hi = c;
          while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (s_pid[a + mid] < pid) lo = mid + 1;
            else hi = mid;
          }
          rank += lo;
        }
        const int base = __shfl_sync(ALL, beg, l) - __shfl_sync(ALL, off, l);
        if (on) {
          const double2* r = reinterpret_cast<const double2*>(P.rec + (long long)P.row_entry[base + e].y * ROW_REC);
          const double2 v[5] = {r[0], r[1], r[2], r[3], r[4]};
          row_entry(v, l, x0, n, cells - 1, con + 6 * rank, s_at + 2 * rank);
        }
      }
      // how many entries of each list were merged: those up to T
      int done = cnt;
      if (lane < 8) {
        int lo = 0, hi = cnt;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s_pid[off + mid] <= T) lo = mid + 1;
          else hi = mid;
        }
        done = lo;
      }
      const int merged = __reduce_add_sync(ALL, lane < 8 ? done : 0);
      __syncwarp();
      row_accumulate(merged, lane, cells, con, s_at, acc);
      beg += done;
    }
    for (int c = lane; c < n; c += 32) {
      out[c] = (A)acc[c];
      out[P.N + c] = (A)acc[cells + c];
      out[2 * P.N + c] = (A)acc[2 * cells + c];
    }
  } else {
    for (int c = lane; c < n; c += 32) out[c] = out[P.N + c] = out[2 * P.N + c] = A(0);
  }
}

#endif  // __CUDACC__
