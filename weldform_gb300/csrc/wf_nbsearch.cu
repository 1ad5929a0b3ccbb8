// Neighbour search of the kick-drift step on sm_103a.
//
// Replaces the reference's linked-list cell search (Neighbour.cpp:10-477) and
// pair-list flattening (CalcPairPosList, Neighbour.cpp:617-694):
//   1. k_cell_keys   — reference cell index (ListGenerate, Neighbour.cpp:183-227:
//                      floor((x - BLPF) / CellSize), clamped) mapped to the cell's
//                      Morton rank; histogram per cell.
//   2. exclusive scan of the histogram -> cell start offsets.
//   3. k_scatter + k_sort_bricks — counting-sort scatter into the cells' lists,
//                      then each brick of cells stored in original particle
//                      index order (deterministic; see k_sort_bricks).
//   4. k_permute / k_copy_back — every persistent state column reordered.
//   5. k_nbr_fill    — one warp per particle scans the 27 neighbouring cells,
//                      applies the reference pair rules (AllocateNbPair,
//                      Neighbour.cpp:374-417: contact-surface pairs, radius test
//                      CheckRadius :361-372, free + same material) and writes its
//                      row in canonical order (j > i ascending, then j < i
//                      ascending by original index) into an ELL array
//                      (entry k of particle i at k * N + i).
// With the Verlet-skin reuse, a full search (steps 1-5) also builds each
// particle's superset over a 5 x 5 x 5 stencil at the pair radius plus the
// skin (k_nbr_fill<true>), and a later search whose particles all moved less
// than half the skin skips steps 1-5 and filters the supersets with the same
// exact rules (k_skin_check, k_nbr_filter).
// The radius test rij / h <= Cellfac is decided bit-exactly: an FP32 distance
// prefilter with a proven-safe relative margin accepts or rejects clear cases,
// and everything inside the margin is decided by the reference's FP64
// expression evaluated with non-contracted IEEE operations.
//
// Every kernel checks st->do_search first (the re-sorting ones also
// search_full), so the search can sit inside a captured step and cost only
// an empty launch on steps that do not rebuild.
#include "wf_launch.h"
#include "wf_step_common.cuh"

namespace wf {

__device__ __forceinline__ bool searching(const DevPtrs& P) { return P.st->do_search != 0; }
// The parts of a search that re-sort the particles run only when the search
// is a full one (always, unless the Verlet-skin reuse is on).
__device__ __forceinline__ bool searching_full(const DevPtrs& P) {
  return P.st->do_search != 0 && P.st->search_full != 0;
}

// A particle with a non-finite coordinate cannot pass CheckRadius with any
// other (its distance is NaN or infinite), so its row is empty and it is in
// no other row.  The reference bins it into a clamped edge cell
// (Neighbour.cpp:185-218), where every later search scans all such particles
// pairwise.  Here it goes to one of ncells shadow buckets after the grid's
// (key ncells + original index mod ncells), which no stencil visits: the rows
// are the same and the search stays linear.  The shadow buckets are sorted
// like cells, so the order stays deterministic.
__global__ void k_cell_keys(DevPtrs P, DomainConst K) {
  if (!searching_full(P)) return;
  int nonfinite = 0;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < K.N; p += gridDim.x * blockDim.x) {
  int c[3];
  bool finite = true;
  for (int d = 0; d < 3; ++d) {
    double xd = P.f[(C_X + d) * (size_t)K.N + p];
    finite = finite && isfinite(xd);
    int q = (int)floor(__ddiv_rn(__dsub_rn(xd, K.BLPF[d]), K.CellSize[d]));
    if (q < 0) q = 0;
    if (q >= K.CellNo[d]) q = K.CellNo[d] - 1;
    c[d] = q;
  }
  int key;
  if (finite) {
    key = P.cell_rank[(c[0] * K.CellNo[1] + c[1]) * K.CellNo[2] + c[2]];
  } else {
    key = K.ncells + P.i[I_ORIG * (size_t)K.N + p] % K.ncells;
    ++nonfinite;
  }
  P.i[I_CELL * (size_t)K.N + p] = key;
  atomicAdd(&P.cell_count[key], 1);
  }
  if (nonfinite) {
    atomicAdd(&P.st->nan_count, nonfinite);
    if (K.nan_check) atomicOr(&P.st->errors, ERR_NAN);
  }
}

// Batched domain, before the reordering (a full search): the rows of
// particles whose specimen does not search this step are saved by old
// position, each entry as the neighbour's original index (with the
// larger-index bit), so k_nbr_fill can put them back at the particles' new
// positions.
__global__ void k_rows_save(DevPtrs P, DomainConst K) {
  if (!searching_full(P)) return;
  const size_t N = K.N;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < K.N; p += gridDim.x * blockDim.x) {
    if (P.sp[P.i[I_SPEC * N + p]].do_search) continue;
    int len = P.row_len[p];
    P.save_len[p] = len;
    for (int k = 0; k < len; ++k) {
      int e = P.nbr[(size_t)k * N + p];
      P.save_nbr[(size_t)k * N + p] = P.i[I_ORIG * N + nb_index(e)] | (int)((unsigned)e & NB_UP);
    }
  }
}

// ---- exclusive scan of an int array into an int array (three phases) ------
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ long long block_exclusive_scan(long long v, long long* sh, long long* total) {
  // Hillis-Steele over a power-of-two block; deterministic.
  int t = threadIdx.x;
  sh[t] = v;
  __syncthreads();
  for (int off = 1; off < blockDim.x; off <<= 1) {
    long long add = (t >= off) ? sh[t - off] : 0;
    __syncthreads();
    sh[t] += add;
    __syncthreads();
  }
  long long incl = sh[t];
  *total = sh[blockDim.x - 1];
  __syncthreads();
  return incl - v;
}

__global__ void k_scan_reduce(DevPtrs P, const int* in, long long n, long long* tot) {
  if (!searching_full(P)) return;
  __shared__ long long sh[SCAN_THREADS];
  long long base = (long long)blockIdx.x * SCAN_TILE;
  long long s = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    long long idx = base + (long long)threadIdx.x * SCAN_ITEMS + k;
    if (idx < n) s += in[idx];
  }
  long long total;
  block_exclusive_scan(s, sh, &total);
  if (threadIdx.x == 0) tot[blockIdx.x] = total;
}
__global__ void k_scan_top(DevPtrs P, long long* tot, int nb) {
  if (!searching_full(P)) return;
  __shared__ long long sh[SCAN_THREADS];
  long long carry = 0;
  for (int base = 0; base < nb; base += SCAN_THREADS) {
    int idx = base + threadIdx.x;
    long long v = (idx < nb) ? tot[idx] : 0;
    long long total;
    long long ex = block_exclusive_scan(v, sh, &total);
    if (idx < nb) tot[idx] = ex + carry;
    carry += total;
    __syncthreads();
  }
}
// The counts are zeroed as they are read: the scatter uses them as cursors next.
__global__ void k_scan_down(DevPtrs P, int* in, long long n, const long long* tot, int* out, int* total_out) {
  if (!searching_full(P)) return;
  __shared__ long long sh[SCAN_THREADS];
  long long base = (long long)blockIdx.x * SCAN_TILE;
  long long vals[SCAN_ITEMS];
  long long s = 0;
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    long long idx = base + (long long)threadIdx.x * SCAN_ITEMS + k;
    vals[k] = (idx < n) ? in[idx] : 0;
    if (idx < n) in[idx] = 0;
    s += vals[k];
  }
  long long total;
  long long ex = block_exclusive_scan(s, sh, &total) + tot[blockIdx.x];
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    long long idx = base + (long long)threadIdx.x * SCAN_ITEMS + k;
    if (idx < n) out[idx] = (int)ex;
    ex += vals[k];
  }
  if (total_out && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) *total_out = (int)ex;
}

// The three phases by one block, for grids of a few tiles.
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_one(DevPtrs P, int* in, int n, int* out, int* total_out) {
  if (!searching_full(P)) return;
  __shared__ long long sh[SCAN_THREADS];
  long long carry = 0;
  for (int base = 0; base < n; base += SCAN_TILE) {
    int v[SCAN_ITEMS];
    long long s = 0, total;
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      const int idx = base + (int)threadIdx.x * SCAN_ITEMS + k;
      v[k] = idx < n ? in[idx] : 0;
      if (idx < n) in[idx] = 0;
      s += v[k];
    }
    long long ex = block_exclusive_scan(s, sh, &total) + carry;
    for (int k = 0; k < SCAN_ITEMS; ++k) {
      const int idx = base + (int)threadIdx.x * SCAN_ITEMS + k;
      if (idx < n) out[idx] = (int)ex;
      ex += v[k];
    }
    carry += total;
  }
  if (threadIdx.x == 0) *total_out = (int)carry;
}

__global__ void k_scatter(DevPtrs P, DomainConst K) {
  if (!searching_full(P)) return;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < K.N; p += gridDim.x * blockDim.x) {
  int key = P.i[I_CELL * (size_t)K.N + p];
  int pos = P.cell_start[key] + atomicAdd(&P.cell_count[key], 1);
  P.perm[pos] = p;
  }
}

// Storage order: within each brick of cells (DevPtrs::brick_cell) the particles
// in ascending original index.  A generator lays its lattice down row by row,
// so the brick's rows along x come out whole and the k-th neighbours of a
// warp's 32 consecutive particles are runs of consecutive records: 6 cache
// lines per warp-wide 16-byte load, against 12 with the particles of one cell
// after the other (the L1 data pipe of the acceleration gather at 982,072
// particles went from 87 to 54 % of its rate).  One block per brick sorts its
// slots by a bitonic sort in shared memory, writes the particles in their
// order (perm) and where each slot of the cells' lists went (cell_list), since
// a cell's particles are no longer contiguous.  A brick that has come to hold
// more than BRICK_CAP particles (a body that left the grid is binned into its
// edge cells) is taken in parts of whole cells that fit, and a cell that does
// not fit by itself ranks its slots by counting the smaller keys tile by tile.
// Shadow buckets are grouped into bricks as well.
// Where the numbering does not run through space (DomainConst::cell_order) the
// key begins with the cell, so that a brick's particles lie cell by cell.
constexpr int BRICK_T = 1024;
constexpr int BRICK_PER = BRICK_CAP / BRICK_T;  // slots per thread
__global__ void __launch_bounds__(BRICK_T) k_sort_bricks(DevPtrs P, DomainConst K) {
  if (!searching_full(P)) return;
  __shared__ unsigned long long kv[BRICK_CAP];  // (cell of the brick,) original index, slot
  const int t = threadIdx.x;
  const int* orig = P.i + I_ORIG * (size_t)K.N;
  const int* cell = P.i + I_CELL * (size_t)K.N;
  static_assert(BRICK_CAP <= 1 << 12, "a slot in 12 bits of the key");
  for (int b = blockIdx.x; b < K.nbricks; b += gridDim.x)
  for (int c0 = P.brick_cell[b], c1 = P.brick_cell[b + 1], ce; c0 < c1; c0 = ce) {  // uniform over the block
    const int s0 = P.cell_start[c0];
    ce = c1;
    if (P.cell_start[c1] - s0 > BRICK_CAP) {  // as many cells as fit, one at least (a brick has up to 256)
      const int fit = __syncthreads_count(c0 + t < c1 && P.cell_start[c0 + t + 1] - s0 <= BRICK_CAP);
      ce = c0 + (fit > 1 ? fit : 1);
    }
    const int n = P.cell_start[ce] - s0;
    if (n <= 0) continue;
    if (n <= BRICK_CAP) {
      int P2 = 2;
      while (P2 < n) P2 <<= 1;
      for (int e = t; e < P2; e += BRICK_T) {
        unsigned long long v = ~0ull;
        if (e < n) {
          const int q = P.perm[s0 + e];
          v = ((unsigned long long)(unsigned)orig[q] << 12) | (unsigned)e;
          if (K.cell_order) v |= (unsigned long long)(cell[q] - c0) << 44;
        }
        kv[e] = v;
      }
      __syncthreads();
      for (int size = 2; size <= P2; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          for (int e = t; e < P2 / 2; e += BRICK_T) {
            const int lo = 2 * e - (e & (stride - 1)), hi = lo + stride;
            const unsigned long long x = kv[lo], y = kv[hi];
            if ((x > y) == ((lo & size) == 0)) { kv[lo] = y; kv[hi] = x; }
          }
          __syncthreads();
        }
      int p[BRICK_PER];
#pragma unroll
      for (int r = 0; r < BRICK_PER; ++r) {
        const int q = t + r * BRICK_T;
        if (q < n) {
          const int e = (int)(kv[q] & 0xfffu);
          p[r] = P.perm[s0 + e];
          P.cell_list[s0 + e] = s0 + q;
        }
      }
      __syncthreads();  // every slot of perm read before any is written
#pragma unroll
      for (int r = 0; r < BRICK_PER; ++r)
        if (t + r * BRICK_T < n) P.perm[s0 + t + r * BRICK_T] = p[r];
    } else {
      int* key = reinterpret_cast<int*>(kv);
      int* tmp = P.i + I_TMP * (size_t)K.N;
      for (int g = 0; g < n; g += BRICK_CAP) {
        int k[BRICK_PER], rank[BRICK_PER];
#pragma unroll
        for (int r = 0; r < BRICK_PER; ++r) {
          const int e = g + t + r * BRICK_T;
          k[r] = e < n ? orig[P.perm[s0 + e]] : 0;
          rank[r] = 0;
        }
        for (int h = 0; h < n; h += BRICK_CAP) {
          const int m = n - h < BRICK_CAP ? n - h : BRICK_CAP;
          __syncthreads();
          for (int e = t; e < m; e += BRICK_T) key[e] = orig[P.perm[s0 + h + e]];
          __syncthreads();
          for (int q = 0; q < m; ++q) {
            const int v = key[q];
#pragma unroll
            for (int r = 0; r < BRICK_PER; ++r) rank[r] += v < k[r];
          }
        }
#pragma unroll
        for (int r = 0; r < BRICK_PER; ++r) {
          const int e = g + t + r * BRICK_T;
          if (e < n) { tmp[s0 + rank[r]] = P.perm[s0 + e]; P.cell_list[s0 + e] = s0 + rank[r]; }
        }
      }
      __syncthreads();
      for (int e = t; e < n; e += BRICK_T) P.perm[s0 + e] = tmp[s0 + e];
    }
    // the cells' counts (the scatter's cursors) back to zero for the next search
    for (int c = c0 + t; c < ce; c += BRICK_T) P.cell_count[c] = 0;
    __syncthreads();  // the shared keys are reused by the next cells
  }
}

// Gather every persistent column into the scratch arenas (new order).  A
// fixed grid strides over (column, particle) so the launch costs nothing on
// steps that do not search.
__global__ void k_permute(DevPtrs P, DomainConst K, double* fdst, int* idst) {
  if (!searching_full(P)) return;
  size_t N = K.N;
  size_t total = (size_t)(NF64_PERSIST + NI32_PERSIST) * N;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < total; k += (size_t)gridDim.x * blockDim.x) {
    size_t col = k / N, p = k - col * N;
    int src = P.perm[p];
    if (col < (size_t)NF64_PERSIST) fdst[col * N + p] = P.f[col * N + src];
    else {
      size_t c = col - NF64_PERSIST;
      idst[c * N + p] = P.i[c * N + src];
    }
  }
}
__global__ void k_copy_back(DevPtrs P, DomainConst K, const double* fsrc, const int* isrc) {
  if (!searching_full(P)) return;
  size_t nf = (size_t)NF64_PERSIST * K.N, ni = (size_t)NI32_PERSIST * K.N;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < nf + ni; k += (size_t)gridDim.x * blockDim.x) {
    if (k < nf) P.f[k] = fsrc[k];
    else P.i[k - nf] = isrc[k - nf];
  }
}

__device__ __forceinline__ bool is_contact_id(const DomainConst& K, int id) {
  for (int m = 0; m < K.nmeshes; ++m)
    if (id == K.contact_surf_id[m]) return true;
  return false;
}

// The FP32 prefilter coordinates of particle p, and its cell coordinates at the
// current positions (ListGenerate's clamped cell index, Neighbour.cpp:185-218,
// the same FP64 expression as k_cell_keys), 21 bits per axis, -1 for a
// non-finite position.  COVER: the filter leaves the cell test out, so only
// the finiteness is recorded.
template <bool COVER>
__device__ __forceinline__ float4 search_coords(const DevPtrs& P, const DomainConst& K, int p) {
  const size_t N = K.N;
  long long code = 0;
  bool finite = true;
  for (int d = 0; d < 3; ++d) {
    double xd = P.f[(C_X + d) * N + p];
    finite = finite && isfinite(xd);
    if (!COVER) {
      int q = (int)floor(__ddiv_rn(__dsub_rn(xd, K.BLPF[d]), K.CellSize[d]));
      if (q < 0) q = 0;
      if (q >= K.CellNo[d]) q = K.CellNo[d] - 1;
      code = (code << 21) | (long long)q;
    }
  }
  const float4 x = make_float4((float)(P.f[(C_X + 0) * N + p] - K.BLPF[0]), (float)(P.f[(C_X + 1) * N + p] - K.BLPF[1]),
                               (float)(P.f[(C_X + 2) * N + p] - K.BLPF[2]), (float)P.f[C_H * N + p]);
  P.cellc[p] = finite ? code : -1;
  reinterpret_cast<float4*>(P.xs)[p] = x;
  return x;
}

// Map original -> sorted index, element -> mesh particle, and the FP32
// prefilter coordinates (relative to BLPF, plus h); and for each slot of the
// cells' lists what the candidate test of a stencil scan reads, in slot order:
// those coordinates, and the particle's sorted index, original index, class
// and specimen.
__global__ void k_after_permute(DevPtrs P, DomainConst K) {
  if (!searching_full(P)) return;
  const size_t N = K.N;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < K.N; s += gridDim.x * blockDim.x) {
  const int p = P.cell_list[s];
  int o = P.i[I_ORIG * N + p];
  P.inv[o] = p;
  int kind = P.i[I_KIND * N + p];
  if (kind == 1) P.elem_particle[P.i[I_ELEM * N + p]] = p;
  P.cand_x[s] = !K.skin_on || K.cells_cover ? search_coords<true>(P, K, p) : search_coords<false>(P, K, p);
  // class word for the pair rules: bit 0 rigid-mesh particle, bit 1 carries a
  // contact-surface id, bits 2.. material index
  P.cand_m[s] = make_int4(p, o, kind | (is_contact_id(K, P.i[I_ID * N + p]) ? 2 : 0) | (P.i[I_MATERIAL * N + p] << 2),
                          P.i[I_SPEC * N + p]);
  }
}


// CheckRadius (Neighbour.cpp:361-372) exactly: rij / ((hi + hj) / 2) <= Cellfac
// with rij = sqrt(dx*dx + dy*dy + dz*dz) summed left to right, no contraction.
__device__ __forceinline__ bool radius_exact(const DevPtrs& P, size_t N, int i, int j, double Cellfac) {
  double hh = __ddiv_rn(__dadd_rn(P.f[C_H * N + i], P.f[C_H * N + j]), 2.0);
  double dx = __dsub_rn(P.f[(C_X + 0) * N + i], P.f[(C_X + 0) * N + j]);
  double dy = __dsub_rn(P.f[(C_X + 1) * N + i], P.f[(C_X + 1) * N + j]);
  double dz = __dsub_rn(P.f[(C_X + 2) * N + i], P.f[(C_X + 2) * N + j]);
  double s = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  double rij = __dsqrt_rn(s);
  return __ddiv_rn(rij, hh) <= Cellfac;
}

// FP32 prefilter of the radius test (positions in x, y, z, h in w): 1 inside,
// -1 outside, 0 within the margin that only the exact test decides.
__device__ __forceinline__ int radius_near(const DomainConst& K, float4 pi, float4 pj) {
  float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
  float d2 = dx * dx + dy * dy + dz * dz;
  float R = K.half_cellfac_f * (pi.w + pj.w);
  float R2 = R * R;
  return d2 < R2 * (1.0f - K.pre_eps) ? 1 : d2 > R2 * (1.0f + K.pre_eps) ? -1 : 0;
}

// Radius test: FP32 prefilter, exact FP64 decision inside the margin.
__device__ __forceinline__ bool radius_ok(const DevPtrs& P, const DomainConst& K, size_t N, int i, int j, float4 pi,
                                          float4 pj) {
  const int near = radius_near(K, pi, pj);
  return near > 0 || (near == 0 && radius_exact(P, N, i, j, K.Cellfac));
}

// SM neighbour rows in canonical order: one warp per particle, 32 consecutive
// particles per block.  Lanes test the candidates of each of the 27 cells in
// parallel; accepted ones are compacted with a ballot into the warp's shared
// buffer (128 slots), placed there by the rank of their canonical key, and the
// block writes its 32 rows to the ELL array one coalesced line per entry
// index.  Also sets Nb and the "free surface at search time" flag used by the
// contact pair rule.
// rank[r] += number of keys in row[0, n4) below key[r], r < NK (n4 a multiple of 4).
template <int NK>
__device__ __forceinline__ void rank_row(const unsigned* row, int n4, const unsigned key[4], int rank[4]) {
  for (int t = 0; t < n4; t += 4) {
    uint4 q = *reinterpret_cast<const uint4*>(row + t);
#pragma unroll
    for (int r = 0; r < NK; ++r)
      rank[r] += (int)(q.x < key[r]) + (int)(q.y < key[r]) + (int)(q.z < key[r]) + (int)(q.w < key[r]);
  }
}

constexpr int FILL_WARPS = 8;                    // warps per block
constexpr int FILL_ROWS = 32;                    // particles (rows) per block group
constexpr int FILL_PER_WARP = FILL_ROWS / FILL_WARPS;
constexpr int FILL_SLOTS = 128;
// SUPER: the Verlet-skin superset instead of the rows: a 5 x 5 x 5 cell
// stencil, every candidate within the pair radius plus the skin (FP32 with a
// margin: extra entries are removed by the exact filter later), up to SUP_W
// entries per particle in canonical order, and the positions they refer to.
// A row that does not fit marks the superset invalid, and this search's rows
// come from the exact form instead.
template <bool SUPER>
__global__ void __launch_bounds__(FILL_WARPS * 32) k_nbr_fill(DevPtrs P, DomainConst K) {
  if (SUPER) {
    if (!searching_full(P) || !K.skin_on) return;
  } else {
    if (!searching_full(P) || (K.skin_on && P.st->sup_valid && K.nspec == 0)) return;
  }
  // With the superset valid the filter forms the rows of the specimens that
  // search; this pass then only puts back the rows of those that do not.
  const bool keep_only = !SUPER && K.skin_on && P.st->sup_valid;
  constexpr int W = SUPER ? 5 : 3, NC = W * W * W;  // stencil
  __shared__ __align__(16) unsigned s_key[FILL_WARPS][FILL_SLOTS];
  __shared__ int s_idx[FILL_ROWS][FILL_SLOTS];
  __shared__ int2 s_rng[FILL_WARPS][NC];  // first candidate and count of a row's non-empty cells
  __shared__ int s_len[FILL_ROWS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  size_t N = K.N;
  const int* ID = P.i + I_ID * N;
  const int* orig = P.i + I_ORIG * N;
  const int* kind = P.i + I_KIND * N;
  const int* material = P.i + I_MATERIAL * N;
  const int ngroups = (K.N + FILL_ROWS - 1) / FILL_ROWS;
  unsigned long long pairs = 0;  // this warp's entries (lane 0), one atomic at the end
  for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
  const int i0 = grp * FILL_ROWS;
  // Each warp builds FILL_PER_WARP consecutive rows, one after the other, so
  // the block barrier below averages the warps' row costs over several rows.
  // Their cells, read for all of them at once: each is the end of a chain of
  // three loads.
  int key_l = 0, lin_l = 0;
  {
    const int il = i0 + w * FILL_PER_WARP + lane;
    if (lane < FILL_PER_WARP && il < K.N) {
      key_l = P.i[I_CELL * N + P.perm[il]];
      if (key_l < K.ncells) lin_l = P.cell_lin[key_l];
    }
  }
  for (int rr = 0; rr < FILL_PER_WARP; ++rr) {
  const int row = w * FILL_PER_WARP + rr;
  const int i = i0 + row;
  unsigned* rkey = &s_key[w][0];
  int* ridx = &s_idx[row][0];
  int cnt = 0, split = 0;
  bool overflow = false, link = false;
  // A particle in a shadow bucket (non-finite position) has an empty row.
  const int key_i = __shfl_sync(0xffffffffu, key_l, rr), lin = __shfl_sync(0xffffffffu, lin_l, rr);
  // Batched domain: a specimen that does not search keeps its rows (saved by
  // k_rows_save in canonical order; their keys here keep that order).
  const bool keep = !SUPER && K.nspec > 0 && i < K.N && !P.sp[P.i[I_SPEC * N + i]].do_search;
  if (keep_only && !keep) {
    if (lane == 0) s_len[row] = 0;
    continue;
  }
  if (keep) {
    const int old = P.perm[i];
    cnt = P.save_len[old];
    for (int e = lane; e < cnt; e += 32) {
      int v = P.save_nbr[(size_t)e * N + old];
      rkey[e] = (unsigned)e;
      ridx[e] = P.inv[v & 0x7fffffff] | (int)((unsigned)v & NB_UP);
    }
    __syncwarp();
  } else if (i < K.N && kind[i] == 0 && key_i < K.ncells) {
    float4 pi = reinterpret_cast<const float4*>(P.xs)[i];
    // The particle's cell: the key it was sorted by (k_cell_keys evaluated the
    // reference's FP64 cell formula once per particle), mapped back to grid
    // coordinates.
    int c[3] = {lin / (K.CellNo[1] * K.CellNo[2]), (lin / K.CellNo[2]) % K.CellNo[1], lin % K.CellNo[2]};
    int idi = ID[i], oi = orig[i], mi = material[i];
    bool ci = K.contact && is_contact_id(K, idi);
    const int spec_i = !SUPER && K.nspec > 0 ? P.i[I_SPEC * N + i] : 0;
    // Cells of the stencil, 32 per round.  A cell whose box lies farther from
    // x_i than the largest pair radius holds no neighbour and is left out
    // (about a quarter of the candidates of the 27-cell stencil, most of the
    // outer cells of the 125-cell one).  Boxes of the outermost cells extend
    // to infinity outwards, since the cell index is clamped there.  The
    // distance is a sum over the axes: lane W * d + q holds the square of the
    // distance along axis d to the stencil's layer q (NaN off the grid).
    // FP32 on the prefilter coordinates x - BLPF; the radius carries a margin
    // above the FP32 rounding of those coordinates and of the cell bounds.
    const float skip_r2 = SUPER ? K.sup_skip_r2 : K.cell_skip_r2;
    float g2_l = 0.f;
    {
      const int d = lane / W, q = lane - d * W;
      const int cd = d == 0 ? c[0] : d == 1 ? c[1] : c[2];
      const int nd = d == 0 ? K.CellNo[0] : d == 1 ? K.CellNo[1] : K.CellNo[2];
      const float sz = d == 0 ? K.CellSizef[0] : d == 1 ? K.CellSizef[1] : K.CellSizef[2];
      const float xd = d == 0 ? pi.x : d == 1 ? pi.y : pi.z;
      const int qd = cd + q - W / 2;
      const float lo = (float)qd * sz, hi = lo + sz;
      float g = 0.f;
      if (qd > 0 && xd < lo) g = lo - xd;
      if (qd < nd - 1 && xd > hi) g = xd - hi;
      // a particle outside the grid (clamped cell) keeps all cells
      const bool in = lane >= 3 * W || (xd >= 0.f && xd <= (float)nd * sz);
      g2_l = __all_sync(0xffffffffu, in) ? g * g : 0.f;
      if (qd < 0 || qd >= nd) g2_l = __int_as_float(0x7fffffff);  // NaN: no radius takes the cell
    }
    int2* rng = &s_rng[w][0];
    int ncell = 0;
#pragma unroll
    for (int q0 = 0; q0 < NC; q0 += 32) {
      const int qc = q0 + lane;
      const int qx = qc / (W * W), qy = (qc / W) % W, qz = qc % W;
      // lanes past the stencil read lane 31's value or less and are masked out
      const float gx = __shfl_sync(0xffffffffu, g2_l, qx), gy = __shfl_sync(0xffffffffu, g2_l, W + qy),
                  gz = __shfl_sync(0xffffffffu, g2_l, 2 * W + qz);
      int cs = 0, cc = 0;
      if (qc < NC && gx + gy + gz <= skip_r2) {
        int key = P.cell_rank[((c[0] + qx - W / 2) * K.CellNo[1] + c[1] + qy - W / 2) * K.CellNo[2] + c[2] + qz - W / 2];
        cs = P.cell_start[key];
        cc = P.cell_start[key + 1] - cs;
      }
      const unsigned full = __ballot_sync(0xffffffffu, cc > 0);
      if (cc > 0) rng[ncell + __popc(full & lt)] = make_int2(cs, cc);
      ncell += __popc(full);
    }
    __syncwarp();
    // Candidates, flattened over 32 non-empty cells at a time so that all
    // lanes work on every iteration: a scan of the counts gives the cells'
    // first flat indices, and the cells that begin within an iteration's 32
    // candidates set one bit each, so a candidate's cell is the number of
    // bits up to its own.  Issue binds this kernel: a binary search over the
    // cells per candidate, in four rounds over all 125 cells, made the superset
    // build take 841 us at 240,300 particles, this 610 us.
    for (int r0 = 0; r0 < ncell; r0 += 32) {
    const int2 rg = r0 + lane < ncell ? rng[r0 + lane] : make_int2(0, 0);
    int incl = rg.y;
    for (int off = 1; off < 32; off <<= 1) {
      int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int excl = incl - rg.y;
    int begun = -1;  // the last cell that began before this iteration
    for (int base = 0; base < total; base += 32) {
      const int t = base + lane;
      const int at = excl - base;
      const unsigned starts = __reduce_or_sync(0xffffffffu, rg.y > 0 && at >= 0 && at < 32 ? 1u << at : 0u);
      const int cell = begun + __popc(starts & (lt | (1u << lane)));
      begun += __popc(starts);
      const int slot = __shfl_sync(0xffffffffu, rg.x - excl, cell) + t;
      bool ok = false;
      int j = -1, oj = 0;
      if (t < total) {
        const int4 mj = P.cand_m[slot];
        const float4 pj = P.cand_x[slot];
        j = mj.x;
        oj = mj.y;
        ok = j != i && !(K.contact && (ci || (mj.z & 2))) && (mj.z & 1) == 0 && (mj.z >> 2) == mi;
        if (ok) {
          if (SUPER) {
            float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            float Rs = K.half_cellfac_f * (pi.w + pj.w) + (float)K.skin;
            ok = dx * dx + dy * dy + dz * dz <= Rs * Rs * (1.0f + 4.0f * K.pre_eps);
          } else {
            ok = radius_ok(P, K, N, i, j, pi, pj);
            if (ok && K.nspec > 0 && mj.w != spec_i) link = true;
          }
        }
      }
      unsigned m = __ballot_sync(0xffffffffu, ok);
      if (ok) {
        int pos = cnt + __popc(m & lt);
        // stored entry: the index, with bit 31 set when j has the larger
        // original index (P2 of the reference's (min, max) pair)
        if (pos < FILL_SLOTS) { rkey[pos] = (unsigned)(oj - oi - 1); ridx[pos] = (int)((unsigned)j | (oj > oi ? NB_UP : 0u)); }
      }
      cnt += __popc(m);
    }
    }  // cells
    if (cnt > (SUPER ? SUP_W : MAX_NB)) overflow = true;
    if (cnt > FILL_SLOTS) cnt = FILL_SLOTS;
    if (__any_sync(0xffffffffu, link) && lane == 0) atomicOr(&P.st->errors, ERR_SPEC_LINK);
  }
  // Order the row's slots by key.  Keys are distinct (one per neighbour), so
  // each entry's final slot is the number of smaller keys: every lane ranks
  // its own (at most four) entries against the whole row, read four keys per
  // broadcast load, then scatters them.  Pads above the row hold the largest
  // key, which no real key reaches (orig[j] - oi - 1 != -1).
  int cnt4 = (cnt + 3) & ~3;
  for (int e = cnt + lane; e < cnt4; e += 32) rkey[e] = 0xffffffffu;
  __syncwarp();
  const int nk = (cnt + 31) >> 5;  // warp-uniform
  unsigned key[4];
  int idx[4], rank[4] = {0, 0, 0, 0};
  for (int r = 0; r < 4; ++r) {
    int e = lane + 32 * r;
    key[r] = e < cnt ? rkey[e] : 0xffffffffu;
    idx[r] = e < cnt ? ridx[e] : 0;
  }
  if (nk <= 2) rank_row<2>(rkey, cnt4, key, rank);
  else if (nk == 3) rank_row<3>(rkey, cnt4, key, rank);
  else rank_row<4>(rkey, cnt4, key, rank);
  __syncwarp();
  for (int r = 0; r < 4; ++r)
    if (lane + 32 * r < cnt) ridx[rank[r]] = idx[r];
  __syncwarp();
  if (SUPER) {
    if (i < K.N && lane == 0) {
      s_len[row] = cnt;
      P.sup_len[i] = cnt;
      if (overflow) P.st->sup_valid = 0;
    } else if (lane == 0) {
      s_len[row] = 0;
    }
    continue;
  }
  if (cnt > MAX_NB) cnt = MAX_NB;
  if (i < K.N) {
    for (int e = lane; e < cnt; e += 32) split += ridx[e] < 0 ? 1 : 0;
    for (int off = 16; off > 0; off >>= 1) split += __shfl_down_sync(0xffffffffu, split, off);
    if (lane == 0) {
      s_len[row] = cnt;
      P.row_len[i] = cnt;
      P.row_split[i] = split;
      P.i[I_NB * N + i] = cnt;
      if (K.contact) P.i[I_NWS * N + i] = (P.i[I_NWS * N + i] & 1) | ((ID[i] == K.id_free_surf) ? 2 : 0);
      if (overflow) atomicOr(&P.st->errors, ERR_NBR_OVERFLOW);
      if (!keep_only) pairs += (unsigned long long)cnt;  // the filter counts the kept rows
    }
  } else if (lane == 0) {
    s_len[row] = 0;
  }
  }  // rows of this warp
  __syncthreads();
  // Block-wide coalesced ELL write: thread (k, t) stores entry k of particle i0 + t.
  int maxlen = 0;
  for (int t = 0; t < FILL_ROWS; ++t) maxlen = max(maxlen, s_len[t]);
  int* ell = SUPER ? P.sup : P.nbr;
  if (SUPER && w < 3 && i0 + lane < K.N) P.xref[w * N + i0 + lane] = P.f[(C_X + w) * N + i0 + lane];
  for (int q = threadIdx.x; q < maxlen * FILL_ROWS; q += blockDim.x) {
    int k = q / FILL_ROWS, t = q - k * FILL_ROWS;
    if (k < s_len[t]) ell[(size_t)k * N + i0 + t] = s_idx[t][k];
  }
  __syncthreads();  // the shared buffers are reused by the next group
  }
  if (!SUPER && lane == 0 && pairs) atomicAdd(&P.st->pair_count, pairs);
}

// ---- Verlet-skin reuse -------------------------------------------------------
// Largest squared displacement since the superset was built (a non-finite
// position gives NaN, whose bit pattern exceeds every finite one: a full
// search follows), and what the filter reads at the current positions
// (search_coords; in a batched domain only for the specimens that search: no
// pair leaves a specimen).  The block that finishes last decides between a
// full search and the filter: a filter suffices while every particle has moved
// less than skin / 2 since the superset was built, since a pair within its
// radius now was then within the radius plus the skin.
template <bool COVER>
__global__ void k_skin_check(DevPtrs P, DomainConst K) {
  if (!searching(P)) return;
  __shared__ bool last;
  StepState* s = P.st;
  const size_t N = K.N;
  if (s->sup_valid) {
    double m = 0.0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < K.N; p += gridDim.x * blockDim.x) {
      double d0 = P.f[(C_X + 0) * N + p] - P.xref[p];
      double d1 = P.f[(C_X + 1) * N + p] - P.xref[N + p];
      double d2 = P.f[(C_X + 2) * N + p] - P.xref[2 * N + p];
      double d = d0 * d0 + d1 * d1 + d2 * d2;
      if (!(d <= m)) m = d;
      if (K.nspec == 0 || P.sp[P.i[I_SPEC * N + p]].do_search) search_coords<COVER>(P, K, p);
    }
    unsigned long long b = (unsigned long long)__double_as_longlong(m);
    for (int off = 16; off > 0; off >>= 1) {
      unsigned long long o = __shfl_down_sync(0xffffffffu, b, off);
      b = o > b ? o : b;
    }
    if ((threadIdx.x & 31) == 0 && b) atomicMax(&s->maxdisp2_bits, b);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&s->skin_blocks, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  s->skin_blocks = 0;
  __threadfence();
  const double md2 = __longlong_as_double((long long)*(volatile unsigned long long*)&s->maxdisp2_bits);
  const double half = 0.5 * K.skin;
  const bool filter_only = s->sup_valid && md2 <= half * half;
  s->search_full = filter_only ? 0 : 1;
  if (!filter_only) {
    s->nb_full_searches += 1;
    s->sup_valid = 1;  // the superset build clears it again if a row does not fit
  }
}

__device__ __forceinline__ bool cells_adjacent(long long a, long long b) {
  for (int d = 0; d < 3; ++d) {
    int qa = (int)((a >> (21 * d)) & 0x1fffff), qb = (int)((b >> (21 * d)) & 0x1fffff);
    if (qa - qb > 1 || qb - qa > 1) return false;
  }
  return true;
}

// Rows from the superset: the entries whose particles sit in adjacent cells
// now and pass the radius rule (FP32 prefilter, exact FP64 CheckRadius),
// in the superset's canonical order — the rows a full search gives.
// COVER: every cell is wider than the largest pair radius (DomainConst::
// cells_cover), so a pair that passes the radius rule is in adjacent cells
// and the cell test is left out (a non-finite position fails the radius rule).
// L lanes per particle: each turn they test the next 4 L superset entries,
// entry and position loads issued before the first test and the next turn's
// entries before that, and append the kept ones to the row in order.  The
// superset is an ELL array like the rows, so a warp's lanes read the same
// entries of consecutive particles, whose positions share cache lines in the
// brick order, and their appends fall in the same lines of the rows.  Issue
// and load latency bind it.  A warp per particle over a row-major superset,
// compacted by ballot into shared memory, spent ~450 warp instructions per
// row, most of them on the row rather than its entries: 580 us at 982,072
// particles, this 232 us (three and five blocks per SM: 253 and 269 us).
// In a batched domain the rows of specimens that do not search stay as they
// are (untouched, or put back by k_nbr_fill after a reordering).
constexpr int FILTER_T = 256;
template <bool COVER, int L>
__global__ void __launch_bounds__(FILTER_T, 4) k_nbr_filter(DevPtrs P, DomainConst K) {
  if (!searching(P) || !K.skin_on || !P.st->sup_valid) return;
  __shared__ unsigned s_pairs;
  if (threadIdx.x == 0) s_pairs = 0;
  __syncthreads();
  const size_t N = K.N;
  const int lane = threadIdx.x & 31, sub = lane & (L - 1);
  const unsigned grp = ((1u << L) - 1u) << (lane - sub);  // the row's lanes
  const unsigned below = grp & ((1u << lane) - 1u);
  const float4* xs = reinterpret_cast<const float4*>(P.xs);
  unsigned pairs = 0;
  const int rows = FILTER_T / L;
  const int nblocks = (K.N + rows - 1) / rows;
  for (int b = blockIdx.x; b < nblocks; b += gridDim.x) {
    const int i = b * rows + threadIdx.x / L;
    bool mine = i < K.N;
    if (mine && K.nspec > 0 && !P.sp[P.i[I_SPEC * N + i]].do_search) {
      mine = false;
      if (sub == 0) pairs += (unsigned)P.row_len[i];
    }
    const int spec_i = K.nspec > 0 && mine ? P.i[I_SPEC * N + i] : 0;
    const long long ci = mine ? P.cellc[i] : -1;
    int len = 0;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (mine && P.i[I_KIND * N + i] == 0 && ci >= 0) {
      pi = xs[i];
      len = P.sup_len[i];
    }
    // lanes of a warp take the same number of turns (ballots below)
    const int most = L == 1 ? len : __reduce_max_sync(0xffffffffu, len);
    constexpr int U = 4;
    const int* sup = P.sup + i;
    int e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) e[u] = u * L + sub < len ? sup[(size_t)(u * L + sub) * N] : 0;
    int cnt = 0, split = 0;
    bool link = false;
    for (int k0 = 0; k0 < most; k0 += U * L) {
      float4 pj[U];
      long long cj[U];
      int en[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (k0 + u * L + sub < len) {
          pj[u] = xs[nb_index(e[u])];
          if (!COVER) cj[u] = P.cellc[nb_index(e[u])];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = k0 + (U + u) * L + sub;
        en[u] = k < len ? sup[(size_t)k * N] : 0;
      }
      // the FP32 prefilter's decisions, and the pairs inside its margin
      unsigned in = 0, edge = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (k0 + u * L + sub < len && (COVER || (cj[u] >= 0 && cells_adjacent(ci, cj[u])))) {
          const int near = radius_near(K, pi, pj[u]);
          in |= (near > 0 ? 1u : 0u) << u;
          edge |= (near == 0 ? 1u : 0u) << u;
        }
      }
#pragma unroll 1
      for (int u = 0; edge; ++u, edge >>= 1)
        if ((edge & 1u) && radius_exact(P, N, i, nb_index(u == 0 ? e[0] : u == 1 ? e[1] : u == 2 ? e[2] : e[3]), K.Cellfac))
          in |= 1u << u;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const bool ok = in >> u & 1u;
        if (ok && K.nspec > 0 && P.i[I_SPEC * N + nb_index(e[u])] != spec_i) link = true;
        int pos = cnt;
        if (L == 1) {
          cnt += ok ? 1 : 0;
        } else {
          const unsigned m = __ballot_sync(0xffffffffu, ok);
          pos += __popc(m & below);
          cnt += __popc(m & grp);
        }
        if (ok && pos < MAX_NB) {
          P.nbr[(size_t)pos * N + i] = e[u];
          split += e[u] < 0 ? 1 : 0;
        }
        e[u] = en[u];
      }
    }
    if (link) atomicOr(&P.st->errors, ERR_SPEC_LINK);
    if (cnt > MAX_NB) {
      cnt = MAX_NB;
      if (sub == 0) atomicOr(&P.st->errors, ERR_NBR_OVERFLOW);
    }
    for (int off = 1; off < L; off <<= 1) split += __shfl_xor_sync(0xffffffffu, split, off);
    if (mine && sub == 0) {
      P.row_len[i] = cnt;
      P.row_split[i] = split;
      P.i[I_NB * N + i] = cnt;
      pairs += (unsigned)cnt;
    }
  }
  pairs = __reduce_add_sync(0xffffffffu, pairs);
  if (lane == 0 && pairs) atomicAdd(&s_pairs, pairs);
  __syncthreads();
  if (threadIdx.x == 0 && s_pairs) atomicAdd(&P.st->pair_count, (unsigned long long)s_pairs);
}

// CalculateSurface (Domain.cpp:1415-1491): n_i = sum_j m_j (x_i - x_j) in row
// order; |n| / totmass >= 0.25 h and Nb <= 46 marks the free surface (ID 1).
__global__ void k_surface(DevPtrs P, DomainConst K) {
  if (!searching(P)) return;
  size_t N = K.N;
  unsigned nsurf = 0;  // summed over the warp, one atomic per warp
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K.N; i += gridDim.x * blockDim.x) {
  if (P.i[I_KIND * N + i] != 0) continue;
  double xi = P.f[C_X * N + i], yi = P.f[(C_X + 1) * N + i], zi = P.f[(C_X + 2) * N + i];
  double n0 = 0, n1 = 0, n2 = 0;
  int len = P.row_len[i];
  for (int k = 0; k < len; ++k) {
    int j = nb_index(P.nbr[(size_t)k * N + i]);
    double mj = P.f[C_MASS * N + j];
    n0 = __dadd_rn(n0, __dmul_rn(mj, __dsub_rn(xi, P.f[C_X * N + j])));
    n1 = __dadd_rn(n1, __dmul_rn(mj, __dsub_rn(yi, P.f[(C_X + 1) * N + j])));
    n2 = __dadd_rn(n2, __dmul_rn(mj, __dsub_rn(zi, P.f[(C_X + 2) * N + j])));
  }
  double s = __ddiv_rn(1.0, K.totmass_mean);
  n0 = __dmul_rn(s, n0); n1 = __dmul_rn(s, n1); n2 = __dmul_rn(s, n2);
  P.f[C_NORMAL * N + i] = n0; P.f[(C_NORMAL + 1) * N + i] = n1; P.f[(C_NORMAL + 2) * N + i] = n2;
  int id = P.i[I_IDORIG * N + i];
  double nn = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(n0, n0), __dmul_rn(n1, n1)), __dmul_rn(n2, n2)));
  bool surf = (nn >= __dmul_rn(0.25, P.f[C_H * N + i])) && (len <= 46);
  if (surf) {
    if (!(P.i[I_NWS * N + i] & 1)) id = 1;
    ++nsurf;
  }
  P.i[I_ID * N + i] = id;
  }
  nsurf = __reduce_add_sync(0xffffffffu, nsurf);
  if ((threadIdx.x & 31) == 0 && nsurf) atomicAdd(&P.st->surface_count, (int)nsurf);
}

// ContactNbSearch (Contact.cpp:57-132): surface particle (at search time and
// now) within h1 + h2 of a rigid-mesh particle in a neighbouring cell.
// Row sorted by the mesh particle's original index.
__global__ void k_contact_pairs(DevPtrs P, DomainConst K) {
  if (!searching(P)) return;
  size_t N = K.N;
  unsigned npairs = 0;  // summed over the warp, one atomic per warp
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K.N; i += gridDim.x * blockDim.x) {
  int cnt = 0;
  bool overflow = false;
  int row[MAX_CP];
  int keys[MAX_CP];
  int idi = P.i[I_ID * N + i];
  bool ok = P.i[I_KIND * N + i] == 0 && (P.i[I_NWS * N + i] & 2) && idi == K.id_free_surf;
  if (ok) {
    double xi = P.f[C_X * N + i], yi = P.f[(C_X + 1) * N + i], zi = P.f[(C_X + 2) * N + i];
    double hi = P.f[C_H * N + i];
    int c[3];
    for (int d = 0; d < 3; ++d) {
      int q = (int)floor(__ddiv_rn(__dsub_rn(P.f[(C_X + d) * N + i], K.BLPF[d]), K.CellSize[d]));
      c[d] = q < 0 ? 0 : (q >= K.CellNo[d] ? K.CellNo[d] - 1 : q);
    }
    for (int a = c[0] - 1; a <= c[0] + 1; ++a) {
      if (a < 0 || a >= K.CellNo[0]) continue;
      for (int b = c[1] - 1; b <= c[1] + 1; ++b) {
        if (b < 0 || b >= K.CellNo[1]) continue;
        for (int e = c[2] - 1; e <= c[2] + 1; ++e) {
          if (e < 0 || e >= K.CellNo[2]) continue;
          int key = P.cell_rank[(a * K.CellNo[1] + b) * K.CellNo[2] + e];
          for (int q = P.cell_start[key]; q < P.cell_start[key + 1]; ++q) {
            const int j = P.cell_list[q];
            if (P.i[I_KIND * N + j] != 1) continue;
            if (!is_contact_id(K, P.i[I_ID * N + j])) continue;
            double dx = __dsub_rn(xi, P.f[C_X * N + j]), dy = __dsub_rn(yi, P.f[(C_X + 1) * N + j]),
                   dz = __dsub_rn(zi, P.f[(C_X + 2) * N + j]);
            double r = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
            if (!(r < __dadd_rn(hi, P.f[C_H * N + j]))) continue;
            int kk = P.i[I_ORIG * N + j];
            if (cnt < MAX_CP) {
              int m = cnt - 1;
              while (m >= 0 && keys[m] > kk) { keys[m + 1] = keys[m]; row[m + 1] = row[m]; --m; }
              keys[m + 1] = kk; row[m + 1] = j;
              ++cnt;
            } else overflow = true;
          }
        }
      }
    }
  }
  for (int k = 0; k < cnt; ++k) P.cp[(size_t)k * N + i] = row[k];
  P.cp_len[i] = cnt;
  if (cnt > 0) P.cp_list[atomicAdd(&P.st->cp_count, 1)] = i;
  if (overflow) atomicOr(&P.st->errors, ERR_CONTACT_OVERFLOW);
  npairs += (unsigned)cnt;
  }
  npairs = __reduce_add_sync(0xffffffffu, npairs);
  if ((threadIdx.x & 31) == 0 && npairs) atomicAdd(&P.st->contact_pair_count, (unsigned long long)npairs);
}

__global__ void k_force_search(DevPtrs P, DomainConst K) {
  P.st->do_search = 1;
  search_begin(P, K);
}
void launch_force_search(const DevPtrs& P, const DomainConst& K, cudaStream_t s) { k_force_search<<<1, 1, 0, s>>>(P, K); }

// ---------------------------------------------------------------- host side
static inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

void launch_neighbour_search(const DevPtrs& P, const DomainConst& K, double* fscratch, int* iscratch,
                             cudaStream_t s) {
  const int T = 256;
  // Gated kernels run on fixed grids with grid-stride loops: on steps that do
  // not search, each launch is a handful of blocks that exit at once.
  const int G = 152 * 4;
  auto grid = [&](long long n) { int b = nblk(n, T); return b < G ? b : G; };
  // buckets: ncells grid cells (Morton ranks), then ncells shadow buckets
  const long long nbk = 2LL * K.ncells;
  if (K.skin_on) {
    if (K.cells_cover) k_skin_check<true><<<grid(K.N), T, 0, s>>>(P, K);
    else k_skin_check<false><<<grid(K.N), T, 0, s>>>(P, K);
    mark(s, "k_skin_check");
  }
  if (K.nspec > 0) {
    k_rows_save<<<grid(K.N), T, 0, s>>>(P, K);
    mark(s, "k_rows_save");
  }
  k_cell_keys<<<grid(K.N), T, 0, s>>>(P, K);
  mark(s, "k_cell_keys");
  if (nbk <= 16 * SCAN_TILE) {  // two launches saved against 4 us more at 16 tiles, when a search re-sorts
    k_scan_one<<<1, SCAN_THREADS, 0, s>>>(P, P.cell_count, (int)nbk, P.cell_start, P.cell_start + nbk);
    mark(s, "k_scan_one");
  } else {
    int nb = nblk(nbk, SCAN_TILE);
    k_scan_reduce<<<nb, SCAN_THREADS, 0, s>>>(P, P.cell_count, nbk, P.scan_tmp);
    mark(s, "k_scan_reduce");
    k_scan_top<<<1, SCAN_THREADS, 0, s>>>(P, P.scan_tmp, nb);
    mark(s, "k_scan_top");
    k_scan_down<<<nb, SCAN_THREADS, 0, s>>>(P, P.cell_count, nbk, P.scan_tmp, P.cell_start, P.cell_start + nbk);
    mark(s, "k_scan_down");
  }
  k_scatter<<<grid(K.N), T, 0, s>>>(P, K);
  mark(s, "k_scatter");
  k_sort_bricks<<<K.nbricks < 152 * 2 ? K.nbricks : 152 * 2, BRICK_T, 0, s>>>(P, K);
  mark(s, "k_sort_bricks");
  k_permute<<<152 * 4, 512, 0, s>>>(P, K, fscratch, iscratch);
  mark(s, "k_permute");
  k_copy_back<<<152 * 4, 512, 0, s>>>(P, K, fscratch, iscratch);
  mark(s, "k_copy_back");
  k_after_permute<<<grid(K.N), T, 0, s>>>(P, K);
  mark(s, "k_after_permute");
  {
    // a few resident blocks per SM, striding over the row groups
    int groups = nblk(K.N, FILL_ROWS), cap = 152 * 4;
    if (K.skin_on) {
      k_nbr_fill<true><<<groups < cap ? groups : cap, FILL_WARPS * 32, 0, s>>>(P, K);
      mark(s, "k_sup_build");
    }
    k_nbr_fill<false><<<groups < cap ? groups : cap, FILL_WARPS * 32, 0, s>>>(P, K);
  }
  mark(s, "k_nbr_fill");
  if (K.skin_on) {
    // Lanes per row: a filtered search of 8,004 / 30,600 / 63,612 / 120,416 /
    // 240,300 particles takes 85 / 87 / 93 / 111 / 145 us with one, 75 / 82 /
    // 92 / 110 / 153 with four (eight: 74 / 84 / 95 / 118 / 172).
    const int L = K.N < 100000 ? 4 : 1;
    const int blocks = nblk((long long)K.N * L, FILTER_T), cap = 152 * 16;
    const auto k = K.cells_cover ? (L == 4 ? k_nbr_filter<true, 4> : k_nbr_filter<true, 1>)
                                 : (L == 4 ? k_nbr_filter<false, 4> : k_nbr_filter<false, 1>);
    k<<<blocks < cap ? blocks : cap, FILTER_T, 0, s>>>(P, K);
    mark(s, "k_nbr_filter");
  }
  if (P.halo) launch_halo_build(P, K, s);
  if (K.contact) {
    k_surface<<<grid(K.N), T, 0, s>>>(P, K);
    mark(s, "k_surface");
    k_contact_pairs<<<grid(K.N), 128, 0, s>>>(P, K);
    mark(s, "k_contact_pairs");
  }
}

}  // namespace wf
