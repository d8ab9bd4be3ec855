// gbmd_neighbors.cu -- cell grid, cell sort and full neighbour list on sm_103a.
//
// Restates exaNBody's move_particles (periodic wrap, rebinning) and
// chunk_neighbors with chunk_size 1 (data/config/config_move_particles.msp
// L54-68).  The pair set is the one the reference decodes in
// src/debug/atom_neighbors_stats.cpp L169-228: every (i, j, image n) with
// d2 <= (rcut_max + skin)^2, d2 computed in FP64 from ((x_j + n*L) - x_i)
// without contraction.  Candidates are screened in FP32 on home-cell-relative
// coordinates; only those within band_tol of the radius are re-tested in FP64,
// so the list is bit-identical to an all-FP64 build.
//
// Kernels (per rebuild):
//   k_wrap_bin    wrap into [lo,hi), bin, count per cell        HBM: 24 B r/w + 8 B
//   k_scan_*      exclusive scan of cell counts                 negligible
//   k_scatter     atoms -> cell segments (atomic slot)          HBM: 12 B
//   k_cell_rank   canonical (id, upload index) order per cell   L1-resident
//   k_gather      permute the FP64 state into cell order, with
//                 the FP32 local + FP64 packed gather copies    HBM: ~130 B r/w, 48 B w
//   k_build_list_cells  warp per home cell over the 27-cell candidates, rows
//                 in canonical order                            HBM: 4 B per entry
//   k_build_list_long   the same rows where they are long, a warp per atom
//
// Every kernel of the chain takes a `gate` word: when it is non-null and
// holds 0 the kernel returns at once.  The displacement-triggered step
// (particle_displ_over, config_move_particles.msp L19-22, L116-118) sets the
// gate on the device and launches the chain unconditionally, so the decision
// to rebuild never goes through the host and the chain can sit inside a CUDA
// graph.  That variant gathers into the spare buffers and copies back, so the
// buffer parity the captured pointers rely on does not depend on the outcome.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <utility>

#include "gbmd_internal.cuh"

namespace gbmd {

int grid_dims(const double lo[3], const double hi[3], double R, int nc[3]) {
  for (int d = 0; d < 3; ++d) {
    const double L = hi[d] - lo[d];
    if (!(L > 0.0) || !(R > 0.0)) return -1;
    double q = floor(L / (R * (1.0 + 0x1p-40)));
    if (q < 1.0) return -2;
    if (q > 1024.0) q = 1024.0;
    nc[d] = (int)q;
  }
  return 0;
}

struct BoxArgs {
  double lo[3], hi[3], L[3], inv_h[3];
  long long klo[3], khi[3];  // order_key of lo, hi
  int nc[3];
};

__global__ void k_wrap_bin(int64_t n, double* __restrict__ x, double* __restrict__ y,
                           double* __restrict__ z, BoxArgs b, int32_t* __restrict__ cell_of,
                           int32_t* __restrict__ cell_count, int* __restrict__ err, const int* __restrict__ gate) {
  if (gate && !*gate) return;
  if (!gate && blockIdx.x == 0 && threadIdx.x == 0) err[ERRW_MAXNB] = 0;  // of the list this chain builds
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
  double* r[3] = {x, y, z};
  int c[3];
  bool lost = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double v = r[d][i];
    // most atoms are inside: two integer comparisons and no store, where the
    // FP64 ones took 16 SM cycles each (4 M atoms: 175 -> 68 us)
    const long long k = order_key(v);
    if (k <= b.klo[d] || k >= b.khi[d]) {
      if (v < b.lo[d]) v = __dadd_rn(v, b.L[d]);
      else if (v >= b.hi[d]) v = __dsub_rn(v, b.L[d]);
      if (!(v >= b.lo[d] && v < b.hi[d])) lost = true;
      r[d][i] = v;
    }
    int q = (int)__dmul_rn(__dsub_rn(v, b.lo[d]), b.inv_h[d]);
    q = q < 0 ? 0 : (q > b.nc[d] - 1 ? b.nc[d] - 1 : q);
    c[d] = q;
  }
  if (lost) {
    atomicAdd(&err[ERRW_LOST], 1);
    atomicOr(&err[ERRW_FLAGS], GBMD_DEVERR_LOST_ATOM);
  }
  const int32_t lin = (int32_t)(((int64_t)c[2] * b.nc[1] + c[1]) * b.nc[0] + c[0]);
  cell_of[i] = lin;
  // atoms stay cell-sorted between rebuilds, so a warp's 32 atoms fall into
  // a few cells: one atomic per cell and warp
  const unsigned peers = __match_any_sync(__activemask(), lin);
  if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&cell_count[lin], __popc(peers));
  }
}

// --- exclusive scan (256 threads x 8 items per block) ----------------------
constexpr int SCAN_T = 256, SCAN_I = 8, SCAN_B = SCAN_T * SCAN_I;

__device__ __forceinline__ int block_exclusive(int v, int* smem, int& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) smem[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    int w = lane < (int)(blockDim.x >> 5) ? smem[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < (int)(blockDim.x >> 5)) smem[lane] = wi - w;
    if (lane == 31) smem[32] = wi;
  }
  __syncthreads();
  total = smem[32];
  const int r = smem[wid] + inc - v;
  __syncthreads();
  return r;
}

// in[0..n) -> out[0..n] exclusive (out[n] = total when this block holds n)
__global__ void k_scan_block(const int32_t* __restrict__ in, int32_t* __restrict__ out, int64_t n,
                             int32_t* __restrict__ sums, const int* __restrict__ gate) {
  if (gate && !*gate) return;  // uniform per block
  __shared__ int smem[33];
  const int64_t base = (int64_t)blockIdx.x * SCAN_B + (int64_t)threadIdx.x * SCAN_I;
  int it[SCAN_I];
  int s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_I; ++k) {
    const int64_t q = base + k;
    it[k] = q < n ? in[q] : 0;
    s += it[k];
  }
  int total;
  int off = block_exclusive(s, smem, total);
#pragma unroll
  for (int k = 0; k < SCAN_I; ++k) {
    const int64_t q = base + k;
    if (q <= n) out[q] = off;
    off += it[k];
  }
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void k_scan_sums(int32_t* sums, int nb, const int* __restrict__ gate) {
  if (gate && !*gate) return;
  __shared__ int smem[33];
  int carry = 0;
  for (int base = 0; base < nb; base += SCAN_B) {
    int it[SCAN_I];
    int s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
      const int q = base + threadIdx.x * SCAN_I + k;
      it[k] = q < nb ? sums[q] : 0;
      s += it[k];
    }
    int total;
    int off = block_exclusive(s, smem, total);
#pragma unroll
    for (int k = 0; k < SCAN_I; ++k) {
      const int q = base + threadIdx.x * SCAN_I + k;
      if (q < nb) sums[q] = off + carry;
      off += it[k];
    }
    carry += total;
  }
}

__global__ void k_scan_add(int32_t* __restrict__ out, int64_t n, const int32_t* __restrict__ sums,
                           const int* __restrict__ gate) {
  if (gate && !*gate) return;
  const int64_t base = (int64_t)blockIdx.x * SCAN_B;
  const int add = sums[blockIdx.x];
  for (int k = threadIdx.x; k < SCAN_B; k += blockDim.x) {
    const int64_t q = base + k;
    if (q <= n) out[q] += add;
  }
}

// The same in one block of 1,024 threads: for a few thousand cells the three
// launches above are all latency (1,331 cells: 12 us).
constexpr int SCAN_SMALL = 1024 * 16;

__global__ void __launch_bounds__(1024) k_scan_small(const int32_t* __restrict__ in, int32_t* __restrict__ out, int n,
                                                     const int* __restrict__ gate) {
  if (gate && !*gate) return;
  __shared__ int smem[33];
  const int base = (int)threadIdx.x * 16;
  int it[16], s = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    it[k] = base + k < n ? in[base + k] : 0;
    s += it[k];
  }
  int total;
  int off = block_exclusive(s, smem, total);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    if (base + k <= n) out[base + k] = off;
    off += it[k];
  }
}

static int64_t scan_blocks(int64_t n) { return (n + 1 + SCAN_B - 1) / SCAN_B; }

// scan_tmp holds scan_blocks(n) words (ensure_cells): nothing here can fail.
static void scan(gbmd_context* c, const int32_t* in, int32_t* out, int64_t n, const int* gate) {
  if (n + 1 <= SCAN_SMALL) {
    k_scan_small<<<1, 1024, 0, c->stream>>>(in, out, (int)n, gate);
    return;
  }
  const int64_t nb = scan_blocks(n);
  k_scan_block<<<(unsigned)nb, SCAN_T, 0, c->stream>>>(in, out, n, c->scan_tmp, gate);
  k_scan_sums<<<1, SCAN_T, 0, c->stream>>>(c->scan_tmp, (int)nb, gate);
  k_scan_add<<<(unsigned)nb, SCAN_T, 0, c->stream>>>(out, n, c->scan_tmp, gate);
}

// The per-cell arrays for `ncells` cells, with the counts cleared.  An
// allocation that fails leaves none, so that the next call starts afresh.
static int ensure_cells(gbmd_context* c, int64_t ncells) {
  if (c->cells_cap >= ncells + 1) return GBMD_OK;
  cudaFree(c->cell_start);
  cudaFree(c->cell_fill);
  cudaFree(c->scan_tmp);
  c->cell_start = c->cell_fill = c->scan_tmp = nullptr;
  c->cells_cap = 0;
  GBMD_CUDA(c, dev_malloc(c, (void**)&c->cell_start, sizeof(int32_t) * (ncells + 1)));
  GBMD_CUDA(c, dev_malloc(c, (void**)&c->cell_fill, sizeof(int32_t) * (ncells + 1)));
  GBMD_CUDA(c, dev_malloc(c, (void**)&c->scan_tmp, sizeof(int32_t) * scan_blocks(ncells)));
  GBMD_CUDA(c, cudaMemsetAsync(c->cell_fill, 0, sizeof(int32_t) * (ncells + 1), c->stream));
  c->cells_cap = ncells + 1;
  return GBMD_OK;
}

__global__ void k_scatter(int64_t n, const int32_t* __restrict__ cell_of, const int32_t* __restrict__ cstart,
                          int32_t* __restrict__ fill, int32_t* __restrict__ order, const int* __restrict__ gate) {
  if (gate && !*gate) return;
  const int lane = threadIdx.x & 31;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t cl = cell_of[i];
    // one atomic per cell and warp; the order inside a cell is fixed later
    // by k_cell_rank, so any slot assignment will do
    const unsigned peers = __match_any_sync(__activemask(), cl);
    const int leader = __ffs(peers) - 1;
    // counting the cell's atoms down: all counts are zero again at the end,
    // ready for the next chain
    int base = 0;
    if (lane == leader) base = atomicSub(&fill[cl], __popc(peers)) - __popc(peers);
    base = __shfl_sync(peers, base, leader);
    order[cstart[cl] + base + __popc(peers & ((1u << lane) - 1u))] = (int32_t)i;
  }
}

// one warp per cell: rank by (id, upload index) -> src[new] = old
__global__ void k_cell_rank(int64_t ncells, const int32_t* __restrict__ cstart, const int32_t* __restrict__ order,
                            const uint64_t* __restrict__ id, const int32_t* __restrict__ user,
                            int32_t* __restrict__ src, const int* __restrict__ gate) {
  const int lane = threadIdx.x & 31;
  if (gate && !*gate) return;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t cell = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; cell < ncells; cell += warps) {
  const int beg = cstart[cell], m = cstart[cell + 1] - beg;
  if (m <= 32) {
    // keys in registers, compared through shuffles
    int32_t a = 0, ua = 0;
    uint64_t ka = 0;
    if (lane < m) {
      a = order[beg + lane];
      ka = id[a];
      ua = user[a];
    }
    int rank = 0;
    for (int f = 0; f < m; ++f) {
      const uint64_t kb = __shfl_sync(0xffffffffu, ka, f);
      const int32_t ub = __shfl_sync(0xffffffffu, ua, f);
      rank += (kb < ka) || (kb == ka && ub < ua);
    }
    if (lane < m) src[beg + rank] = a;
    continue;
  }
  for (int e = lane; e < m; e += 32) {
    const int32_t a = order[beg + e];
    const uint64_t ka = id[a];
    const int32_t ua = user[a];
    int rank = 0;
    for (int f = 0; f < m; ++f) {
      const int32_t b = order[beg + f];
      const uint64_t kb = id[b];
      rank += (kb < ka) || (kb == ka && user[b] < ua);
    }
    src[beg + rank] = a;
  }
  }
}

struct GatherArgs {
  const double *r0, *v0, *a0;
  double *r1, *v1, *a1;
  const uint8_t* t0;
  uint8_t* t1;
  const uint64_t* i0;
  uint64_t* i1;
  const int32_t* u0;
  int32_t* u1;
  const double* ep0;
  double* ep1;
  int64_t cap;
};

// Permutes the state into cell order and, with the positions at hand, writes
// their gather copies (a pass of their own read 29 bytes an atom again: 4 M
// atoms 186 + 98 -> 189 us).
__global__ void k_gather(int64_t n, const int32_t* __restrict__ src, GatherArgs g,
                         const int32_t* __restrict__ cell_of, Grid grid, int32_t* __restrict__ cellpack,
                         float4* __restrict__ pf, double4_32a* __restrict__ pd, const int* __restrict__ gate) {
  if (gate && !*gate) return;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
  const int64_t o = src[p];
  double r[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    r[d] = g.r0[d * g.cap + o];
    g.r1[d * g.cap + p] = r[d];
    g.v1[d * g.cap + p] = g.v0[d * g.cap + o];
    g.a1[d * g.cap + p] = g.a0[d * g.cap + o];
  }
  const int t = g.t0[o];
  g.t1[p] = (uint8_t)t;
  g.i1[p] = g.i0[o];
  g.u1[p] = g.u0[o];
  g.ep1[p] = g.ep0[o];
  const int32_t lin = cell_of[o];
  const int cx = lin % grid.nc[0], cy = (lin / grid.nc[0]) % grid.nc[1], cz = lin / (grid.nc[0] * grid.nc[1]);
  const int cp = cx | (cy << 10) | (cz << 20);
  cellpack[p] = cp;
  store_gather(grid, p, cp, t, r[0], r[1], r[2], pf, pd);
  }
}

// gated variant only: the sorted state, gathered into the spare buffers, is
// copied back so the current buffer index does not change
__global__ void k_copy_back(int64_t n, GatherArgs g, const int* __restrict__ gate) {
  if (!*gate) return;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
  double* r0 = const_cast<double*>(g.r0);
  double* v0 = const_cast<double*>(g.v0);
  double* a0 = const_cast<double*>(g.a0);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    r0[d * g.cap + p] = g.r1[d * g.cap + p];
    v0[d * g.cap + p] = g.v1[d * g.cap + p];
    a0[d * g.cap + p] = g.a1[d * g.cap + p];
  }
  const_cast<uint8_t*>(g.t0)[p] = g.t1[p];
  const_cast<uint64_t*>(g.i0)[p] = g.i1[p];
  const_cast<int32_t*>(g.u0)[p] = g.u1[p];
  const_cast<double*>(g.ep0)[p] = g.ep1[p];
  }
}

__global__ void k_posf(int64_t n, const double* __restrict__ x, const double* __restrict__ y,
                       const double* __restrict__ z, const uint8_t* __restrict__ type,
                       const int32_t* __restrict__ cellpack, Grid g, float4* __restrict__ pf,
                       double4_32a* __restrict__ pd, const int* __restrict__ gate) {
  if (gate && !*gate) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
  store_gather(g, i, cellpack[i], type[i], x[i], y[i], z[i], pf, pd);
  }
}

// FP64 re-test of a candidate whose FP32 d2 fell within the band around R^2.  Out of
// line so the compiler cannot predicate it into every iteration of the
// candidate loop (it runs for ~1e-4 of the candidates).
__device__ __noinline__ bool exact_within(const double* __restrict__ x, const double* __restrict__ y,
                                          const double* __restrict__ z, int64_t i, int64_t k, uint32_t code,
                                          int cx, int cy, int cz, const Grid g, double R2) {
  const int nxi = image_of(cx, code_dx(code), g.nc[0]);
  const int nyi = image_of(cy, code_dy(code), g.nc[1]);
  const int nzi = image_of(cz, code_dz(code), g.nc[2]);
  double a, b, c;
  return exact_d2(x[i], y[i], z[i], x[k], y[k], z[k], (double)nxi * g.L[0], (double)nyi * g.L[1],
                  (double)nzi * g.L[2], a, b, c) <= R2;
}

// ---------------------------------------------------------------------------
// The list builder: one warp per home cell (or several, each taking its share
// of the cell's groups), the cell's atoms 16 at a time.
//
// Lanes l and l + 16 hold home atom l of the group.  The candidates, the atoms
// of the 27 stencil cells in stencil order, are staged in shared memory 32 at
// a time for each half-warp, shifted into the home cell's frame; those farther
// than R from the bounding box of the group's atoms, about a quarter, are left
// out.  The low half-warp tests the first half of the candidates in order and
// appends to the front of the atom's row in shared memory; the high half-warp
// tests the second half from the end backwards and fills the row from its end
// towards the front.  So both know where a hit goes without asking the other,
// and the row ends in the canonical order (stencil code, then cell order).
//
// The walk is bound by instruction issue: a test costs about nine
// instructions (two candidates at a time in packed FP32, one broadcast read
// of 16 bytes, one predicated shared-memory store), where appending straight to the rows in
// global memory, with their 64-bit slot address and an exchange between the
// half-warps on every step, took over thirty.  A row leaves shared memory
// once, complete, as 16-byte stores of neighbouring atoms.
// Whole rebuild: 4 M-atom Cu, R = 5.3, 2,380 -> 1,845 us; 16.6 M-atom LJ mixture, 111
// entries an atom, 17.6 -> 13.1 ms; 1 M-atom LJ 888 -> 765 us.
//
// The walk keeps every candidate with FP32 d2 <= R2hi; atoms with a hit above
// R2lo (the band of band_tol, below one per cent) have their band entries
// re-tested in FP64 afterwards by the whole warp.
// ---------------------------------------------------------------------------
constexpr int BUILD_G = 16;       // home atoms per group
constexpr int BUILD_CHUNK = 32;   // candidates staged per half-warp: one round of the warp
constexpr int BUILD_WARPS = 4;    // warps per block, where shared memory allows
constexpr int BUILD_LONG = 900;   // row capacity from which k_build_list_long builds the list
constexpr int BUILD_SLACK = 16;   // row slots beyond maxnb: 8 tests at either end run unchecked

// One warp's shared memory, followed by its BUILD_G rows of (maxnb + BUILD_SLACK) entries.
struct BuildSmem {
  // x, y, z, w of the low half-warp's candidates, then of the high one's, 64
  // bytes further so that both broadcasts of a step read different banks
  float4 chunk[2 * BUILD_CHUNK + 4];
  float4 shift[28];    // nonempty stencil cells in order: first atom - first candidate, shift into the home frame
  uint32_t code[28];   // their stencil code << 26
  int pre[28];         // their first candidate; pre[ncell] = all candidates
};

__host__ __device__ inline int build_rowlen(int maxnb) { return (maxnb + BUILD_SLACK) | 1; }  // odd: rows start in different banks
__host__ __device__ inline size_t build_smem(int maxnb, int homes) {
  return sizeof(BuildSmem) + (size_t)((homes * build_rowlen(maxnb) + 3) & ~3) * sizeof(uint32_t);
}

struct BuildArgs {
  int64_t ncells;
  const float4* pf;
  const double *x, *y, *z;
  const int32_t* cstart;
  double R2;
  float R2lo, R2hi;
  uint32_t* nbr;
  int32_t* nnb;
  int maxnb, W, wsh, tsh, homes, parts;  // homes: atoms per group; parts: warps per cell
  int64_t stride;
  int* err;
  int64_t n;
  const int32_t* cellpack;
};

// One round of staging: the candidates qa .. qa + 31, in reverse with `rev`,
// as far as they lie in [q0, q1).  Lane s describes stencil cell s: s_pre its
// first candidate, s_any whether it has any.  fetch() reads a lane's candidate,
// store() writes those near the box [blo, bhi], in order, to the front of
// `dst`, fills the rest of the 32 slots with candidates out of reach, and
// returns how many are in.
struct BuildRound {
  float4 pj, sh;
  uint32_t w;
  bool valid;
  __device__ __forceinline__ void fetch(const BuildSmem& S, const float4* __restrict__ pf, int s_pre, bool s_any,
                                        int qa, int q0, int q1, bool rev, int lane) {
    const unsigned FULL = 0xffffffffu;
    const int off = s_pre - qa, pos = rev ? 31 - lane : lane, q = qa + pos;
    // cell of candidate qa + pos: the nonempty cells that start up to there
    const unsigned starts = __reduce_or_sync(FULL, s_any && (unsigned)off < 32u ? 1u << off : 0u);
    const int before = __popc(__ballot_sync(FULL, s_any && off < 0));
    valid = q >= q0 && q < q1;
    const int sc = valid ? before + __popc(starts & (0xffffffffu >> (31 - pos))) - 1 : 0;
    sh = S.shift[sc];
    const int k = valid ? q + __float_as_int(sh.x) : 0;
    w = (uint32_t)k | S.code[sc];
    pj = pf[k];
  }
  __device__ __forceinline__ int store(float4* dst, int lane, const float3& blo, const float3& bhi, float R2keep) {
    const float ex = __fadd_rn(pj.x, sh.y), ey = __fadd_rn(pj.y, sh.z), ez = __fadd_rn(pj.z, sh.w);
    const float bx = fmaxf(0.f, fmaxf(blo.x - ex, ex - bhi.x));
    const float by = fmaxf(0.f, fmaxf(blo.y - ey, ey - bhi.y));
    const float bz = fmaxf(0.f, fmaxf(blo.z - ez, ez - bhi.z));
    const bool keep = valid && fmaf(bx, bx, fmaf(by, by, bz * bz)) <= R2keep;
    const unsigned km = __ballot_sync(0xffffffffu, keep), lt = (1u << lane) - 1u;
    const int kept = __popc(km), slot = keep ? __popc(km & lt) : kept + __popc(~km & lt);
    float* d = reinterpret_cast<float*>(dst) + slot;
    d[0] = keep ? ex : 1e18f;
    d[BUILD_CHUNK] = ey;
    d[2 * BUILD_CHUNK] = ez;
    d[3 * BUILD_CHUNK] = __uint_as_float(w);
    return kept;
  }
};

// FP32 d2 of home atom pi and entry w, as the walk computes it.
__device__ __forceinline__ float build_d2(const float4* __restrict__ pf, const Grid& g, const float4& pi, uint32_t w) {
  const uint32_t code = w >> GBMD_IDX_BITS;
  const float4 pj = pf[w & GBMD_IDX_MASK];
  const float sx = __fmul_rn((float)code_dx(code), g.hf[0]);
  const float sy = __fmul_rn((float)code_dy(code), g.hf[1]);
  const float sz = __fmul_rn((float)code_dz(code), g.hf[2]);
  const float dx = __fsub_rn(__fadd_rn(pj.x, sx), pi.x);
  const float dy = __fsub_rn(__fadd_rn(pj.y, sy), pi.y);
  const float dz = __fsub_rn(__fadd_rn(pj.z, sz), pi.z);
  return fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
}

__device__ __forceinline__ float4 shfl4(const float4& v, int src) {
  return make_float4(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                     __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src));
}

// A row's n entries (front: the first `front`, the rest at the row's end)
// without the band entries that FP64 excludes, packed at the front; returns
// how many stay.  By the whole warp.
__device__ __noinline__ int build_retest_row(const BuildArgs& A, const Grid& g, uint32_t* row, int rowlen, int front,
                                             int n, float4 pi, int i, int cx, int cy, int cz, int lane) {
  int kept = 0;
  for (int p0 = 0; p0 < n; p0 += 32) {
    const int p = p0 + lane;
    uint32_t w = 0;
    bool keep = p < n;
    if (keep) {
      w = row[p < front ? p : p + rowlen - n];
      if (build_d2(A.pf, g, pi, w) >= A.R2lo)
        keep = exact_within(A.x, A.y, A.z, i, (int64_t)(w & GBMD_IDX_MASK), w >> GBMD_IDX_BITS, cx, cy, cz, g, A.R2);
    }
    const unsigned km = __ballot_sync(0xffffffffu, keep);
    // slots below p0 + 32: this step's entries are read, later ones lie above
    if (keep) row[kept + __popc(km & ((1u << lane) - 1u))] = w;
    kept += __popc(km);
    __syncwarp();
  }
  return kept;
}

// All neighbours (FP32) of an atom whose row overflowed, for the regrow.  By
// the whole warp.
template <bool HALF>
__device__ __noinline__ int build_count(const BuildArgs& A, const Grid& g, const BuildSmem& S, int ncell, float4 pi,
                                        int i, int lane) {
  int n = 0;
  for (int c = 0; c < ncell; ++c)
    for (int q = S.pre[c] + lane; q < S.pre[c + 1]; q += 32) {
      const int k = q + __float_as_int(S.shift[c].x);
      n += (HALF ? k > i : k != i) && build_d2(A.pf, g, pi, (uint32_t)k | S.code[c]) <= A.R2hi;
    }
  return __reduce_add_sync(0xffffffffu, n);
}

template <bool LOOP, bool HALF>
__global__ void __launch_bounds__(BUILD_WARPS * 32, 6) k_build_list_cells(const __grid_constant__ BuildArgs A,
                                                                       const __grid_constant__ Grid g,
                                                                       const int* __restrict__ gate) {
  if (gate && !*gate) return;
  extern __shared__ float4 build_shared[];
  const unsigned FULL = 0xffffffffu;
  const float FAR = 1e18f;
  const int lane = threadIdx.x & 31, half = lane >> 4, hl = lane & 15;
  const int rowlen = build_rowlen(A.maxnb);
  unsigned char* const mine =
      reinterpret_cast<unsigned char*>(build_shared) + (threadIdx.x >> 5) * build_smem(A.maxnb, A.homes);
  BuildSmem& S = *reinterpret_cast<BuildSmem*>(mine);
  uint32_t* const rows = reinterpret_cast<uint32_t*>(mine + sizeof(BuildSmem));
  const int64_t items = A.ncells * A.parts;
  const int64_t warps = LOOP ? (int64_t)gridDim.x * (blockDim.x >> 5) : items;
  for (int64_t item = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); item < items; item += warps) {
    const int64_t cell = item / A.parts;
    const int part = (int)(item - cell * A.parts);
    const int hb = A.cstart[cell], nh = A.cstart[cell + 1] - hb;
    if (part * A.homes >= nh) continue;
    const int cx = (int)(cell % g.nc[0]), cy = (int)((cell / g.nc[0]) % g.nc[1]),
              cz = (int)(cell / ((int64_t)g.nc[0] * g.nc[1]));
    // stencil cell of this lane
    int s_cnt = 0, s_start = 0;
    uint32_t s_code = 0;
    float s_sx = 0.f, s_sy = 0.f, s_sz = 0.f;
    if (lane < 27) {
      const int dx = lane % 3 - 1, dy = (lane / 3) % 3 - 1, dz = lane / 9 - 1;
      const int nx = image_of(cx, dx, g.nc[0]), ny = image_of(cy, dy, g.nc[1]), nz = image_of(cz, dz, g.nc[2]);
      const int64_t cj =
          ((int64_t)(cz + dz - nz * g.nc[2]) * g.nc[1] + (cy + dy - ny * g.nc[1])) * g.nc[0] + (cx + dx - nx * g.nc[0]);
      s_start = A.cstart[cj];
      s_cnt = A.cstart[cj + 1] - s_start;
      s_code = code_of(dx, dy, dz);
      s_sx = __fmul_rn((float)dx, g.hf[0]);
      s_sy = __fmul_rn((float)dy, g.hf[1]);
      s_sz = __fmul_rn((float)dz, g.hf[2]);
    }
    int incl = s_cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += t;
    }
    const int s_pre = incl - s_cnt, total = __shfl_sync(FULL, incl, 31);
    const bool s_any = s_cnt > 0;
    const unsigned any = __ballot_sync(FULL, s_any);
    const int ncell = __popc(any);
    if (s_any) {
      const int c = __popc(any & ((1u << lane) - 1u));
      S.shift[c] = make_float4(__int_as_float(s_start - s_pre), s_sx, s_sy, s_sz);
      S.code[c] = s_code << GBMD_IDX_BITS;
      S.pre[c] = s_pre;
    }
    if (lane == 0) S.pre[ncell] = total;
    // the low half-warp's candidates: whole staging rounds
    const int mid = min(total, (((total + 1) >> 1) + 31) & ~31);
    // box distance bound with a margin far above the FP32 rounding of the
    // walk's d2, so no candidate the walk would keep is dropped
    const float R2keep = A.R2hi * (1.0f + 0x1p-10f);
    int warp_max = 0;
    for (int h0 = part * A.homes; h0 < nh; h0 += A.parts * A.homes) {
      const bool hv = hl < A.homes && h0 + hl < nh;
      const int i = hb + h0 + hl;
      float4 pi = make_float4(FAR, FAR, FAR, 0.f);
      if (hv) pi = A.pf[i];
      // bounding box of the group's atoms (cell frame)
      float3 blo = make_float3(hv ? pi.x : FAR, hv ? pi.y : FAR, hv ? pi.z : FAR);
      float3 bhi = make_float3(hv ? pi.x : -FAR, hv ? pi.y : -FAR, hv ? pi.z : -FAR);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        blo.x = fminf(blo.x, __shfl_xor_sync(FULL, blo.x, o));
        blo.y = fminf(blo.y, __shfl_xor_sync(FULL, blo.y, o));
        blo.z = fminf(blo.z, __shfl_xor_sync(FULL, blo.z, o));
        bhi.x = fmaxf(bhi.x, __shfl_xor_sync(FULL, bhi.x, o));
        bhi.y = fmaxf(bhi.y, __shfl_xor_sync(FULL, bhi.y, o));
        bhi.z = fmaxf(bhi.z, __shfl_xor_sync(FULL, bhi.z, o));
      }
      // shared-memory addresses of the lane's row end and of its next slot
      const uint32_t row = (uint32_t)__cvta_generic_to_shared(rows + (hv ? hl : 0) * rowlen);
      const uint32_t first = half ? row + 4 * (rowlen - 1) : row;
      uint32_t put = first;
      const int step = half ? -4 : 4;
      float thr = hv ? A.R2hi : -1.f;  // -1: no candidate is a hit
      float far2 = -1.f;               // largest d2 of the hits
      bool full = false;
      const float2 npx = make_float2(-pi.x, -pi.x), npy = make_float2(-pi.y, -pi.y), npz = make_float2(-pi.z, -pi.z);
      const uint32_t self = (uint32_t)i;
      const float4* const cand = S.chunk + half * (BUILD_CHUNK + 4);
      // Predicated, so that eight tests are one straight line.  An atom never
      // pairs with itself: its images sit at least one box edge >= R away, so
      // only its entry of the home cell is itself.
      auto test = [&](float d2, float wf) {
        const uint32_t w = __float_as_uint(wf);
        if (HALF)
          asm volatile("{\n.reg .pred p, q;\nsetp.gt.s32 q, %6, %7;\nsetp.le.and.f32 p, %2, %3, q;\n"
                       "@p st.shared.u32 [%0], %4;\n@p max.f32 %1, %1, %2;\n@p add.s32 %0, %0, %5;\n}"
                       : "+r"(put), "+f"(far2)
                       : "f"(d2), "f"(thr), "r"(w), "r"(step), "r"((int)(w & GBMD_IDX_MASK)), "r"(i)
                       : "memory");
        else
          asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 q, %4, %6;\nsetp.le.and.f32 p, %2, %3, q;\n"
                       "@p st.shared.u32 [%0], %4;\n@p max.f32 %1, %1, %2;\n@p add.s32 %0, %0, %5;\n}"
                       : "+r"(put), "+f"(far2)
                       : "f"(d2), "f"(thr), "r"(w), "r"(step), "r"(self)
                       : "memory");
      };
      for (int qa = 0; qa < mid; qa += BUILD_CHUNK) {
        __syncwarp();  // the last chunk's reads, and S, are done
        BuildRound lo, hi;
        lo.fetch(S, A.pf, s_pre, s_any, qa, 0, mid, false, lane);
        hi.fetch(S, A.pf, s_pre, s_any, total - qa - BUILD_CHUNK, mid, total, true, lane);
        const int m0 = lo.store(S.chunk, lane, blo, bhi, R2keep);
        const int m1 = hi.store(S.chunk + BUILD_CHUNK + 4, lane, blo, bhi, R2keep);
        const int m = max(m0, m1);
        __syncwarp();
        for (int t = 0; t < m; t += 8) {
          // fewer than 8 free slots: the row (more than maxnb entries) has overflowed
          if (half ? put < row + 4 * 7 : put > row + 4 * (rowlen - 8)) {
            thr = -1.f;
            full = true;
          }
#pragma unroll
          for (int u = 0; u < 8; u += 4) {
            if (u && t + u >= m) break;
            const float4* const c = cand + (t + u) / 4;
            const float4 x = c[0], y = c[BUILD_CHUNK / 4], z = c[BUILD_CHUNK / 2], w = c[3 * BUILD_CHUNK / 4];
            const float2 dx0 = __fadd2_rn(make_float2(x.x, x.y), npx), dx1 = __fadd2_rn(make_float2(x.z, x.w), npx);
            const float2 dy0 = __fadd2_rn(make_float2(y.x, y.y), npy), dy1 = __fadd2_rn(make_float2(y.z, y.w), npy);
            const float2 dz0 = __fadd2_rn(make_float2(z.x, z.y), npz), dz1 = __fadd2_rn(make_float2(z.z, z.w), npz);
            const float2 d0 = __ffma2_rn(dx0, dx0, __ffma2_rn(dy0, dy0, __fmul2_rn(dz0, dz0)));
            const float2 d1 = __ffma2_rn(dx1, dx1, __ffma2_rn(dy1, dy1, __fmul2_rn(dz1, dz1)));
            test(d0.x, w.x);
            test(d0.y, w.y);
            test(d1.x, w.z);
            test(d1.y, w.w);
          }
        }
      }
      __syncwarp();
      // entries at the front and in all (stored); full, far2 of either half
      const int mycnt = (half ? (int)(first - put) : (int)(put - first)) >> 2;
      int front = __shfl_sync(FULL, mycnt, hl), n = front + __shfl_sync(FULL, mycnt, hl + 16);
      full = (__ballot_sync(FULL, full) & (0x10001u << hl)) != 0;
      far2 = fmaxf(far2, __shfl_xor_sync(FULL, far2, 16));
      const bool over = hv && (full || n > A.maxnb);
      int found = n;
      unsigned todo = __ballot_sync(FULL, hv && half == 0 && !over && far2 >= A.R2lo);
      while (todo) {
        const int h = __ffs(todo) - 1;
        todo &= todo - 1;
        const int k = build_retest_row(A, g, rows + h * rowlen, rowlen, __shfl_sync(FULL, front, h),
                                       __shfl_sync(FULL, n, h), shfl4(pi, h), hb + h0 + h, cx, cy, cz, lane);
        if (hl == h) front = n = found = k;
      }
      todo = __ballot_sync(FULL, half == 0 && over);
      while (todo) {
        const int h = __ffs(todo) - 1;
        todo &= todo - 1;
        const int k = build_count<HALF>(A, g, S, ncell, shfl4(pi, h), hb + h0 + h, lane);
        if (hl == h) found = k;
      }
      if (!hv) n = found = 0;
      // rows out: unit (r, h, t) is what lane t of atom h's T lanes reads of
      // list row r, V adjacent words.  An overflowed row's first maxnb slots
      // hold entries too (stored counts above maxnb), so a reader stays in
      // bounds until the host sees the error.
      const int nrow = (min(__reduce_max_sync(FULL, n), A.maxnb) + A.W - 1) >> A.wsh;
      const int units = nrow << (4 + A.tsh), T = 1 << A.tsh;
      for (int u0 = 0; u0 < units; u0 += 32) {
        const int u = u0 + lane, r = u >> (4 + A.tsh), h = (u >> A.tsh) & 15, t = u & (T - 1);
        const int hn = __shfl_sync(FULL, n, h), hf = __shfl_sync(FULL, front, h);
        if (u < units && r * A.W < hn) {
          const uint32_t* const from = rows + h * rowlen;
          auto entry = [&](int q) {
            const int p = (r << A.wsh) + (q << A.tsh) + t;
            return p >= hn ? 0u : from[p < hf ? p : p + rowlen - hn];
          };
          uint32_t* const to = A.nbr + (size_t)r * A.stride + (size_t)(hb + h0 + h) * A.W;
          if (A.wsh - A.tsh == 2) *reinterpret_cast<uint4*>(to + 4 * t) = make_uint4(entry(0), entry(1), entry(2), entry(3));
          else to[t] = entry(0);
        }
      }
      if (hv && half == 0) {
        A.nnb[i] = found;
        if (found > A.maxnb) atomicOr(&A.err[ERRW_FLAGS], GBMD_DEVERR_NBR_OVERFLOW);
        warp_max = max(warp_max, found);
      }
    }
    warp_max = __reduce_max_sync(FULL, warp_max);
    if (lane == 0 && warp_max > 0) atomicMax(&A.err[ERRW_MAXNB], warp_max);
    __syncwarp();  // the next cell overwrites S
  }
}

// The same list where rows are long: a warp per atom, 32 candidates at a time,
// the hits straight to the row in global memory.  The walk above holds 16 rows
// a warp in shared memory: at BUILD_LONG entries an SM has 3 of its warps, and
// longer rows need fewer atoms a warp, up to 51,000 entries where one row does
// not fit.  Rebuild, us, walk above (fewer atoms a warp from 3,000 entries) / this:
// 256,000 atoms, capacity 560: 1,492 / 2,091; 728: 2,217 / 2,485; 1,000: 3,761 /
// 3,035; 62,500 atoms, 560: 623 / 623; 1,000: 1,330 / 861; 2,750: 8,400 / 2,270;
// 8,788 atoms, 6,200: 39,000 / 3,290; 19,600: 6,150,000 / 157,000.
template <bool HALF>
__global__ void __launch_bounds__(128) k_build_list_long(const __grid_constant__ BuildArgs A,
                                                         const __grid_constant__ Grid g,
                                                         const int* __restrict__ gate) {
  if (gate && !*gate) return;
  const int lane = threadIdx.x & 31;
  int longest = 0;
  for (int64_t a = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; a < A.n;
       a += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int i = (int)a, cp = A.cellpack[a], cx = cp & 1023, cy = (cp >> 10) & 1023, cz = cp >> 20;
    const float4 pi = A.pf[a];
    uint32_t* const row = A.nbr + (size_t)a * A.W;
    int found = 0;
    for (int s = 0; s < 27; ++s) {
      const int dx = s % 3 - 1, dy = (s / 3) % 3 - 1, dz = s / 9 - 1;
      const int64_t x = cx + dx - image_of(cx, dx, g.nc[0]) * g.nc[0], y = cy + dy - image_of(cy, dy, g.nc[1]) * g.nc[1],
                    z = cz + dz - image_of(cz, dz, g.nc[2]) * g.nc[2], c = (z * g.nc[1] + y) * g.nc[0] + x;
      const uint32_t code = code_of(dx, dy, dz), self = (uint32_t)i;
      const int end = A.cstart[c + 1];
      for (int q = A.cstart[c]; q < end; q += 32) {
        const int k = q + lane;
        const uint32_t w = (uint32_t)k | code << GBMD_IDX_BITS;
        bool hit = k < end && (HALF ? k > i : w != self);
        if (hit) {
          const float d2 = build_d2(A.pf, g, pi, w);
          hit = d2 <= A.R2hi;
          if (hit && d2 >= A.R2lo) hit = exact_within(A.x, A.y, A.z, i, k, code, cx, cy, cz, g, A.R2);
        }
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        const int p = found + __popc(hits & ((1u << lane) - 1u));
        if (hit && p < A.maxnb) row[(size_t)(p >> A.wsh) * A.stride + list_word(p & (A.W - 1), A.wsh, A.tsh)] = w;
        found += __popc(hits);
      }
    }
    if (lane == 0) {
      A.nnb[a] = found;
      if (found > A.maxnb) atomicOr(&A.err[ERRW_FLAGS], GBMD_DEVERR_NBR_OVERFLOW);
    }
    longest = max(longest, found);
  }
  if (lane == 0 && longest > 0) atomicMax(&A.err[ERRW_MAXNB], longest);
}

static inline unsigned nblk(int64_t n, int b) { return (unsigned)((n + b - 1) / b); }

// Blocks of a rebuild-chain launch.  Ungated launches cover the data once;
// gated ones (launched every step, mostly to find the gate closed) get at most
// per_sm blocks per SM (no more than fit at once) and stride over the data,
// so a closed gate costs a few microseconds instead of a full grid of empty
// blocks.
unsigned chain_blocks(const gbmd_context* c, int64_t items, int per_block, const int* gate, int per_sm) {
  const unsigned full = nblk(items, per_block);
  if (!gate || c->full_chain_grids) return full;
  const unsigned cap = (unsigned)(per_sm * (c->nsm > 0 ? c->nsm : 1));
  return full < cap ? full : cap;
}

void launch_posf(gbmd_context* c, const int* gate) {
  if (c->n == 0) return;
  k_posf<<<chain_blocks(c, c->n, 256, gate, 8), 256, 0, c->stream>>>(c->n, c->X(), c->Y(), c->Z(), c->TYPE(),
                                                                   c->cellpack, c->grid, c->POSF(), c->POSD(),
                                                                   gate);
}

static int build_list(gbmd_context* c, const int* gate) {
  const double R = c->rlist;
  const double R2 = R * R;
  float R2lo, R2hi;
  band_limits(R, c->grid_tol, R2lo, R2hi);
  const int64_t npad = ((c->n + 31) / 32) * 32;
  const int W = list_width(c);
  const int64_t stride = npad * W;
  const int64_t need = (int64_t)(c->maxnb / W) * stride;
  if (need > c->nbr_cap) {
    cudaFree(c->nbr);
    c->nbr = nullptr;
    c->nbr_cap = 0;
    GBMD_CUDA(c, dev_malloc(c, (void**)&c->nbr, sizeof(uint32_t) * (size_t)need));
    c->nbr_cap = need;
  }
  c->npad = npad;
  BuildArgs A;
  A.ncells = c->grid.ncells;
  A.pf = c->POSF();
  A.x = c->X(); A.y = c->Y(); A.z = c->Z();
  A.cstart = c->cell_start;
  A.R2 = R2;
  A.R2lo = R2lo;
  A.R2hi = R2hi;
  A.nbr = c->nbr;
  A.nnb = c->nnb;
  A.maxnb = c->maxnb;
  A.W = W;
  A.wsh = log2_of(W);
  A.tsh = log2_of(c->tpa);
  A.stride = stride;
  A.err = c->d_err;
  A.n = c->n;
  A.cellpack = c->cellpack;
  A.homes = BUILD_G;  // as a constant in the kernel it costs 2 % (16.6 M-atom mixture: 12.03 -> 12.28 ms)
  if (c->maxnb >= BUILD_LONG) {
    auto kern = c->newton3 ? k_build_list_long<true> : k_build_list_long<false>;
    kern<<<chain_blocks(c, c->n, 4, gate, 8), 128, 0, c->stream>>>(A, c->grid, gate);
    return GBMD_OK;
  }
  const size_t per_warp = build_smem(c->maxnb, BUILD_G);
  // the widest blocks of which an SM holds several
  int nw = BUILD_WARPS;
  while (nw > 1 && nw * per_warp > 56 * 1024) nw >>= 1;
  // a second warp for a cell's second group while cells are few (an SM holds
  // some 20 warps of this kernel)
  A.parts = c->grid.ncells < 20ll * c->nsm ? 2 : 1;
  const int64_t items = c->grid.ncells * A.parts;
  const bool loop = gate && !c->full_chain_grids;  // capped grid striding over the cells
  auto kern = loop ? (c->newton3 ? k_build_list_cells<true, true> : k_build_list_cells<true, false>)
                   : (c->newton3 ? k_build_list_cells<false, true> : k_build_list_cells<false, false>);
  const size_t smem = nw * per_warp, most = 200 * 1024;
  if (smem > 48 * 1024)
    GBMD_CUDA(c, cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
  const int per_sm = (int)std::max<size_t>(1, 220 * 1024 / (smem + 1024));
  const unsigned blocks = loop ? chain_blocks(c, items, nw, gate, std::min(per_sm, 8)) : nblk(items, nw);
  kern<<<blocks, 32 * nw, smem, c->stream>>>(A, c->grid, gate);
  return GBMD_OK;
}

// The rebuild chain for the list in c->nbr / c->nnb / c->maxnb at radius
// c->rlist (the outer list's buffers and radius while an OuterScope holds).
static int rebuild_chain(gbmd_context* c, bool check_capacity, const int* gate) {
  if (gate && (!c->list_valid || !c->grid_valid || c->maxnb <= 0))
    return set_error(c, GBMD_ERR_INVALID, "gated rebuild needs a built list");
  if (!c->box_set) return set_error(c, GBMD_ERR_INVALID, "box not set");
  if (c->pot == GBMD_POT_NONE) return set_error(c, GBMD_ERR_INVALID, "no potential set");
  if (c->n == 0) {
    c->list_valid = true;
    return GBMD_OK;
  }
  const double R = c->rlist;
  if (!c->grid_valid) {
    int nc[3];
    const int rc = grid_dims(c->lo, c->hi, R, nc);
    if (rc != 0)
      return set_error(c, GBMD_ERR_INVALID, "box edge shorter than neighbour radius %g%s", R,
                       c->list_buffer > 0.0 ? " (list radius + list buffer)" : "");
    Grid& g = c->grid;
    g.ncells = (int64_t)nc[0] * nc[1] * nc[2];
    if (g.ncells > (1ll << 27)) return set_error(c, GBMD_ERR_TOO_LARGE, "too many cells");
    for (int d = 0; d < 3; ++d) {
      g.nc[d] = nc[d];
      g.L[d] = c->hi[d] - c->lo[d];
      g.h[d] = g.L[d] / nc[d];
      g.hf[d] = (float)g.h[d];
      g.hh[d] = 0.5f * g.hf[d];
      g.lo[d] = c->lo[d];
    }
    // not in Grid: the exact tests take it by value, and 16 bytes more put it on
    // the stack (list builder 215 -> 238 us, 256,000-atom LJ)
    c->grid_tol = band_tol(R, std::max(g.h[0], std::max(g.h[1], g.h[2])));
    c->grid_reach = R;
    int ra = ensure_cells(c, g.ncells);
    if (ra) return ra;
    c->grid_valid = true;
    if ((ra = set_bands(c))) return ra;
  }
  Grid& g = c->grid;
  BoxArgs b;
  for (int d = 0; d < 3; ++d) {
    b.lo[d] = c->lo[d];
    b.hi[d] = c->hi[d];
    b.L[d] = g.L[d];
    b.inv_h[d] = (double)g.nc[d] / g.L[d];
    b.klo[d] = order_key_host(c->lo[d]);
    b.khi[d] = order_key_host(c->hi[d]);
    b.nc[d] = g.nc[d];
  }
  const int64_t n = c->n;
  cudaStream_t s = c->stream;
  // cell_fill is zero here: cleared when allocated, counted up by k_wrap_bin and
  // down again by k_scatter, with nothing between the two that can fail
  k_wrap_bin<<<chain_blocks(c, n, 256, gate, 8), 256, 0, s>>>(n, c->X(), c->Y(), c->Z(), b, c->cell_of, c->cell_fill,
                                                            c->d_err, gate);
  scan(c, c->cell_fill, c->cell_start, g.ncells, gate);
  k_scatter<<<chain_blocks(c, n, 256, gate, 8), 256, 0, s>>>(n, c->cell_of, c->cell_start, c->cell_fill, c->order,
                                                           gate);
  k_cell_rank<<<chain_blocks(c, g.ncells * 32, 256, gate, 8), 256, 0, s>>>(g.ncells, c->cell_start, c->order, c->ID(),
                                                                       c->USER(),
                                                        c->src, gate);
  GatherArgs ga;
  const int o = c->cur, os = c->cur_s;
  ga.r0 = c->rbuf[o]; ga.r1 = c->rbuf[o ^ 1];
  ga.v0 = c->vbuf[os]; ga.v1 = c->vbuf[os ^ 1];
  ga.a0 = c->abuf[os]; ga.a1 = c->abuf[os ^ 1];
  ga.t0 = c->typeb[os]; ga.t1 = c->typeb[os ^ 1];
  ga.i0 = c->idb[os]; ga.i1 = c->idb[os ^ 1];
  ga.u0 = c->userb[os]; ga.u1 = c->userb[os ^ 1];
  ga.ep0 = c->ep; ga.ep1 = c->stage;
  ga.cap = c->cap;
  // the gather copies go with the buffer that holds the sorted positions in
  // the end: the spare one, or under a gate the current one
  const int to = gate ? o : o ^ 1;
  k_gather<<<chain_blocks(c, n, 256, gate, 8), 256, 0, s>>>(n, c->src, ga, c->cell_of, g, c->cellpack, c->posf[to],
                                                          c->posd[to], gate);
  if (gate) {
    k_copy_back<<<chain_blocks(c, n, 256, gate, 8), 256, 0, s>>>(n, ga, gate);
  } else {
    GBMD_CUDA(c, cudaMemcpyAsync(c->ep, c->stage, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    c->cur ^= 1;
    c->cur_s ^= 1;
  }
  if (c->maxnb <= 0) {
    // first estimate: 1.35x the mean count of an ideal gas at this density
    const double V = g.L[0] * g.L[1] * g.L[2];
    const double mean = (double)n / V * 4.18879020478639 * R * R * R;
    int m = (int)(mean * 1.35) + 16;
    c->maxnb = ((m + list_width(c) - 1) / list_width(c)) * list_width(c);
  }
  int rc = build_list(c, gate);
  if (rc) return rc;
  c->list_valid = true;
  if (check_capacity) {
    rc = sync_error_word(c);
    if (c->h_err[ERRW_FLAGS] & GBMD_DEVERR_LOST_ATOM)
      return set_error(c, GBMD_ERR_LOST_ATOM, "%d atoms left the box by more than one image",
                       c->h_err[ERRW_LOST]);
    const int maxc = c->h_err[ERRW_MAXNB];
    if (maxc > c->maxnb) {
      int m = (int)(maxc * 1.2) + 8;
      c->maxnb = ((m + list_width(c) - 1) / list_width(c)) * list_width(c);
      GBMD_CUDA(c, cudaMemsetAsync(c->d_err + ERRW_FLAGS, 0, sizeof(int) * 2, s));  // flags, max count
      rc = build_list(c, nullptr);
      if (rc) return rc;
      rc = sync_error_word(c);
      if (c->h_err[ERRW_FLAGS] & GBMD_DEVERR_NBR_OVERFLOW)
        return set_error(c, GBMD_ERR_NEIGHBOR_OVERFLOW, "neighbour list overflow after regrow");
    }
  }
  return GBMD_OK;
}

// --- two-level list ---------------------------------------------------------
//
// With a list buffer d set, the sort into cells and the cell walk build an
// outer list of radius R + d (R = rcut + skin), and every rebuild filters the
// list the pair kernels read (radius R) from it: the outer row's entries that
// lie within R now, in the outer row's order.  The filter is complete while
// no atom has moved more than d/2 since the outer build: a pair within R now
// was then within R + d.  So a rebuild first tests every atom against d/2
// from its position at the outer build and runs the outer build again only
// when one moved that far.  Between outer builds the atoms keep their cells
// and are not wrapped into the box, so the cell-relative FP32 copies, the
// stencil codes and the FP64 band re-test all see continuous coordinates.
// The filtered list holds the same pairs as a fresh build; its rows follow
// the cell order of the outer build.

bool two_level(const gbmd_context* c) { return c->list_buffer > 0.0; }

void free_outer(gbmd_context* c) {
  cudaFree(c->rout);
  cudaFree(c->nnb_out);
  c->rout = nullptr;
  c->nnb_out = nullptr;
  c->outer_cap = 0;
  c->outer_valid = false;
}

static int ensure_outer(gbmd_context* c) {
  if (c->rout && c->outer_cap >= c->cap) return GBMD_OK;
  free_outer(c);
  GBMD_CUDA(c, dev_malloc(c, (void**)&c->rout, sizeof(double) * 3 * c->cap));
  GBMD_CUDA(c, dev_malloc(c, (void**)&c->nnb_out, sizeof(int32_t) * c->cap));
  c->outer_cap = c->cap;
  return GBMD_OK;
}

// The outer list's buffers and radius in the fields the rebuild chain uses.
struct OuterScope {
  gbmd_context* c;
  double saved;
  explicit OuterScope(gbmd_context* ctx) : c(ctx), saved(ctx->rlist) {
    swap();
    c->rlist = saved + c->list_buffer;
  }
  ~OuterScope() {
    c->rlist = saved;
    swap();
  }
  void swap() {
    std::swap(c->nbr, c->nbr_out);
    std::swap(c->nnb, c->nnb_out);
    std::swap(c->nbr_cap, c->nbr_out_cap);
    std::swap(c->maxnb, c->maxnb_out);
  }
};

// flag = 1 when some atom moved more than sqrt(thr2) since the outer build
// (|dr|^2 summed x, y, z without contraction); with a gate, only when *gate
__global__ void k_outer_check(int64_t n, const double* __restrict__ x, const double* __restrict__ y,
                              const double* __restrict__ z, const double* __restrict__ rout, int64_t cap,
                              double thr2, const int* __restrict__ gate, int* __restrict__ flag) {
  if (gate && !*gate) return;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const double dx = __dsub_rn(x[p], rout[p]), dy = __dsub_rn(y[p], rout[cap + p]),
                 dz = __dsub_rn(z[p], rout[2 * cap + p]);
    const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    if (d2 > thr2) *flag = 1;
  }
}

// positions at a gated outer build; thread 0 counts the build
__global__ void k_save_outer(int64_t n, const double* __restrict__ r, double* __restrict__ rout, int64_t cap,
                             const int* __restrict__ gate, int* __restrict__ count) {
  if (!*gate) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(count, 1);
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int d = 0; d < 3; ++d) rout[d * cap + p] = r[d * cap + p];
  }
}

// One thread per atom: the entries of its outer row within R now, in the
// order of the row's words.
// The FP32 distance of the cell-relative copies (the builder's expression)
// decides outside the band [R2lo, R2hi]; band entries are re-tested in
// FP64 with the pair-set rounding.  A row never grows, so the list has the
// outer list's capacity.  V4 (4 entries per lane
// and load): the row is read 4 words per 16-byte load with the next load in
// flight, and the 4 neighbour positions are gathered together.
struct FilterArgs {
  int64_t n;
  const float4* pf;
  const double *x, *y, *z;
  const int32_t* cellpack;
  const uint32_t* outer;
  const int32_t* nnb_out;
  uint32_t* nbr;
  int32_t* nnb;
  int maxnb_out, W, wsh, tsh;
  int64_t stride;
  double R2;
  float R2lo, R2hi;
};

__device__ __forceinline__ bool filter_keep(const FilterArgs& A, const Grid& g, int64_t i, const float4& pi,
                                            uint32_t w, const float4& pj, int cx, int cy, int cz) {
  const uint32_t code = w >> GBMD_IDX_BITS;
  const float sx = __fmul_rn((float)code_dx(code), g.hf[0]);
  const float sy = __fmul_rn((float)code_dy(code), g.hf[1]);
  const float sz = __fmul_rn((float)code_dz(code), g.hf[2]);
  const float dx = __fsub_rn(__fadd_rn(pj.x, sx), pi.x);
  const float dy = __fsub_rn(__fadd_rn(pj.y, sy), pi.y);
  const float dz = __fsub_rn(__fadd_rn(pj.z, sz), pi.z);
  const float d2f = fmaf(dx, dx, fmaf(dy, dy, __fmul_rn(dz, dz)));
  if (d2f > A.R2hi) return false;
  if (d2f < A.R2lo) return true;
  return exact_within(A.x, A.y, A.z, i, (int64_t)(w & GBMD_IDX_MASK), code, cx, cy, cz, g, A.R2);
}

template <bool V4>
__global__ void __launch_bounds__(256) k_filter_list(FilterArgs A, Grid g, const int* __restrict__ gate) {
  if (gate && !*gate) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < A.n; i += (int64_t)gridDim.x * blockDim.x) {
    const int nn = min(A.nnb_out[i], A.maxnb_out);
    const float4 pi = A.pf[i];
    const int cp = A.cellpack[i];
    const int cx = cp & 1023, cy = (cp >> 10) & 1023, cz = cp >> 20;
    const uint32_t* orow = A.outer + (size_t)i * A.W;
    uint32_t* row = A.nbr + (size_t)i * A.W;
    int cnt = 0;
    auto put = [&](uint32_t w) {
      row[(size_t)(cnt >> A.wsh) * A.stride + list_word(cnt & (A.W - 1), A.wsh, A.tsh)] = w;
      ++cnt;
    };
    if (V4) {
      // words k .. k + 3 (k a multiple of 4) of row k / W are one lane's
      // aligned uint4: its entries q * T + lane, q = 0 .. 3.  Rows hold
      // maxnb_out words, a multiple of W, so the loads of every row that
      // holds an entry stay in
      auto group = [&](int k) {
        return *reinterpret_cast<const uint4*>(orow + (size_t)(k >> A.wsh) * A.stride + (k & (A.W - 1)));
      };
      const int ng = ((nn + A.W - 1) >> A.wsh) << (A.wsh - 2);
      auto entry_of = [&](int k, int q) {  // which entry word k + q holds
        return (k & ~(A.W - 1)) + (q << A.tsh) + ((k & (A.W - 1)) >> 2);
      };
      uint4 cur = ng > 0 ? group(0) : make_uint4(0u, 0u, 0u, 0u);
      for (int t = 0; t < ng; ++t) {
        const int k0 = t << 2;
        uint4 nxt = cur;
        if (t + 1 < ng) nxt = group(k0 + 4);
        const uint32_t e[4] = {cur.x, cur.y, cur.z, cur.w};
        float4 pj[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) pj[q] = A.pf[entry_of(k0, q) < nn ? (int64_t)(e[q] & GBMD_IDX_MASK) : i];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (entry_of(k0, q) < nn && filter_keep(A, g, i, pi, e[q], pj[q], cx, cy, cz)) put(e[q]);
        cur = nxt;
      }
    } else {
      for (int k = 0; k < nn; ++k) {
        const uint32_t w = orow[(size_t)(k >> A.wsh) * A.stride + list_word(k & (A.W - 1), A.wsh, A.tsh)];
        const float4 pj = A.pf[w & GBMD_IDX_MASK];
        if (filter_keep(A, g, i, pi, w, pj, cx, cy, cz)) put(w);
      }
    }
    A.nnb[i] = cnt;
  }
}

// The outer list: the rebuild chain at radius R + d into the outer buffers,
// then the positions it leaves saved for the displacement test.
static int outer_chain(gbmd_context* c, bool check_capacity, const int* gate) {
  int rc;
  if (!gate) {
    if ((rc = ensure_outer(c))) return rc;
  } else if (!c->rout || c->outer_cap < c->n) {
    return set_error(c, GBMD_ERR_INVALID, "gated rebuild needs an outer list");
  }
  {
    const OuterScope on(c);
    rc = rebuild_chain(c, check_capacity, gate);
  }
  if (rc) return rc;
  if (gate) {
    k_save_outer<<<chain_blocks(c, c->n, 256, gate, 8), 256, 0, c->stream>>>(c->n, c->rbuf[c->cur], c->rout, c->cap,
                                                                          gate, c->d_err + ERRW_OUTER_BUILDS);
  } else {
    for (int d = 0; d < 3; ++d)
      GBMD_CUDA(c, cudaMemcpyAsync(c->rout + d * c->cap, c->rbuf[c->cur] + d * c->cap, sizeof(double) * c->n,
                                   cudaMemcpyDeviceToDevice, c->stream));
    c->outer_builds++;
    c->outer_valid = true;
  }
  return GBMD_OK;
}

static int filter_list(gbmd_context* c, const int* gate) {
  const int W = list_width(c);
  const int64_t stride = c->npad * W;
  const int64_t need = (int64_t)(c->maxnb_out / W) * stride;
  if (need > c->nbr_cap) {
    if (gate || c->capturing) return set_error(c, GBMD_ERR_INVALID, "the list outgrew its buffer in a gated rebuild");
    if (c->nbr) cudaFree(c->nbr);
    c->nbr = nullptr;
    c->nbr_cap = 0;
    GBMD_CUDA(c, dev_malloc(c, (void**)&c->nbr, sizeof(uint32_t) * (size_t)need));
    c->nbr_cap = need;
  }
  c->maxnb = c->maxnb_out;
  const double R2 = c->rlist * c->rlist;
  float R2lo, R2hi;
  band_limits(c->rlist, c->grid_tol, R2lo, R2hi);
  FilterArgs A;
  A.n = c->n;
  A.pf = c->POSF();
  A.x = c->X(); A.y = c->Y(); A.z = c->Z();
  A.cellpack = c->cellpack;
  A.outer = c->nbr_out;
  A.nnb_out = c->nnb_out;
  A.nbr = c->nbr;
  A.nnb = c->nnb;
  A.maxnb_out = c->maxnb_out;
  A.W = W;
  A.wsh = log2_of(W);
  A.tsh = log2_of(c->tpa);
  A.stride = stride;
  A.R2 = R2;
  A.R2lo = R2lo;
  A.R2hi = R2hi;
  const unsigned blocks = gate ? chain_blocks(c, c->n, 256, gate, 8) : nblk(c->n, 256);
  if (!gate && !c->capturing) ensure_bpair(c);
  if (c->vec == 4) k_filter_list<true><<<blocks, 256, 0, c->stream>>>(A, c->grid, gate);
  else k_filter_list<false><<<blocks, 256, 0, c->stream>>>(A, c->grid, gate);
  c->list_valid = true;
  if (!gate) c->list_builds++;
  return GBMD_OK;
}

// More lanes per atom while the atoms alone cannot fill the chip; then the
// fewest, since each doubling adds a step of the shuffle reduction and of the
// epilogue's exchange.  Two lanes win longest where the pair work per entry is
// largest, because their gathers touch fewer cache lines (ListRows).
// Measured on GB300, us, lanes 1 / 2 / 4 / 8 / 16; force evaluations:
//   eam_alloy, one element      4,000 atoms    36 / 24 / 18 / 15 / 13
//                              16,384          39 / 28 / 22 / 18 / 22
//   LJ                          4,000          14 / 10 /  8 /  6 /  6
//                              16,384          14 / 10 /  8 /  8 /  9
//                              32,000          14 / 12 / 11 / 10 / 14
// and 20 NVE steps with two rebuilds, lanes 1 / 2 / 4:
//   eam_alloy, one element     32,000           760 / 549 / 489
//                              62,500           878 / 726 / 786
//                             256,000         2,364 / 2,335 / 2,521
//                             864,000         7,013 / 7,007 / 7,769
//                           4,000,000        29,841 / 30,355 / 33,621
//   two elements              256,000         3,425 / 3,125 / 3,096
//                           2,048,000        21,073 / 20,706 / 22,275
//   LJ                         32,000           513 / 440 / 428
//                              62,500           630 / 577 / 591
//                             256,000         1,597 / 1,557 / 1,653
//   LJ mixture                253,000         2,104 / 2,098 / 2,192
// The analytic EAM functions, bound by the SFU, take one lane where LJ takes two.
void choose_launch(gbmd_context* c) {
  if (c->launch_set) return;
  const bool alloy = c->pot == GBMD_POT_EAM_ALLOY, single = alloy && c->eam.nel == 1;
  const bool lj = c->pot == GBMD_POT_LJ || c->pot == GBMD_POT_LJ_MULTI;
  int tpa = 1;
  if (c->n <= 8192) tpa = 16;
  else if (c->n <= 24576) tpa = 8;
  else if (c->n <= (alloy && !single ? 327680 : 49152)) tpa = 4;
  else if (single ? c->n <= 1500000 : alloy || (lj && c->n <= 262144)) tpa = 2;
  if (c->newton3 || c->staged) tpa = 1;  // the layout of the half list and of the staged kernels
  c->vec = 4;
  c->block = tpa == 1 || (tpa == 2 && alloy && !single) ? 256 : 128;
  if (tpa == c->tpa) return;
  c->tpa = tpa;
  const int W = list_width(c);
  if (c->maxnb > 0) c->maxnb = ((c->maxnb + W - 1) / W) * W;
  if (c->maxnb_out > 0) c->maxnb_out = ((c->maxnb_out + W - 1) / W) * W;
}

// Words of the list the pair kernels read.
static int64_t list_words(const gbmd_context* c) {
  return (int64_t)(c->maxnb / list_width(c)) * c->npad * list_width(c);
}

void ensure_bpair(gbmd_context* c) {
  if (c->precision != GBMD_PRECISION_MIXED || c->pot != GBMD_POT_EAM_ALLOY || c->eam.nel != 1 || c->newton3 ||
      c->vec != 4) {
    release_bpair(c);  // nothing reads it
    return;
  }
  // without them the force pass forms the pair terms again
  if (!c->f0 && cudaMalloc(&c->f0, sizeof(float4) * c->cap) != cudaSuccess) {
    (void)cudaGetLastError();
    c->f0 = nullptr;
    return;
  }
  const int64_t need = list_words(c);
  if (need <= c->bpair_cap) return;
  release_bpair(c);
  // no more than half of what is free: the caller's memory comes first
  size_t free_bytes = 0, total = 0;
  if (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess || sizeof(float) * (size_t)need > free_bytes / 2) return;
  if (cudaMalloc(&c->bpair, sizeof(float) * (size_t)need) == cudaSuccess) c->bpair_cap = need;
  else (void)cudaGetLastError(), c->bpair = nullptr;
}

int rebuild(gbmd_context* c, bool check_capacity, const int* gate) {
  if (!gate && !c->capturing) choose_launch(c);
  if (c->n == 0 || !two_level(c)) {
    const int rc = rebuild_chain(c, check_capacity, gate);
    if (rc == GBMD_OK && !gate) {
      c->list_builds++;
      if (!c->capturing) ensure_bpair(c);
    }
    return rc;
  }
  if (gate && !c->outer_valid) return set_error(c, GBMD_ERR_INVALID, "gated rebuild needs an outer list");
  const int rc = outer_chain(c, check_capacity, gate);
  if (rc) return rc;
  return filter_list(c, gate);
}

static int outer_body(gbmd_context* c, const int* flag) {
  c->full_chain_grids = true;
  const int rc = outer_chain(c, false, flag);
  c->full_chain_grids = false;
  return rc;
}

int rebuild_two_level(gbmd_context* c, bool check_capacity, const int* gate) {
  if (c->n == 0 || !c->outer_valid || !c->list_valid || !c->grid_valid) {
    if (gate || c->capturing) return set_error(c, GBMD_ERR_INVALID, "gated or captured rebuild needs an outer list");
    return rebuild(c, check_capacity, nullptr);
  }
  int* flag = c->d_err + ERRW_OUTER;
  cudaStream_t s = c->stream;
  GBMD_CUDA(c, cudaMemsetAsync(flag, 0, sizeof(int), s));
  const double h = 0.5 * c->list_buffer;
  const double thr2 = h * h * (1.0 - 0x1p-20);  // a margin far above the rounding of the test
  const unsigned blocks = gate ? chain_blocks(c, c->n, 256, gate, 8) : nblk(c->n, 256);
  k_outer_check<<<blocks, 256, 0, s>>>(c->n, c->X(), c->Y(), c->Z(), c->rout, c->cap, thr2, gate, flag);
  int rc;
  if (gate) {
    // the flag stays 0 unless the gate is open: it gates the outer chain
    rc = outer_chain(c, false, flag);
  } else if (c->capturing) {
    rc = capture_if(c, flag, outer_body);
  } else {
    if ((rc = sync_error_word(c))) return rc;
    rc = c->h_err[ERRW_OUTER] ? outer_chain(c, check_capacity, nullptr) : GBMD_OK;
  }
  if (rc) return rc;
  return filter_list(c, gate);
}

int export_pairs(gbmd_context* c, int64_t cap, uint64_t* id_i, uint64_t* id_j, int8_t* img, int64_t* count) {
  if (!c->list_valid) {
    int rc = rebuild(c, true);
    if (rc) return rc;
  }
  const int64_t n = c->n;
  std::vector<int32_t> nnb(n), cp(n);
  std::vector<uint64_t> ids(n);
  GBMD_CUDA(c, cudaMemcpyAsync(nnb.data(), c->nnb, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, c->stream));
  GBMD_CUDA(c, cudaMemcpyAsync(cp.data(), c->cellpack, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, c->stream));
  GBMD_CUDA(c, cudaMemcpyAsync(ids.data(), c->ID(), sizeof(uint64_t) * n, cudaMemcpyDeviceToHost, c->stream));
  GBMD_CUDA(c, cudaStreamSynchronize(c->stream));
  int64_t total = 0;
  for (int64_t i = 0; i < n; ++i) total += nnb[i];
  *count = total;
  if (cap < total || !id_i) return GBMD_OK;
  const int W = list_width(c);
  const int wsh = log2_of(W), tsh = log2_of(c->tpa);
  const int64_t stride = c->npad * W;
  std::vector<uint32_t> nb((size_t)c->nbr_cap);
  GBMD_CUDA(c, cudaMemcpy(nb.data(), c->nbr, sizeof(uint32_t) * c->nbr_cap, cudaMemcpyDeviceToHost));
  int64_t row = 0;
  const Grid& g = c->grid;
  for (int64_t i = 0; i < n; ++i) {
    const int cx = cp[i] & 1023, cy = (cp[i] >> 10) & 1023, cz = cp[i] >> 20;
    for (int k = 0; k < nnb[i] && k < c->maxnb; ++k) {
      const uint32_t e = nb[(size_t)(k / W) * stride + (size_t)i * W + list_word(k % W, wsh, tsh)];
      const uint32_t j = e & GBMD_IDX_MASK, code = e >> GBMD_IDX_BITS;
      const int d[3] = {code_dx(code), code_dy(code), code_dz(code)};
      const int cc[3] = {cx + d[0], cy + d[1], cz + d[2]};
      id_i[row] = ids[i];
      id_j[row] = ids[j];
      for (int q = 0; q < 3; ++q) img[3 * row + q] = (int8_t)(cc[q] < 0 ? -1 : (cc[q] >= g.nc[q] ? 1 : 0));
      ++row;
    }
  }
  return GBMD_OK;
}

}  // namespace gbmd
