// Device cell-list / neighbour build: the B200 replacement of Topology::updateCellLists
// (topology/Topology.h:44-81) and CellListEnumerator<PBC, CubicCellManager>
// (topology/CellListEnumeratorPeriodicBoundaries.h:25-134).
//
// Instead of linked cell lists walked pair-of-cells by pair-of-cells, atoms are binned on a fine
// Hilbert-ordered grid with a deterministic counting sort, packed into 8-atom blocks of slots,
// and each block I gets a compacted list of atoms of blocks J > I that lie within the list
// cutoff of I's bounding box.  The pair kernel then sees (I, 32 j-atoms) tiles; the pair set it
// evaluates is exactly the reference's: every unordered pair once, minimal image, r^2 <= rc^2.
#include <algorithm>

#include "pmb_internal.h"
#include "pmb_update.cuh"

namespace pmb {

namespace {

// Index of cell (x, y, z) along a 3-D Hilbert curve over a 2^bits grid (J. Skilling, "Programming
// the Hilbert curve", AIP Conf. Proc. 707, 381 (2004): axes -> transposed index, then bit
// interleave).  Consecutive cells are face neighbours, so a run of slots never jumps across the
// box the way a Morton order does at its octant boundaries.
__device__ __forceinline__ unsigned hilbert3(unsigned x, unsigned y, unsigned z, int bits) {
  if (bits <= 0) return 0u;
  unsigned X[3] = {x, y, z};
  const unsigned M = 1u << (bits - 1);
  for (unsigned Q = M; Q > 1; Q >>= 1) {
    const unsigned P = Q - 1;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      if (X[i] & Q) {
        X[0] ^= P;
      } else {
        unsigned t = (X[0] ^ X[i]) & P;
        X[0] ^= t;
        X[i] ^= t;
      }
    }
  }
  X[1] ^= X[0];
  X[2] ^= X[1];
  unsigned t = 0;
  for (unsigned Q = M; Q > 1; Q >>= 1)
    if (X[2] & Q) t ^= Q - 1;
  X[0] ^= t;
  X[1] ^= t;
  X[2] ^= t;
  unsigned h = 0;
  for (int b = bits - 1; b >= 0; b--)
#pragma unroll
    for (int i = 0; i < 3; i++) h = (h << 1) | ((X[i] >> b) & 1u);
  return h;
}

// ---------------------------------------------------------------- scans
__device__ int block_exclusive_scan(int v, int *total) {
  __shared__ int warp_tot[32];
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[w] = x;
  __syncthreads();
  if (w == 0) {
    int nw = blockDim.x >> 5;
    int t = lane < nw ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nw) warp_tot[lane] = t;
  }
  __syncthreads();
  int off = w > 0 ? warp_tot[w - 1] : 0;
  if (total) *total = warp_tot[(blockDim.x >> 5) - 1];
  __syncthreads();
  return off + x - v;
}

// ---------------------------------------------------------------- binning and sort
__global__ void __launch_bounds__(UPDATE_THREADS) k_update(SystemDev s, NbListDev nb) {
  const int i = blockIdx.x * UPDATE_THREADS + threadIdx.x;
  double x[3] = {0.0, 0.0, 0.0};
  if (i < s.natoms)
#pragma unroll
    for (int c = 0; c < 3; c++) x[c] = s.pos[3 * i + c];
  update_atom(s, nb, i, x, nullptr);
}

// ---- the sort into slots, a deterministic counting sort: histogram of the atoms over the
// Hilbert-ordered cells, exclusive scan, scatter, placing (an atom's slot is its bin's start plus
// the number of smaller atom indices in the bin) with the slot records, then the extents of the
// 8-slot blocks and of the runs of 32 blocks (superblocks, per box).  Each phase is a loop of
// thread t of T over one box; bins and slots are counted from the box's first.  Loads of what
// other threads of the same launch may have written go past L1.
__device__ __forceinline__ void sort_bin(const SystemDev &s, const NbListDev &nb, const BoxDev &b, int t, int T) {
  const int nc = b.nc[0], bits = __ffs(nc) - 1;
  for (int p = t; p < b.natoms; p += T) {
    const int i = b.atom0 + p;
    unsigned c[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const unsigned f = frac_fixed(s.pos[3 * i + k], b.Lr[k]);
      c[k] = (unsigned)(((unsigned long long)f * (unsigned)nc) >> 32);
    }
    const int kk = (int)hilbert3(c[0], c[1], c[2], bits);
    nb.key[i] = kk;
    nb.rank[i] = atomicAdd(nb.bin_count + b.key0 + kk, 1);  // (the bins are zero between builds)
  }
}
constexpr int SCAN_PER = 16;  // bins of a thread per round of the scan
// The bins k .. k + SCAN_PER of a thread: counts in v, their sum returned.  (nk is 1 or a multiple of 8; the
// boxes' regions start at multiples of 4.)
__device__ __forceinline__ int scan_load(const int *count, int k, int nk, int4 v[SCAN_PER / 4]) {
  int sum = 0;
#pragma unroll
  for (int q = 0; q < SCAN_PER / 4; q++) {
    v[q] = make_int4(0, 0, 0, 0);
    if (k + 4 * q < nk) v[q] = __ldcg(reinterpret_cast<const int4 *>(count + k + 4 * q));
    sum += v[q].x + v[q].y + v[q].z + v[q].w;
  }
  return sum;
}
// Their starts, ex the first.
__device__ __forceinline__ void scan_store(int *start, int k, int nk, int ex, const int4 v[SCAN_PER / 4]) {
#pragma unroll
  for (int q = 0; q < SCAN_PER / 4; q++) {
    if (k + 4 * q < nk)
      *reinterpret_cast<int4 *>(start + k + 4 * q) =
          make_int4(ex, ex + v[q].x, ex + v[q].x + v[q].y, ex + v[q].x + v[q].y + v[q].z);
    ex += v[q].x + v[q].y + v[q].z + v[q].w;
  }
}
// The counts of a CTA's round, k0 the first, cleared once all its threads have read theirs: the bins are
// zero for the next build whichever kernels follow the scan.
__device__ __forceinline__ void scan_clear(int *count, int k0, int nk) {
#pragma unroll
  for (int q = 0; q < SCAN_PER / 4; q++) {
    const int k = k0 + 4 * (q * blockDim.x + threadIdx.x);
    if (k < nk) *reinterpret_cast<int4 *>(count + k) = make_int4(0, 0, 0, 0);
  }
}
// by one CTA
__device__ __forceinline__ void sort_scan(const NbListDev &nb, const BoxDev &b) {
  const int nk = b.nc[0] * b.nc[0] * b.nc[0], T = blockDim.x;
  int *count = nb.bin_count + b.key0, *start = nb.bin_start + b.key0;
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int k0 = 0; k0 < nk; k0 += SCAN_PER * T) {
    const int k = k0 + SCAN_PER * threadIdx.x;
    int4 v[SCAN_PER / 4];
    const int sum = scan_load(count, k, nk, v);
    int tot;
    const int ex = carry + block_exclusive_scan(sum, &tot);
    scan_store(start, k, nk, ex, v);
    scan_clear(count, k0, nk);  // (the block scan holds barriers)
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
}
__device__ __forceinline__ void sort_scatter(const NbListDev &nb, const BoxDev &b, int t, int T) {
  const int *start = nb.bin_start + b.key0;
  int *raw = nb.slot_raw + b.blk0 * BLOCK;
  for (int p = t; p < b.natoms; p += T) {
    const int i = b.atom0 + p;
    raw[__ldcg(start + nb.key[i]) + nb.rank[i]] = i;
  }
}
__device__ __forceinline__ void sort_place(const SystemDev &s, const NbListDev &nb, const BoxDev &b, int bi, int t, int T) {
  const int *start = nb.bin_start + b.key0;
  const int *raw = nb.slot_raw + b.blk0 * BLOCK;
  const int nk = b.nc[0] * b.nc[0] * b.nc[0];
  for (int p = t; p < b.nblk * BLOCK; p += T) {
    if (p >= b.natoms) {  // padding of the last block
      const int sl = b.blk0 * BLOCK + p;
      nb.slot_orig[sl] = -1;
      nb.slot_meta[sl] = make_int4(-1, -1, 0, bi);
      nb.slot_fx[sl] = make_uint4(0, 0, 0, 0);
      if (nb.want_fp64) nb.slot_pq[sl] = make_double4(0, 0, 0, 0);
      continue;
    }
    const int i = __ldcg(raw + p);
    const int k = __ldcg(nb.key + i);
    const double x = s.pos[3 * i], y = s.pos[3 * i + 1], z = s.pos[3 * i + 2], q = s.charge[i];
    const int mol = s.molecule[i], type = s.type[i];
    const int s0 = __ldcg(start + k), s1 = k + 1 < nk ? __ldcg(start + k + 1) : b.natoms;
    int below = 0;
    for (int r = s0; r < s1; r++) below += __ldcg(raw + r) < i;
    const int sl = b.blk0 * BLOCK + s0 + below;
    nb.slot_of[i] = sl;
    nb.slot_orig[sl] = i;
    nb.slot_meta[sl] = make_int4(i, mol, type, bi);
    nb.slot_fx[sl] = make_uint4(frac_fixed(x, b.Lr[0]), frac_fixed(y, b.Lr[1]), frac_fixed(z, b.Lr[2]),
                                __float_as_uint((float)q));
    if (nb.want_fp64) nb.slot_pq[sl] = make_double4(x, y, z, q);
    nb.xref[3 * i] = x;  // the box's new reference positions
    nb.xref[3 * i + 1] = y;
    nb.xref[3 * i + 2] = z;
  }
}
// extents in fractional fixed point, a warp per superblock and GROUPS blocks at a time
__device__ __forceinline__ void sort_extents(const NbListDev &nb, const BoxDev &b, int t, int T) {
  const int lane = threadIdx.x & 31, li = lane & (BLOCK - 1), g = lane / BLOCK;
  for (int S = t >> 5; S * 32 < b.nblk; S += T / 32) {
    unsigned slo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, shi[3] = {0u, 0u, 0u};
    int scnt = 0;
#pragma unroll 2
    for (int j0 = S * 32; j0 < min(b.nblk, S * 32 + 32); j0 += GROUPS) {
      const int j = j0 + g;
      const bool inr = j < b.nblk;
      const int blk = b.blk0 + j;
      const bool valid = inr && j * BLOCK + li < b.natoms;
      uint4 f = make_uint4(0, 0, 0, 0);
      if (valid) f = __ldcg(nb.slot_fx + (long long)blk * BLOCK + li);
      unsigned lo[3] = {valid ? f.x : 0xffffffffu, valid ? f.y : 0xffffffffu, valid ? f.z : 0xffffffffu};
      unsigned hi[3] = {f.x, f.y, f.z};
#pragma unroll
      for (int o = BLOCK / 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; k++) {
          lo[k] = min(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
          hi[k] = max(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
      const unsigned bal = __ballot_sync(0xffffffffu, valid);
      const int cnt = __popc(bal & (((1u << BLOCK) - 1u) << (lane & ~(BLOCK - 1))));
      if (inr && li == 0) {  // (a box's blocks all hold at least one atom)
        nb.blk_lo[blk] = make_uint4(lo[0], lo[1], lo[2], (unsigned)cnt);
        nb.blk_hi[blk] = make_uint4(hi[0], hi[1], hi[2], 0u);
        nb.blk_c[blk] = make_uint4(lo[0] + (hi[0] - lo[0]) / 2u, lo[1] + (hi[1] - lo[1]) / 2u,
                                   lo[2] + (hi[2] - lo[2]) / 2u, (unsigned)cnt);
        nb.blk_h[blk] = make_uint4((hi[0] - lo[0]) / 2u + 1u, (hi[1] - lo[1]) / 2u + 1u, (hi[2] - lo[2]) / 2u + 1u, 0u);
      }
      if (inr) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
          slo[k] = min(slo[k], lo[k]);
          shi[k] = max(shi[k], hi[k]);
        }
        scnt += cnt;
      }
    }
#pragma unroll
    for (int o = 16; o >= BLOCK; o >>= 1) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        slo[k] = min(slo[k], __shfl_xor_sync(0xffffffffu, slo[k], o));
        shi[k] = max(shi[k], __shfl_xor_sync(0xffffffffu, shi[k], o));
      }
      scnt += __shfl_xor_sync(0xffffffffu, scnt, o);
    }
    if (lane == 0) {
      nb.sblk_c[b.sblk0 + S] = make_uint4(slo[0] + (shi[0] - slo[0]) / 2u, slo[1] + (shi[1] - slo[1]) / 2u,
                                          slo[2] + (shi[2] - slo[2]) / 2u, (unsigned)scnt);
      nb.sblk_h[b.sblk0 + S] = make_uint4((shi[0] - slo[0]) / 2u + 1u, (shi[1] - slo[1]) / 2u + 1u,
                                          (shi[2] - slo[2]) / 2u + 1u, 0u);
    }
  }
}

// Every phase in one launch, a CTA per box: small boxes, and systems of many.  About a thread an atom of
// the largest box (sort_box_threads): with 1024 threads for 24 atoms two boxes an SM wait at barriers (5,000
// boxes of 24 atoms, an evaluation that rebuilds 271 us, now 115, without a rebuild 84 and 76; 20,000
// boxes 1032 and 327; 300 boxes of 648 atoms as before).
constexpr int SORT_THREADS = 512, SORT_BOX_THREADS = 1024;
int sort_box_threads(const NbListDev &nb) {
  int t = 64;
  while (t < SORT_BOX_THREADS && t < nb.max_box_atoms) t *= 2;
  return t;
}
__global__ void __launch_bounds__(SORT_BOX_THREADS) k_sort_box(SystemDev s, NbListDev nb) {
  if (!nb.ctl[CTL_REBUILD]) return;
  const int bi = blockIdx.x, t = threadIdx.x, T = blockDim.x;
  if (!nb.box_rb[bi]) return;  // the box keeps its slots
  const BoxDev &b = s.box[bi];
  sort_bin(s, nb, b, t, T);
  __syncthreads();
  sort_scan(nb, b);
  __syncthreads();
  sort_scatter(nb, b, t, T);
  __syncthreads();
  sort_place(s, nb, b, bi, t, T);
  __syncthreads();
  sort_extents(nb, b, t, T);
}

// One launch per phase over the whole chip: large boxes.  A CTA takes one item of nb.sort_work,
// SORT_PART slots of one box, so the launches follow the atoms however uneven the boxes are.  The last
// CTA of a box to finish its histogram also scans the box's bins, if they are few.
static_assert(SORT_THREADS == SORT_PART, "a thread takes a slot");
constexpr int EXT_THREADS = SORT_PART / 8;  // a warp takes a superblock, 32 blocks of 8 slots
static_assert(BLOCK == 8, "256 slots a superblock");
__device__ __forceinline__ int2 sort_item(const NbListDev &nb) {  // box, part (of one box: no table to wait for)
  return nb.nbox == 1 ? make_int2(0, blockIdx.x) : nb.sort_work[blockIdx.x];
}
__global__ void __launch_bounds__(SORT_THREADS) k_sort_bin(SystemDev s, NbListDev nb) {
  const int2 it = sort_item(nb);
  if (!nb.ctl[CTL_REBUILD] || !nb.box_rb[it.x]) return;
  const BoxDev &b = s.box[it.x];
  const int parts = (b.nblk * BLOCK + SORT_PART - 1) / SORT_PART;
  sort_bin(s, nb, b, it.y * SORT_PART + threadIdx.x, parts * SORT_PART);
  __threadfence();
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(nb.box_done + it.x, 1u) == (unsigned)parts - 1u;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x == 0) nb.box_done[it.x] = 0u;
  if (b.nc[0] * b.nc[0] * b.nc[0] <= SCAN_ONE_CTA) sort_scan(nb, b);
}
// The bins of a wide box, SCAN_CHUNK to a CTA and turn: the chunks' sums, then each chunk from the sum
// of those before it.  (The number of bins follows the longest edge, not the atoms: 32,768 up to 154 A,
// 2.1 million at 307 to 614 A.)  An evaluation that rebuilds, by one CTA's scan and by these: 217,000 atoms
// in 60 x 60 x 600 A 1224 and 619 us, 30,000 atoms within 1000 A 5027 and 208 us, 216 atoms within 700 A
// 5240 and 132 us; the 97,000 atoms of a 99 A cube (32,768 bins, scanned by one CTA) take 271 us.
static_assert(SCAN_CHUNK == SORT_THREADS * SCAN_PER, "a thread scans SCAN_PER bins of a chunk");
__global__ void __launch_bounds__(SORT_THREADS) k_scan_sums(SystemDev s, NbListDev nb) {
  if (!nb.ctl[CTL_REBUILD]) return;
  for (int w = blockIdx.x; w < nb.nscan; w += gridDim.x) {
    const int2 it = nb.scan_work[w];  // box, chunk
    if (!nb.box_rb[it.x]) continue;
    const BoxDev &b = s.box[it.x];
    const int nk = b.nc[0] * b.nc[0] * b.nc[0], k = it.y * SCAN_CHUNK + SCAN_PER * threadIdx.x;
    int4 v[SCAN_PER / 4];
    int tot;
    block_exclusive_scan(scan_load(nb.bin_count + b.key0, k, nk, v), &tot);
    if (threadIdx.x == 0) nb.bin_sums[w] = tot;
  }
}
__global__ void __launch_bounds__(SORT_THREADS) k_scan_apply(SystemDev s, NbListDev nb) {
  if (!nb.ctl[CTL_REBUILD]) return;
  for (int w = blockIdx.x; w < nb.nscan; w += gridDim.x) {
    const int2 it = nb.scan_work[w];
    if (!nb.box_rb[it.x]) continue;
    const BoxDev &b = s.box[it.x];
    const int nk = b.nc[0] * b.nc[0] * b.nc[0], k = it.y * SCAN_CHUNK + SCAN_PER * threadIdx.x;
    int before = 0, base;
    for (int c = w - it.y + threadIdx.x; c < w; c += SORT_THREADS) before += __ldg(nb.bin_sums + c);
    block_exclusive_scan(before, &base);
    int4 v[SCAN_PER / 4];
    const int sum = scan_load(nb.bin_count + b.key0, k, nk, v);
    const int ex = base + block_exclusive_scan(sum, nullptr);
    scan_store(nb.bin_start + b.key0, k, nk, ex, v);
    scan_clear(nb.bin_count + b.key0, it.y * SCAN_CHUNK, nk);
  }
}
__global__ void __launch_bounds__(SORT_THREADS) k_sort_scatter(SystemDev s, NbListDev nb) {
  const int2 it = sort_item(nb);
  if (!nb.ctl[CTL_REBUILD] || !nb.box_rb[it.x]) return;
  const BoxDev &b = s.box[it.x];
  sort_scatter(nb, b, it.y * SORT_PART + threadIdx.x, b.nblk * BLOCK + SORT_PART);
}
__global__ void __launch_bounds__(SORT_THREADS) k_sort_place(SystemDev s, NbListDev nb) {
  const int2 it = sort_item(nb);
  if (!nb.ctl[CTL_REBUILD] || !nb.box_rb[it.x]) return;
  const BoxDev &b = s.box[it.x];
  sort_place(s, nb, b, it.x, it.y * SORT_PART + threadIdx.x, b.nblk * BLOCK + SORT_PART);
}
__global__ void __launch_bounds__(EXT_THREADS) k_sort_extents(SystemDev s, NbListDev nb) {
  const int2 it = sort_item(nb);
  if (!nb.ctl[CTL_REBUILD] || !nb.box_rb[it.x]) return;
  const BoxDev &b = s.box[it.x];
  sort_extents(nb, b, it.y * EXT_THREADS + threadIdx.x, b.nblk + EXT_THREADS);
}

// Gap^2 (A^2) between the box (c1, h1 half extents in A) and the box (c2, h2 fixed-point half
// extents) in FP32: the fixed-point difference (minimal image by 32-bit wrap-around) converts
// with an error of < 1e-5 A, far below the 1e-3 A margin of the list radius over the cutoff.
__device__ __forceinline__ float gap2f(const float sL[3], const unsigned c1[3], const float h1[3],
                                       uint4 c2, uint4 h2) {
  const unsigned c[3] = {c2.x, c2.y, c2.z}, h[3] = {h2.x, h2.y, h2.z};
  float g2 = 0.f;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const float d = fmaxf((fabsf((float)(int)(c[k] - c1[k])) - (float)h[k]) * sL[k] - h1[k], 0.f);
    g2 = fmaf(d, d, g2);
  }
  return g2;
}

#ifndef BL_BLOCK_THREADS
#define BL_BLOCK_THREADS 256
#endif
#ifndef BL_MINB
#define BL_MINB 4
#endif
constexpr int BL_THREADS = BL_BLOCK_THREADS;
constexpr int BL_CAP = 128;  // candidate blocks buffered per warp before their atoms are tested
constexpr float PAD_NORM = 1e12f;  // |q|^2 of a block's padding atoms

// One warp per block I: its own slots, then the candidate blocks J > I of the same box by
// bounding-box gap (superblocks of 32 blocks first), compacted into a shared-memory list, then
// the atoms of GROUPS listed blocks per pass within the list cutoff of I's box, compacted into
// I's j-list (tiles of 32 entries).  The loads of the next pass are issued before the current
// pass is tested.
// One block's list; cl [BL_CAP] and ipos [BLOCK] are the warp's shared memory.  Returns its tiles.
__device__ __forceinline__ int build_block(const SystemDev &s, NbListDev &nb, double rlist2, int I, const BoxDev &b, int *cl,
                                           float4 *ipos) {
  const int lane = threadIdx.x & 31;
  const uint4 cIv = nb.blk_c[I], hIv = nb.blk_h[I];
  const float sL[3] = {(float)(b.L[0] * (1.0 / 4294967296.0)), (float)(b.L[1] * (1.0 / 4294967296.0)),
                       (float)(b.L[2] * (1.0 / 4294967296.0))};
  const unsigned cI[3] = {cIv.x, cIv.y, cIv.z};
  const float hI[3] = {(float)hIv.x * sL[0], (float)hIv.y * sL[1], (float)hIv.z * sL[2]};
  const int jend = b.blk0 + b.nblk;
  const int cap = nb.jcap_off[I + 1] - nb.jcap_off[I];
  int *out = nb.jlist + nb.jcap_off[I];
  const bool multi = b.multi_image != 0;
  const float rl2 = (float)rlist2;
  const int g = lane / BLOCK, li = lane & (BLOCK - 1);
  // molecules of the cluster's atoms (-2: padding): a listed j-atom of one of them is flagged
  // JSAME, so the pair kernel runs the exclusion test only on tiles holding such an atom; the
  // block's own slots open its list (the pair kernel takes j > i among them)
  // and the block's atom positions q: a candidate atom p is listed when it is within the list
  // radius of one of them, the exact Verlet condition per pair (the bounding-box gap alone would
  // list about a third more atoms).  In shared memory, FP32 relative to the block's first atom, as
  // -2 q and |q|^2 of pairs of atoms {t, t + BLOCK/2}: x x' y y' | z z' n n', so that a pair of
  // atoms takes three two-wide products, |p - q|^2 <= r^2 as |q|^2 - 2 p.q <= r^2 - |p|^2 (rounding:
  // see `diff` below); padding atoms have |q|^2 = 1e12.
  int imol[BLOCK];
  unsigned r0[3];
  {
    const int4 m = nb.slot_meta[I * BLOCK + li];
    const uint4 f = nb.slot_fx[I * BLOCK + li];
    if (lane < BLOCK) out[lane] = m.x >= 0 ? ((I * BLOCK + lane) | JSAME) : -1;
    const int mine = m.x >= 0 ? m.y : -2;
#pragma unroll
    for (int t = 0; t < BLOCK; t++) imol[t] = __shfl_sync(0xffffffffu, mine, t);
    r0[0] = __shfl_sync(0xffffffffu, f.x, 0);
    r0[1] = __shfl_sync(0xffffffffu, f.y, 0);
    r0[2] = __shfl_sync(0xffffffffu, f.z, 0);
    float px = 0.f, py = 0.f, pz = 0.f, pn = PAD_NORM;
    if (m.x >= 0) {
      px = (float)(int)(f.x - r0[0]) * sL[0];
      py = (float)(int)(f.y - r0[1]) * sL[1];
      pz = (float)(int)(f.z - r0[2]) * sL[2];
      pn = fmaf(pz, pz, fmaf(py, py, px * px));
    }
    const float qx = __shfl_down_sync(0xffffffffu, px, BLOCK / 2), qy = __shfl_down_sync(0xffffffffu, py, BLOCK / 2),
                qz = __shfl_down_sync(0xffffffffu, pz, BLOCK / 2), qn = __shfl_down_sync(0xffffffffu, pn, BLOCK / 2);
    __syncwarp();  // (the previous block's reads)
    if (lane < BLOCK / 2) {
      ipos[2 * lane] = make_float4(-2.f * px, -2.f * qx, -2.f * py, -2.f * qy);
      ipos[2 * lane + 1] = make_float4(-2.f * pz, -2.f * qz, pn, qn);
    }
    __syncwarp();
  }
  // offsets from the first atom are minimal images of candidate-atom differences unless the box
  // is under about twice the list radius plus the block's extent: then each difference is
  // wrapped again
  const float rlf = sqrtf(rl2);
  const bool rewrap = rlf + 2.f * hI[0] >= 0.5f * (float)b.L[0] || rlf + 2.f * hI[1] >= 0.5f * (float)b.L[1] ||
                      rlf + 2.f * hI[2] >= 0.5f * (float)b.L[2];
  // The expanded test cancels |p|^2 and |q|^2.  With |q| <= X, the block's extent, and |p| <= P = X + r
  // its ten roundings, u = 2^-24 each, add up to at most u (3 X^2 + 3 (X^2 + 2 X P) + 4 P^2) <= 16 u P^2
  // = 9.5e-7 P^2 A^2.  The list radius r exceeds what is needed by 1e-3 A, 2e-3 r A^2: half of that is
  // left to the coordinates' own rounding.  A block spread wider (P > 104 A at r = 10.8; blocks of a
  // liquid have P < 20) takes the differences themselves, as the re-wrapped test does.
  const float P = rlf + 2.f * sqrtf(fmaf(hI[2], hI[2], fmaf(hI[1], hI[1], hI[0] * hI[0])));
  const bool diff = rewrap || 1e-6f * P * P > 1e-3f * rlf;
  const float Lf[3] = {(float)b.L[0], (float)b.L[1], (float)b.L[2]},
              Lrf[3] = {(float)b.Lr[0], (float)b.Lr[1], (float)b.Lr[2]};
  auto near_any = [&](uint4 f) {
    const float px = (float)(int)(f.x - r0[0]) * sL[0], py = (float)(int)(f.y - r0[1]) * sL[1],
                pz = (float)(int)(f.z - r0[2]) * sL[2];
    bool near = false;
    if (diff) {
#pragma unroll
      for (int t = 0; t < BLOCK / 2; t++) {
        const float4 a = ipos[2 * t], c = ipos[2 * t + 1];
        const float qx[2] = {a.x, a.y}, qy[2] = {a.z, a.w}, qz[2] = {c.x, c.y}, qn[2] = {c.z, c.w};
#pragma unroll
        for (int u = 0; u < 2; u++) {
          float dx = fmaf(0.5f, qx[u], px), dy = fmaf(0.5f, qy[u], py), dz = fmaf(0.5f, qz[u], pz);
          dx -= Lf[0] * rintf(dx * Lrf[0]);
          dy -= Lf[1] * rintf(dy * Lrf[1]);
          dz -= Lf[2] * rintf(dz * Lrf[2]);
          near |= (fmaf(dz, dz, fmaf(dy, dy, dx * dx)) <= rl2) & (qn[u] < PAD_NORM);
        }
      }
      return near;
    }
    const float2 px2 = make_float2(px, px), py2 = make_float2(py, py), pz2 = make_float2(pz, pz);
    const float lim = rl2 - fmaf(pz, pz, fmaf(py, py, px * px));
#pragma unroll
    for (int t = 0; t < BLOCK / 2; t++) {
      const float4 a = ipos[2 * t], c = ipos[2 * t + 1];
      const float2 d = __ffma2_rn(
          make_float2(c.x, c.y), pz2,
          __ffma2_rn(make_float2(a.z, a.w), py2, __ffma2_rn(make_float2(a.x, a.y), px2, make_float2(c.z, c.w))));
      near |= (d.x <= lim) | (d.y <= lim);
    }
    return near;
  };
  int count = BLOCK, ncand = 0;
  bool overflow = false;

  // atoms of the listed candidate blocks, GROUPS blocks (32 slots) per pass
  auto atoms = [&]() {
    __syncwarp();
    // (slots past the box's last atom are padding)
    const int slot_end = b.blk0 * BLOCK + b.natoms;
    auto fetch = [&](int q, int &sl, uint4 &f, int &mol) {
      sl = q < ncand ? cl[q] * BLOCK + li : -1;
      if (sl >= slot_end) sl = -1;
      f = make_uint4(0, 0, 0, 0);
      mol = -1;
      if (sl >= 0) {
        f = nb.slot_fx[sl];
        mol = nb.slot_meta[sl].y;
      }
    };
    int sl, mol;
    uint4 f;
    fetch(g, sl, f, mol);
    for (int p = 0; p < ncand; p += GROUPS) {
      int sl2, mol2;
      uint4 f2;
      fetch(p + GROUPS + g, sl2, f2, mol2);
      const bool take = sl >= 0 && (multi || near_any(f));
      const unsigned tm = __ballot_sync(0xffffffffu, take);
      const int n = __popc(tm);
      if (count + n > cap) {
        overflow = true;
        break;
      }
      if (take) {
        bool same = false;
#pragma unroll
        for (int t = 0; t < BLOCK; t++) same |= mol == imol[t];
        out[count + __popc(tm & ((1u << lane) - 1u))] = same ? (sl | JSAME) : sl;
      }
      count += n;
      sl = sl2;
      mol = mol2;
      f = f2;
    }
    ncand = 0;
    __syncwarp();
  };

  // superblocks (the box's runs of 32 blocks), 32 per ballot; then the 32 blocks of each candidate
  const int send = (b.nblk + 31) / 32;
  for (int S0 = (I + 1 - b.blk0) / 32; S0 < send && !overflow; S0 += 32) {
    const int S = S0 + lane;
    bool scand = false;
    if (S < send) {
      const uint4 cS = nb.sblk_c[b.sblk0 + S];
      if (cS.w > 0) scand = multi || gap2f(sL, cI, hI, cS, nb.sblk_h[b.sblk0 + S]) <= rl2;
    }
    unsigned sm = __ballot_sync(0xffffffffu, scand);
    while (sm && !overflow) {
      const int J = b.blk0 + (S0 + __ffs(sm) - 1) * 32 + lane;
      sm &= sm - 1;
      bool cand = false;
      if (J > I && J < jend) {
        const uint4 cJ = nb.blk_c[J];
        if (cJ.w > 0) cand = multi || gap2f(sL, cI, hI, cJ, nb.blk_h[J]) <= rl2;
      }
      const unsigned m = __ballot_sync(0xffffffffu, cand);
      if (ncand + __popc(m) > BL_CAP) atoms();
      if (cand) cl[ncand + __popc(m & ((1u << lane) - 1u))] = J;
      ncand += __popc(m);
    }
  }
  if (!overflow && ncand > 0) atoms();
  const int padded = (count + 31) & ~31;
  if (!overflow)
    for (int k = count + lane; k < padded; k += 32) out[k] = -1;
  const int tiles = overflow ? 0 : padded / 32;
  if (lane == 0) {
    if (overflow) atomicExch(&nb.status[0], 1);
    nb.jcount[I] = tiles;
  }
  return tiles;
}

// Warps claim nb.claim_blocks consecutive blocks from a counter, in ascending order (the early
// blocks' lists are the longest).  Their lists then join the pair kernel's work as units of at most
// nb.unit_tiles tiles (about equal parts of a list, starting at multiples of CLOSE_TILES tiles); a
// block of a box that keeps its list appends the units it has.  The units of boxes that need lattice
// images grow from the end of the array.  Their order varies from build to build and changes no
// result: the pair kernel closes its floating-point sums every CLOSE_TILES tiles of a list.
// One claim and one append per several blocks in a large system: with three atomics per block the
// counters' words were the bound of an ensemble's build (810,000 atoms, a quarter of the boxes
// rebuilt: 590 us a step); one block per claim where there are few per warp, and no barrier between
// warps (8 blocks to a CTA's claim: 13% of the warps' time).
__global__ void __launch_bounds__(BL_THREADS, BL_MINB) k_build_lists(SystemDev s, NbListDev nb, double rlist2) {
  __shared__ int cand_all[BL_THREADS / 32][BL_CAP];
  __shared__ float4 ipos_all[BL_THREADS / 32][BLOCK];
  if (!nb.ctl[CTL_REBUILD]) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = nb.claim_blocks, per = nb.unit_tiles / CLOSE_TILES;
  for (;;) {
    int I0 = 0;
    if (lane == 0) I0 = (int)atomicAdd(nb.ctl + CTL_CLAIM, 1u) * G;
    I0 = __shfl_sync(0xffffffffu, I0, 0);
    if (I0 >= nb.nblk_total) return;
    const int n = min(G, nb.nblk_total - I0);
    int tiles = 0, multi = 0;  // lane q: block I0 + q
    for (int q = 0; q < n; q++) {
      const int I = I0 + q, bi = nb.blk_box[I];
      const BoxDev &b = s.box[bi];
      const int t = nb.box_rb[bi] ? build_block(s, nb, rlist2, I, b, cand_all[w], ipos_all[w]) : nb.jcount[I];
      if (lane == q) {
        tiles = t;
        multi = b.multi_image != 0;
      }
    }
    const int nc = (tiles + CLOSE_TILES - 1) / CLOSE_TILES, nu = (nc + per - 1) / per;
    int at = 0;
    const unsigned all = __ballot_sync(0xffffffffu, nu > 0), images = __ballot_sync(0xffffffffu, multi != 0);
    for (int kind = 0; kind < 2; kind++) {  // units without and with lattice images
      if (!(all & (kind ? images : ~images))) continue;
      const int mine = multi == kind ? nu : 0;
      int sum = mine;  // inclusive sum over the lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += y;
      }
      int base = 0;
      if (lane == 31) base = (int)atomicAdd(nb.ctl + CTL_UNITS + kind, (unsigned)sum);
      base = __shfl_sync(0xffffffffu, base, 31);
      if (multi == kind) at = base + sum - mine;
    }
    for (int q = 0; q < n; q++) {
      const int nuq = __shfl_sync(0xffffffffu, nu, q), ncq = __shfl_sync(0xffffffffu, nc, q),
                tq = __shfl_sync(0xffffffffu, tiles, q), atq = __shfl_sync(0xffffffffu, at, q);
      const bool mq = (images >> q) & 1u;
      for (int p = lane; p < nuq; p += 32) {
        const int k0 = (int)((long long)ncq * p / nuq) * CLOSE_TILES;
        const int k1 = min(tq, (int)((long long)ncq * (p + 1) / nuq) * CLOSE_TILES);
        const int u = atq + p;  // (within the array: it is sized for full lists)
        nb.units[mq ? nb.unit_cap - 1 - u : u] = make_int4(I0 + q, k0, k1 - k0, nb.jcap_off[I0 + q] + k0 * JCHUNK);
      }
    }
  }
}
constexpr int CLAIMS_PER_WARP = 4;  // at least, before a claim takes more than one block

// One CTA per box up to SORT_SMALL atoms, and up to SORT_MANY when the boxes alone fill the chip and the
// largest is not the one that all wait for; not where a box has more bins than one CTA scans.  An
// evaluation that rebuilds every box, by one CTA per box and by a launch per phase: 80 boxes of 6,000
// atoms 934 and 945 us, of 12,000 1641 and 1639, of 24,000 3365 and 3340; 80 of 600 beside one of 24,000
// 347 and 222.
constexpr int SORT_SMALL = 3072, SORT_MANY = 8192;
bool sort_by_box(const SystemDev &s, const NbListDev &nb) {
  if (nb.nscan > 0) return false;
  if (nb.max_box_atoms <= SORT_SMALL) return true;
  return s.nbox >= nb.n_sm / 2 && nb.max_box_atoms <= SORT_MANY &&
         (long long)nb.max_box_atoms * s.nbox <= 3ll * s.natoms;
}

}  // namespace

// First half of a build: displacement check and this step's slot records (unless the kernel that
// moved the atoms made them), then the sort into
// slots of the boxes that rebuild (the PME kernels need no more than these).  Every kernel after
// the displacement check exits at once unless ctl[CTL_REBUILD] asks for a rebuild.
int nblist_sort(const SystemDev &s, NbListDev &nb, bool updated, cudaStream_t st) {
  const int na = s.natoms;
  if (na <= 0) return 0;
  if (!updated) k_update<<<(na + UPDATE_THREADS - 1) / UPDATE_THREADS, UPDATE_THREADS, 0, st>>>(s, nb);
  if (sort_by_box(s, nb)) {
    k_sort_box<<<s.nbox, sort_box_threads(nb), 0, st>>>(s, nb);
    return 0;
  }
  k_sort_bin<<<nb.nsort, SORT_THREADS, 0, st>>>(s, nb);
  if (nb.nscan > 0) {
    const int scan_grid = std::min(nb.nscan, 4 * nb.n_sm);
    k_scan_sums<<<scan_grid, SORT_THREADS, 0, st>>>(s, nb);
    k_scan_apply<<<scan_grid, SORT_THREADS, 0, st>>>(s, nb);
  }
  k_sort_scatter<<<nb.nsort, SORT_THREADS, 0, st>>>(s, nb);
  k_sort_place<<<nb.nsort, SORT_THREADS, 0, st>>>(s, nb);
  return 0;
}

// Second half: the extents of the blocks (large boxes), the cluster j-lists and the units of the pair kernel.
int nblist_lists(const SystemDev &s, NbListDev &nb, double list_cutoff, cudaStream_t st) {
  if (s.natoms <= 0) return 0;
  if (!sort_by_box(s, nb)) k_sort_extents<<<nb.nsort, EXT_THREADS, 0, st>>>(s, nb);
  // as many blocks as fit at once (blocks are claimed), so that the exit without a rebuild is short
  const int warps = BL_THREADS / 32, need = (nb.nblk_total + warps - 1) / warps;
  nb.claim_blocks = std::max(1, std::min(8, nb.nblk_total / (nb.n_sm * BL_MINB * warps * CLAIMS_PER_WARP)));
  k_build_lists<<<need < nb.n_sm * BL_MINB ? need : nb.n_sm * BL_MINB, BL_THREADS, 0, st>>>(s, nb, list_cutoff * list_cutoff);
  return 0;
}

}  // namespace pmb
