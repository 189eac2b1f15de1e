// Displacement check and slot records of one step, by the kernel that has the new positions in
// registers: the list's own pass over the atoms, or the integrator's drift.
#pragma once
#include "pmb_internal.h"

namespace pmb {

constexpr int UPDATE_THREADS = 256;

__device__ __forceinline__ unsigned frac_fixed(double x, double Lr) {
  double u = x * Lr;
  u -= floor(u);
  double s = u * 4294967296.0;
  if (!(s >= 0.0)) s = 0.0;                 // also catches NaN
  if (s >= 4294967295.0) s = 4294967295.0;
  return (unsigned)s;
}

__device__ __forceinline__ int ford(float f) {  // order-preserving int image of a float
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float fuord(int o) { return __int_as_float(o >= 0 ? o : o ^ 0x7fffffff); }

// Thread i of UPDATE_THREADS-thread blocks over the atoms, every thread of the block: atom i now at
// x.  Rebuild decision, box by box: max |x - x_ref|^2 over each box's atoms (box_d2), then the last
// block sets box_rb[b] for every box that moved more than half the skin and ctl[CTL_REBUILD] when
// any did (no host round trip).
// It sees every position of every evaluation, so it also raises status[2] for a non-finite one
// (the host reports PMB_ERR_NUMERIC; every later kernel maps such a position to an in-range cell
// and grid index, so nothing reads out of bounds meanwhile), and, for a system whose boxes stand
// in for vacuum (ctl[CTL_VACUUM]), status[3] once the atoms of a box spread over half an edge (the
// minimal image would no longer be the plain difference).
// The same pass writes this step's coordinates into the atom's slot record (the slot it got at its
// box's last build; a box that is rebuilt packs its records again afterwards), so a step without a
// rebuild has no pass of its own for that.  The last block also advances *step, if given.
__device__ __forceinline__ void update_atom(const SystemDev &s, NbListDev &nb, int i, const double x[3], long long *step) {
  float d2 = 0.f;
  int box = -1;
  const bool vacuum = nb.ctl[CTL_VACUUM] != 0u;
  if (i < s.natoms) {
    box = s.atom_box[i];
    const int sl = nb.slot_of[i];
    double r[3];
#pragma unroll
    for (int c = 0; c < 3; c++) r[c] = nb.xref[3 * i + c];
    if (sl >= 0) {
      const BoxDev &b = s.box[box];
      // x, y, z of the record; the charge in its last word stays
      uint4 *f = nb.slot_fx + sl;
      *reinterpret_cast<uint2 *>(f) = make_uint2(frac_fixed(x[0], b.Lr[0]), frac_fixed(x[1], b.Lr[1]));
      f->z = frac_fixed(x[2], b.Lr[2]);
      if (nb.want_fp64) {
        double4 *q = nb.slot_pq + sl;
        *reinterpret_cast<double2 *>(q) = make_double2(x[0], x[1]);
        q->z = x[2];
      }
    }
    if (!(isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]))) atomicExch(&nb.status[2], 1);
    if (vacuum) {
      int *e = nb.vext + 6 * box;
#pragma unroll
      for (int d = 0; d < 3; d++) {
        const int o = ford((float)x[d]);
        atomicMin(e + d, o);
        atomicMax(e + 3 + d, o);
      }
      __threadfence();
    }
    const double dx = x[0] - r[0], dy = x[1] - r[1], dz = x[2] - r[2];
    const double r2 = dx * dx + dy * dy + dz * dz;
    d2 = r2 < 3.0e38 ? (float)r2 : 3.0e38f;
    if (!(d2 >= 0.f)) d2 = 3.0e38f;  // NaN positions force a rebuild
  }
  // per-box maxima (float bits of non-negative values order as unsigned): a warp whose atoms
  // belong to one box takes its maximum first, and the block adds one atomic per run of such
  // warps of the same box
  constexpr int NW = UPDATE_THREADS / 32;
  __shared__ int wbox[NW];
  __shared__ float wmax[NW];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned act = __ballot_sync(0xffffffffu, box >= 0);
  int wb = -1;  // the warp's box when all its atoms share one, else -1 (atomics already added)
  float m = 0.f;
  if (act) {
    const int b0 = __shfl_sync(0xffffffffu, box, __ffs(act) - 1);
    if (__all_sync(0xffffffffu, box < 0 || box == b0)) {
      m = d2;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      wb = b0;
    } else if (box >= 0) {
      atomicMax(&nb.box_d2[box], __float_as_uint(d2));
    }
  }
  if (lane == 0) {
    wbox[w] = wb;
    wmax[w] = m;
  }
  // one fence and one count per block: thread 0 makes the block's maxima (and, through the barrier,
  // its other writes) visible before it counts the block
  if (vacuum || wb < 0) __threadfence();  // this thread's own atomics
  __syncthreads();
  __shared__ bool last;
  if (threadIdx.x == 0) {
    for (int k = 0; k < NW;) {
      const int b = wbox[k];
      float mm = wmax[k];
      int k2 = k + 1;
      for (; k2 < NW && wbox[k2] == b; k2++) mm = fmaxf(mm, wmax[k2]);
      if (b >= 0) atomicMax(&nb.box_d2[b], __float_as_uint(mm));
      k = k2;
    }
    __threadfence();
    last = atomicAdd(&nb.ctl[CTL_BLOCKS], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const bool forced = nb.ctl[CTL_FORCED] != 0u;
  int any = 0;
  for (int b = threadIdx.x; b < s.nbox; b += blockDim.x) {
    const float mx = __uint_as_float(atomicExch(&nb.box_d2[b], 0u));  // read and reset
    const unsigned rb = (forced || mx > nb.half_skin2) ? 1u : 0u;
    nb.box_rb[b] = rb;
    any |= (int)rb;
    if (vacuum)
      for (int d = 0; d < 3; d++) {
        // read and reset for the next evaluation
        const float lo = fuord(atomicExch(nb.vext + 6 * b + d, 0x7fffffff));
        const float hi = fuord(atomicExch(nb.vext + 6 * b + 3 + d, (int)0x80000000));
        if (!((double)hi - (double)lo < 0.5 * s.box[b].L[d])) atomicExch(&nb.status[3], 1);
      }
  }
  any = __syncthreads_or(any);
  if (threadIdx.x == 0) {
    nb.ctl[CTL_REBUILD] = any ? 1u : 0u;
    if (any) {
      ++*reinterpret_cast<unsigned long long *>(nb.ctl + CTL_BUILDS);
      // the build starts its list of pair units anew
      nb.ctl[CTL_CLAIM] = nb.ctl[CTL_UNITS] = nb.ctl[CTL_UNITS + 1] = 0u;
    }
    nb.ctl[CTL_BLOCKS] = 0u;
    nb.ctl[CTL_FORCED] = 0u;
    if (step) *step += 1;  // (every block has read it)
  }
}

}  // namespace pmb
