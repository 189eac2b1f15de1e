// Host-side declarations shared by the .cu translation units of libpmb200.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "pmb_common.cuh"

namespace pmb {

void set_error(const std::string &msg);

#define PMB_CUDA(expr)                                                                   \
  do {                                                                                   \
    cudaError_t _e = (expr);                                                             \
    if (_e != cudaSuccess) {                                                             \
      ::pmb::set_error(std::string(#expr) + ": " + cudaGetErrorString(_e));              \
      return PMB_ERR_CUDA;                                                               \
    }                                                                                    \
  } while (0)

enum {
  PMB_OK_ = 0,
};

// Index of the current device for per-device one-time settings (a kernel's attributes, such as
// its dynamic shared-memory limit, belong to the device they were set on).
constexpr int PMB_MAX_DEVICES = 64;
inline int device_slot() {
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= PMB_MAX_DEVICES) d = 0;
  return d;
}

// ------------------------------------------------------------------ neighbour list (nblist.cu)
// Control words of a list.
enum {
  CTL_REBUILD = 1,  // some box rebuilds this step
  CTL_BLOCKS = 2,   // finished blocks of the displacement check
  CTL_FORCED = 3,   // every box rebuilds at the next check
  CTL_BUILDS = 4,   // list builds so far (64 bits)
  CTL_PAIR = 6,     // the pair kernel's next unit and finished warps, two launches; zero between them
  CTL_VACUUM = 10,  // check the extent of vacuum boxes
  CTL_CLAIM = 11,   // the list build's next claim
  CTL_UNITS = 12,   // pair units of boxes without and with lattice images
  CTL_WORDS = 16
};
constexpr int SORT_PART = 512;  // slots of a CTA of the sort's launches per phase
// Sort bins: one CTA scans a box's up to here, in chunks of SCAN_CHUNK; more are scanned chunk by chunk
// over the whole chip.
constexpr int SCAN_CHUNK = 8192, SCAN_ONE_CTA = 4 * SCAN_CHUNK;
struct NbListDev {
  // per block
  int nblk_total;
  const int *blk_box;          // [nblk]
  float4 *blk_center;          // [nblk] fractional-fixed centre (as uint bits) and count
  uint4 *blk_lo, *blk_hi;      // [nblk] fixed-point extents (x, y, z)
  uint4 *blk_c, *blk_h;        // [nblk] the same as centre (.w = atoms) and half extent
  int nsblk;                   // superblocks: runs of 32 consecutive blocks of a box
  uint4 *sblk_c, *sblk_h;      // [nsblk] union of their blocks' extents: centre (.w = atoms), half extent
  int *jcap_off;               // [nblk+1] offset of each block's j-slot list region
  int *jcount;                 // [nblk] tiles per block (its j-list, own slots first, in 32s)
  int *jlist;                  // [jcap_off[nblk]] j slots (-1 padding), JSAME flag bit
  int4 *units;                 // [unit_cap] pair kernel work: block, first tile, tiles, offset of the
                               // first tile in jlist; boxes that
                               // need lattice images from the end of the array, the others from
                               // the front (ctl[CTL_UNITS + 1] and ctl[CTL_UNITS] of them)
  int unit_cap;
  int claim_blocks;            // consecutive blocks of a claim of the list build
  bool fills_chip;             // about a unit or more for every warp the chip holds
  int unit_tiles;              // most tiles of a unit: CLOSE_TILES .. UNIT_TILES
  int *status;                 // [4]: list / tile overflow, non-finite position, vacuum extent
  // per slot
  int nslot;
  int *slot_orig;              // [nslot] original atom index or -1
  uint4 *slot_fx;              // [nslot] fractional fixed-point x, y, z (2^32 per edge) + q bits
  double4 *slot_pq;            // [nslot] raw double position + q (FP64 path)
  int4 *slot_meta;             // [nslot] orig, molecule, type, box
  long long *fslot;            // [3][nslot] pair forces by slot (component-major), fixed point
  // sort
  int nkeys;
  int *key;                    // [natoms] sort bin within the atom's box
  int *rank;                   // [natoms]
  int *bin_count;              // [nkeys] zero between builds
  int *bin_start;              // [nkeys] relative to the box's first slot
  const int2 *sort_work;       // [nsort] box, part of SORT_PART slots
  int nsort;
  const int2 *scan_work;       // [nscan] bins of boxes of more than SCAN_ONE_CTA: box, chunk of SCAN_CHUNK
  int nscan;
  int *bin_sums;               // [nscan] atoms in each of those chunks
  int *slot_raw;               // [nslot] atoms by bin, before they are ordered within the bins
  int *slot_of;                // [natoms] slot of each atom (-1 before the first build)
  int max_box_atoms, n_sm;     // largest box; SMs of the device
  int want_fp64;               // also pack raw double positions
  // list reuse: the list is built with cutoff + skin and rebuilt only once some atom moved more
  // than skin/2 since the last build (decided on the device, every step)
  double *xref;                // [3 natoms] positions at the last build
  unsigned *ctl;               // [CTL_WORDS], see below
  float half_skin2;
  // per box: rebuilds are decided box by box (a box's list, slot order and therefore its
  // rounding do not depend on the other boxes of the system); ctl[CTL_REBUILD]: any box rebuilds
  int nbox;
  unsigned *box_d2;            // [nbox] max displacement^2 since the box's last build (float bits)
  unsigned *box_rb;            // [nbox] 1: the box rebuilds this step
  unsigned *box_done;          // [nbox] finished CTAs of the histogram; zero between launches
  int *vext;                   // [6 nbox] vacuum extent per box: smallest and largest x, y, z as
                               // order-preserving int images of their float values (CTL_VACUUM on)
};

struct SystemDev {
  int nbox, natoms;
  const BoxDev *box;           // [nbox]
  const int *atom_box;         // [natoms]
  const double *pos;           // [3 natoms] caller order
  const double *charge;        // [natoms]
  const int *type, *molecule;  // [natoms]
  const int *excl_start, *excl_partner, *excl_kind;  // CSR by atom
  // the forces of the last evaluation, fixed point: facc by atom plus fslot by slot (component-major
  // [3][nslot], the pair kernel's part; slot_of null without a list), summed by who reads them
  long long *facc;             // [3 natoms]
  long long *fslot;
  const int *slot_of;          // [natoms]
  int nslot;
  long long *eacc;             // [nbox * ACC_PER_BOX]
};

int nblist_sort(const SystemDev &s, NbListDev &nb, bool updated, cudaStream_t st);
int nblist_lists(const SystemDev &s, NbListDev &nb, double list_cutoff, cudaStream_t st);
int fp32_peak_probe(double *tflops);

// ------------------------------------------------------------------ pair kernel (pair.cu)
struct PairLaunch {
  int precision;                  // 0 fp64, 1 mixed
  int do_lj, coul_mode, virial;
  const double *lj;               // [ntypes*ntypes*4] device
  const float *ljf;               // float copy
  const double *lattice;          // [nlat_total*3]
  int multi;                      // some box needs Ewald lattice images
  int ctas_per_sm;                // resident CTAs per SM of the persistent kernel (0: all that fit)
  int unit_kinds;                 // units it evaluates: bit 0 those of boxes without lattice images,
                                  // bit 1 those of boxes with
  int wslot;                      // which unit counter of the list's ctl words it uses (0 or 1)
  PairParams p;
};
int pair_launch(const SystemDev &s, const NbListDev &nb, const PairLaunch &pl, cudaStream_t st);
int pair_fold(const SystemDev &s, const NbListDev &nb, cudaStream_t st);

// Allocation-free all-pairs variant (FP64): energy/virial accumulators in a static device array
// of STATIC_MAX_BOXES boxes.  static_eacc_address looks the array up once per device (current
// device); pair_allpairs_launch zeroes s.nbox boxes of it on st, then writes fout [3 natoms].
constexpr int STATIC_MAX_BOXES = 1024;
cudaError_t static_eacc_address(long long **out);
cudaError_t pair_allpairs_launch(const SystemDev &s, const PairParams &p, const double *ljd,
                                 const double *pos, double *fout, long long *eacc,
                                 int max_box_atoms, cudaStream_t st);

// ------------------------------------------------------------------ PME (pme.cu)
struct PmeBoxPlan {
  int n[3];
  long long grid0;    // offset of this box's real/fixed grid (elements)
  long long cgrid0;   // offset of this box's half-complex grid (elements)
  int tw0[3];         // offsets of twiddle tables (complex elements)
  int inf0[3];        // offsets of influence tables
  int rad0[3], nrad[3];
  int prad0[3], npr[3];  // radices of the register-stage transforms (x and y: plane kernel)
  double hr[3];       // n / L
  double mr[3];       // 1 / L
  double piVr, fac;   // 1/(pi V), pi^2 / alpha^2
};

struct PmeDev {
  int nbox, order, precision;
  const PmeBoxPlan *plan;     // [nbox] device
  long long *qgrid;           // fixed-point charge grid
  void *cgrid;                // half-complex grid (float2 or double2), layout [kz][x][y]
  void *rgrid;                // real potential grid (float or double), layout [x][y][z]
  const double2 *twiddle;     // per dim tables exp(-2 pi i k / n)
  const float2 *twiddlef;
  const double *infl;         // per dim influence factor B(m) exp(-pi^2 m^2/alpha^2)
  const void *theta;          // influence function per half-spectrum point (float / double,
                              // layout as cgrid), 0 at m = 0
  const int *radix;           // radices per dim
  const int4 *zwork;          // z-pass work items: box, x, y0, count
  int nzwork;
  // planes too large for the plane kernel: line work items, those of lines of 32 R points
  // (WARP_R_MIN <= R <= WARP_R_MAX, the warp-shuffle transforms) from item [R] up to [R + 1], those of the shared-memory ones from [0]
  const int4 *ywork;          // box, kz, x0, rows
  int nywork[7];
  const int4 *xwork;          // box, kz, y0, columns
  int nxwork[7];
  const int2 *pwork;          // planes of the plane kernel: box, kz
  int npwork, pthreads;
  size_t psmem;
  const int *pradix;          // its radices
  const int *perm;            // (offsets tw0) x and y: index at each position of the plane kernel's
                              // transformed lines, theta is in that order then; z: position of index
  int zpairs;                 // packed lines of a full work item of the z kernels
  size_t zsmem;               // shared memory of the z kernels
  int lbuf;                   // complex elements per ping-pong buffer of the line kernels
  double alpha, a2pi;
  int virial;
};
// Block size of the warp-transform x kernel (one column per warp).
#ifndef PME_WX_THREADS
#define PME_WX_THREADS 256
#endif
// Optional stage marker (profiling): called on the host between kernel launches.
typedef void (*StageMark)(void *ctx, const char *stage);
// head: recorded on st once the z transforms are enqueued (null: not)
int pme_recip_launch(const SystemDev &s, const NbListDev &nb, const PmeDev &pm, cudaStream_t st, cudaEvent_t head = nullptr,
                     StageMark mark = nullptr, void *mark_ctx = nullptr);
int pme_line_capacity();
// Plane kernel: most threads, most shared memory, the stages of a line, a plane's shared memory.
constexpr int PLANE_MAX_THREADS = 512;
constexpr int PLANE_SMEM_MAX = 227 * 1024;
// Warp-shuffle lines of 32 R points: the shortest in a plane that does not fit (FP64, mixed), the longest.
constexpr int WARP_R_MIN[2] = {2, 4}, WARP_R_MAX = 5;
bool pme_plane_radices(int n, std::vector<int> &radices);
size_t pme_plane_smem(int nx, int ny, int precision);
constexpr int Z_SMEM_MAX = 48 * 1024;  // z kernels: 16 lines of 256 points in FP64 take 37 KB
// Stride of a packed line in the z kernels' buffer.  Consecutive threads take the same point of
// consecutive lines: with 16 / pairs + 16 i eight-byte numbers (an odd count of sixteen-byte ones)
// between lines a half (quarter) warp falls on different banks, whatever the stage.
__host__ __device__ inline int z_line_stride(int nz, int pairs, bool f32) {
  if (!f32) return nz | 1;
  const int off = pairs > 8 ? 1 : pairs > 4 ? 2 : 4;
  return nz + ((off - nz) & 15);
}
size_t pme_z_smem(int nz, int lines, int precision);
// Exact Ewald reciprocal sum of one box (pmb_ewald.cu): S, C [nk] and the box's forces in fout.
int ewald_recip_launch(const double *pos, const double *charge, int atom0, int n, const double3 *kv,
                       const double *a, int nk, double *S, double *Cc, double *fout, cudaStream_t st);

// ------------------------------------------------------------------ bonded / integrator (md.cu)
struct BondedDev {
  int nbonds, nangles;
  const int *bonds;
  const double *bond_k, *bond_r0;
  const int *angles;
  const double *angle_k, *angle_theta0, *ub_k, *ub_r0;
  int virial;
};
// Exclusion corrections of a PME force: the pairs, and its splitting parameter.
struct CorrectionDev {
  int n;
  const int *pairs, *kind;
  double alpha, a2pi, coulomb_scaling;
  int virial;
};
// Exclusion corrections and bonded terms in one launch (either may be null).
int atom_terms_launch(const SystemDev &s, const CorrectionDev *c, const BondedDev *b, cudaStream_t st);
// fout = base + the accumulated forces (base may be null), eout = the energies; either may be null
int results_to_double(const SystemDev &s, double *fout, const double *base, double *eout, cudaStream_t st);
int forces_to_double(const SystemDev &s, double *out, cudaStream_t st);
int energies_to_double(const SystemDev &s, double *out, cudaStream_t st);
int zero_accumulators(const SystemDev &s, cudaStream_t st);

struct IntegratorDev {
  int kind;            // 0 leapfrog, 1 Langevin
  double h;            // dt * INV_TIMEFACTOR
  double gamma, kT;    // Langevin (internal units)
  unsigned long long seed;
  // per box: the noise seed and the offset of the box's step count from the run's (a box that
  // joined the run part-way); an atom's noise is keyed by its box's seed, its index within the
  // box and its box's step, so a box draws the same numbers alone and beside other boxes
  const unsigned long long *box_seed;  // [nbox]
  const long long *box_step0;          // [nbox]
  double fdt, vdt, ndt;  // Langevin half kick factors (langevin_half_kick)
  const double *mass;  // [natoms]
  double *pos, *vel;
  long long *step;     // device step counter
};
// SHAKE / RATTLE bond constraints, one thread per connected group of constraints (a rigid water:
// 3 constraints on 3 atoms).  A group's constraints keep their order in the reference's list.
constexpr int CON_MAX_ATOMS = 8;    // atoms of one group
constexpr int CON_MAX_CONS = 16;    // constraints of one group
constexpr double CON_ERR_SCALE = 1099511627776.0;  // 2^40: fixed point of the per-sweep error sums
struct ConstraintDev {
  int ngroup, ncons;
  int max_atoms, max_cons;  // largest group (selects the kernel: rigid waters have 3 and 3)
  int water3;               // every group: three atoms, constraints 0-1, 0-2, 1-2 in that order
  const int *group_con;    // [ngroup + 1] constraint offsets of each group
  const int *group_atom;   // [ngroup + 1] offsets into atoms
  const int *atoms;        // group atoms (global indices), each group's first-use order
  const int2 *con_local;   // [ncons] the two atoms of a constraint as indices into its group
  const double *len;       // [ncons] rest lengths
  double *rab;             // [3 ncons] SHAKE reference vectors x[a1] - x[a2] of the last SHAKE
  long long *err;          // [2][CON_ERR_BLOCK]: per modifier, the per-sweep error sums of the
                           // two rounds and the hand-over words (continue flag, first-round sweeps)
  int *sweeps;             // [2] sweeps of the last SHAKE and RATTLE (the next first round scans
                           // up to two more)
  double *win;             // [CON_WINDOW][6][max_atoms][ngroup] group states at the sweep counts
                           // around the last one, written by the first scan
  double clamp;            // largest group error added to a sum (keeps the int64 sums in range)
  double dt;               // timestep / TIMEFACTOR, as the modifiers use it
  double shake_eps, rattle_eps;
  int shake_max, rattle_max;
  // RATTLE's constraint virial (ModifierRattle.cpp:58), added to the box accumulators when set
  int virial;
  long long *eacc;
  const int *atom_box;
};
constexpr int CON_MAX_SWEEPS = 256;  // max_iter + 1 bound
constexpr int CON_ERR_BLOCK = 2 * (CON_MAX_SWEEPS + 1) + 2;
constexpr int CON_WINDOW = 3;
int constraints_init(const ConstraintDev &c, const IntegratorDev &in, cudaStream_t st);
int constraints_apply(const ConstraintDev &c, const IntegratorDev &in, int rattle, cudaStream_t st);
// kick and drift; with nb also the list's displacement check and slot records (update_atom)
int integrate_kick_drift(const SystemDev &s, const IntegratorDev &in, double kick, NbListDev *nb, cudaStream_t st);
int integrate_half_kick(const SystemDev &s, const IntegratorDev &in, cudaStream_t st);
// parts [KIN_PARTS nbox] and done [nbox] (zero between launches): scratch
constexpr int KIN_PARTS = 64;
int kinetic_energy(const SystemDev &s, const IntegratorDev &in, double *out_per_box, double *parts, unsigned *done,
                   int max_box_atoms, cudaStream_t st);

}  // namespace pmb
