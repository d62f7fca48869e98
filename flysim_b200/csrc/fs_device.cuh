// Device-side data of the flysim step engine (shared by the kernels and the
// C ABI implementation).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "flysim_b200.h"

namespace fsd {

constexpr uint32_t kFull = 0xffffffffu;

// Reference-order layout of one receptor on the device (fs_rec_layout).
struct RecDev {
  uint32_t n_gates;
  const uint32_t *gate_pre, *gate_post0;
  const float *gate_g;
  float *gate_st, *gate_xt;      // gate_st: [2][n_gates] by step parity
  const uint32_t *grow, *ggate;  // gather CSR by post
  uint32_t n_recs;
  const uint32_t *rpre, *rpost;
  const uint8_t *rloc;           // post of each record, counted from its tile's first
  float *rg, *rst, *rxt;
  const uint32_t *rrow;  // records CSR by post
};

constexpr uint32_t kCompatTile = 64;  // posts of a k_compat tile at most

// Per-neuron words of a k_compat tile: parameters and state (five in a row per
// receptor where the reference has one per receptor, four for CS_EST).
enum {
  CP_ACT = 0, CP_VREV = 1, CP_DFST = 6, CP_EXTG = 11, CP_PB = 16, CP_NDFXT = 21, CP_NEFST, CP_NAS, CP_NMG, CP_GL, CP_EL,
  CP_CM, CP_VRESET, CP_DF, CP_EF, CP_DVMAX, CP_VTH, CP_RF, CP_SD, CP_IMEAN, CP_ISTD, CP_DRAWOFF, CP_INJOFF, CP_DFLP,
  CP_SPILP, CP_N
};
enum {
  CS_V = 0, CS_COUNT, CS_NS, CS_ISYN, CS_G = 4, CS_EST = 9, CS_EXT = 13, CS_ESTN, CS_IREP = 15, CS_LP = 20, CS_CLP, CS_N
};

// Everything the compat kernels touch; passed by value.
struct CompatDev {
  uint32_t n;
  uint32_t glob;  // global ActCtr (STP/STD/LTP)
  // parameters
  const float *Vth, *El, *gl, *Cm, *Vreset, *df, *ef, *dVmax;
  const int32_t *RfPed, *SpiDy;
  const float *Vrev, *dfst, *nmda_dfxt, *nmda_efst, *nmda_as, *nmda_mg, *ext_g;
  const float *pb;
  const uint32_t *act;
  const float *inj_mean, *inj_std;
  const float *stp_pv, *stp_dfD, *stp_efD, *stp_aF, *stp_dfF, *stp_efF, *stp_aCap, *stp_dfCap,
      *stp_aCar, *stp_dfCar, *stp_efCar;
  const float *ltp_dfLP, *ltp_Pos, *ltp_Neg;
  const int32_t *ltp_SpiLPDy;
  // state
  float *V, *Isyn, *G, *ext_st, *ext_xt_n, *ext_st_n, *Irep, *D, *F, *Cap, *Car, *LP;
  int32_t *Count, *CountLP;
  uint32_t *NS;
  const uint32_t *npar[CP_N];  // the parameters and state above as words (k_compat)
  uint32_t *nst[CS_N];
  float *LP2, *V2, *inc2;  // [2][n] by step parity (null unless LTP / gap junctions / STP or STD)
  RecDev R[FS_NREC];
  const uint32_t *gby_row, *gby_ent;  // all receptors' gates by presynaptic neuron (null: none)
  uint32_t gate_off[FS_NREC + 1];  // prefix of n_gates
  uint32_t rec_off[FS_NREC + 1];   // prefix of n_recs
  const uint32_t *gap_row, *gap_other;
  const float *gap_g;
  // random streams of one batch
  const uint32_t *drawoff;  // [n] first draw of neuron i within a step
  const uint32_t *injoff;   // [n] rank of neuron i among injected neurons
  uint32_t draws_per_step, inj_per_step;
  uint32_t jcong_base;      // congruential state before the batch's first Gaussian
  // glibc-exact expf / logf exception tables: hashed (hash_fill), or, for
  // expf without one, sorted by key
  const uint4 *expf_tab, *logf_tab;
  const uint32_t *expf_keys;
  const float *expf_vals;
  uint32_t expf_n;
  // per-step outputs of the batch
  uint32_t *spikebits;      // [nsteps][words]
  uint32_t words;
  float *outV, *outIrep;
  uint32_t *outNS;
  const uint32_t *gv_sel;
  uint32_t gv_n;
  float *gv_st, *gv_xt;
  int *err;                 // device error word
};

// One call's steps (k_compat).
struct CompatRun {
  uint32_t nsteps;
  uint32_t gpar;   // parity of the group gates' buffer the first step writes
  uint32_t blocks, tiles;  // blocks that own tiles; tile t: posts [tile_post[t], tile_post[t + 1])
  const uint32_t *tile_post;
  // the random stream: the last block of 624 words drawn and how many of them
  // were used; a ring of ring_blocks blocks (set by compat_steps) that holds
  // the words of two steps (draws_ring_words(5 n) words always do)
  uint32_t *mt_state, *mt_pos, *ring;
  uint32_t ring_blocks;
  unsigned int *bar;
};

constexpr size_t draws_ring_words(size_t draws_per_step) { return 2 * draws_per_step + 3 * 624; }

// Launch wrappers (fs_compat.cu)
void compat_set_tables(const uint32_t kn[128], const float fn[128], const float wn[128],
                       const uint32_t jump_a[32], const uint32_t jump_c[32], cudaStream_t st);
cudaError_t compat_blocks(uint32_t sm_count, uint32_t *blocks);
cudaError_t compat_steps(const CompatDev &d, CompatRun R, cudaStream_t st, uint64_t *launches);
cudaError_t compat_varinit(const CompatDev &d, cudaStream_t st);
cudaError_t spikes_compact(const uint32_t *bits, uint32_t nsteps, uint32_t words, uint32_t *counts,
                           uint32_t *offsets, uint32_t *idx, cudaStream_t st, uint64_t *launches);
// Hash of an exception table (2^kHashBits buckets of four key-value pairs).
constexpr uint32_t kHashBits = 17, kHashEmpty = 0xffffffffu;
constexpr size_t kHashBytes = (size_t)32 << kHashBits;
cudaError_t hash_fill(const uint32_t *keys, const float *vals, uint32_t n, uint4 *tab, cudaStream_t st);
// loc[e] = in_tile[p] for the records e of post p (row: records by post)
cudaError_t fill_loc(const uint32_t *row, const uint8_t *in_tile, uint32_t n, uint8_t *loc, cudaStream_t st);
// test hooks
cudaError_t expf_ref_eval(const float *x, float *y, uint64_t k, const uint32_t *keys, const float *vals,
                          uint32_t nk, const uint4 *tab, cudaStream_t st);

}  // namespace fsd
