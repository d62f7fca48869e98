// Reference-order FP32 kernels of the flysim step (FS_MODE_COMPAT).
//
// Compiled with -fmad=false and IEEE division/denormals (no fast math): every
// floating-point expression below is evaluated with the operand order and
// rounding of the reference's g++ -O3 SSE2 build, so the spike raster equals
// the reference's bit for bit.  Kernel map (reference code they replace):
//   k_compat      all steps of a call in one persistent launch:
//     activate      EqsGnl2::Activation = BgInit + VmEul + firing (+ firLP/ltpEul)
//                   (code/EqsGnl2.cpp:152-337, :1098-1105); one thread per neuron
//     tile_gates    ThdPGatVar / STD / STP: group gate updates (code/EqsGnl2.cpp:728-932)
//     tile_terms,   ThdPSynapse + ThdSynapse* + ThdGapSyn (code/EqsGnl2.cpp:404-725,
//     tile_sums     :937-1002): a tile's terms formed by all threads in shared
//                   memory, then added by one thread per (post, receptor) in the
//                   reference's order; LTP (code/EqsGnl2.cpp:1005-1044) rewrites a
//                   record's weight right after its term
//     MtBlock       the std::mt19937 output stream the reference draws from, on a
//                   block of its own, one step ahead
//   k_count / k_write   ordered spike-list compaction (ballot bitmaps, block prefix)
#include <cstdint>
#include <cuda_runtime.h>
#include "fs_barrier.cuh"
#include "fs_device.cuh"

namespace fsd {

__constant__ uint32_t c_kn[128];
__constant__ float c_fn[128];
__constant__ float c_wn[128];
__constant__ uint32_t c_jump_a[32];  // congruential map x -> a*x + c raised to 2^i
__constant__ uint32_t c_jump_c[32];

// ---- glibc-exact float exp/log ----------------------------------------
// (float)exp((double)x) rounds correctly except when e^x lies within a few
// double ulps of a float rounding boundary; glibc's expf itself is not always
// correctly rounded.  The exception table holds glibc's result for every
// input of the tabulated range where the two may differ (generated at build
// time by calling glibc, see fs_tables.cpp).
__device__ __forceinline__ float table_patch(float r, float x, const uint32_t *keys, const float *vals,
                                             uint32_t n) {
  const uint32_t k = __float_as_uint(x);
  uint32_t lo = 0, hi = n;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(keys + mid) < k) lo = mid + 1;
    else hi = mid;
  }
  if (lo < n && __ldg(keys + lo) == k) r = __ldg(vals + lo);
  return r;
}
// The same look-up through a hash of the table: 2^kHashBits buckets of four
// (key, value) pairs, one 32-byte sector each; a full bucket runs over into
// the next (0.4 % at 140,931 entries).  The binary search is 18 dependent
// loads, about 10 us on the critical path of every step; a bucket is one.
__device__ __forceinline__ uint32_t hash_bucket(uint32_t key) { return (key * 0x9E3779B1u) >> (32 - kHashBits); }
__device__ __forceinline__ float hash_patch(float r, float x, const uint4 *tab) {
  const uint32_t k = __float_as_uint(x);
  for (uint32_t b = hash_bucket(k), i = 0; i < (1u << kHashBits); b = (b + 1) & ((1u << kHashBits) - 1u), i++) {
    const uint4 p = __ldg(tab + 2 * b), q = __ldg(tab + 2 * b + 1);
    if (p.x == k) return __uint_as_float(p.y);
    if (p.z == k) return __uint_as_float(p.w);
    if (q.x == k) return __uint_as_float(q.y);
    if (q.z == k) return __uint_as_float(q.w);
    if (q.z == kHashEmpty) break;
  }
  return r;
}
// tab: all bytes 0xff (empty) before the call
__global__ void k_hash_fill(const uint32_t *keys, const float *vals, uint32_t n, uint32_t *tab) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t k = keys[i];
  for (uint32_t b = hash_bucket(k), j = 0; j < (1u << kHashBits); b = (b + 1) & ((1u << kHashBits) - 1u), j++)
    for (uint32_t q = 0; q < 4; q++) {
      uint32_t *slot = tab + 8 * (size_t)b + 2 * q;
      if (atomicCAS(slot, kHashEmpty, k) == kHashEmpty) {
        slot[1] = __float_as_uint(vals[i]);
        return;
      }
    }
}
cudaError_t hash_fill(const uint32_t *keys, const float *vals, uint32_t n, uint4 *tab, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(tab, 0xff, kHashBytes, st);
  if (e == cudaSuccess && n) {
    k_hash_fill<<<(n + 255) / 256, 256, 0, st>>>(keys, vals, n, (uint32_t *)tab);
    e = cudaGetLastError();
  }
  return e;
}

// A warp per post.
__global__ void __launch_bounds__(256) k_fill_loc(const uint32_t *row, const uint8_t *in_tile, uint32_t n, uint8_t *loc) {
  const uint32_t p = blockIdx.x * 8u + (threadIdx.x >> 5);
  if (p >= n) return;
  const uint8_t v = in_tile[p];
  for (uint32_t e = row[p] + (threadIdx.x & 31u), e1 = row[p + 1]; e < e1; e += 32) loc[e] = v;
}
cudaError_t fill_loc(const uint32_t *row, const uint8_t *in_tile, uint32_t n, uint8_t *loc, cudaStream_t st) {
  k_fill_loc<<<(n + 7) / 8, 256, 0, st>>>(row, in_tile, n, loc);
  return cudaGetLastError();
}

// Every expf exception lies within 0.0017 float ulp of a rounding boundary
// (checked against the table by tests/test_expf_table.py); only results
// within 2^-8 ulp of one, about one in 128, look the table up.
__device__ __forceinline__ float expf_ref(float x, const CompatDev &d) {
  const double v = exp((double)x);
  const int off = (int)((uint32_t)__double2loint(v) & 0x1fffffffu) - 0x10000000;
  const float r = (float)v;
  if (off > 0x00200000 || off < -0x00200000) return r;
  return d.expf_tab ? hash_patch(r, x, d.expf_tab) : table_patch(r, x, d.expf_keys, d.expf_vals, d.expf_n);
}
__device__ __forceinline__ float logf_ref(float x, const CompatDev &d) {
  return hash_patch((float)log((double)x), x, d.logf_tab);
}

// ---- random streams ----------------------------------------------------
// The standard MT19937 recurrence (Matsumoto & Nishimura 1998; the
// parameters are those std::mt19937 fixes): x[k+624] = x[k+397] ^ A(x[k], x[k+1]).
__device__ __forceinline__ uint32_t mt_twist(uint32_t xi, uint32_t xi1) {
  const uint32_t y = (xi & 0x80000000u) | (xi1 & 0x7fffffffu);
  return (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
}
__device__ __forceinline__ uint32_t mt_temper(uint32_t y) {
  y ^= (y >> 11);
  y ^= (y << 7) & 0x9d2c5680u;
  y ^= (y << 15) & 0xefc60000u;
  y ^= (y >> 18);
  return y;
}
// uniform_real_distribution<float>(0,1) over mt19937 (libstdc++
// generate_canonical<float,24>: one 32-bit draw, float(x) * 2^-32, values
// rounding up to 1 replaced by the largest float below 1).
__device__ __forceinline__ float u01(uint32_t x) {
  float u = __uint2float_rn(x) * 2.3283064365386963e-10f;
  return (u >= 1.0f) ? 0.99999994f : u;
}

__device__ __forceinline__ uint32_t shr3(uint32_t &jsr) {
  const uint32_t in = jsr;
  jsr = jsr ^ (jsr << 13);
  jsr = jsr ^ (jsr >> 17);
  jsr = jsr ^ (jsr << 5);
  return in + jsr;
}
__device__ __forceinline__ float zuni(uint32_t &jsr) {
  const uint32_t in = jsr;
  jsr = jsr ^ (jsr << 13);
  jsr = jsr ^ (jsr >> 17);
  jsr = jsr ^ (jsr << 5);
  return (float)fmod(0.5 + (double)__uint2float_rn(in + jsr) / 65536.0 / 65536.0, 1.0);
}
// Marsaglia–Tsang ziggurat normal (code/StiExt.h:262-319).
__device__ float zig_nor(uint32_t &jsr, const CompatDev &d) {
  const float r = 3.442620f;
  int hz = (int)shr3(jsr);
  uint32_t iz = (uint32_t)(hz & 127);
  if (fabs((double)hz) < (double)c_kn[iz]) return (float)hz * c_wn[iz];
  for (int guard = 0; guard < 100000; guard++) {
    if (iz == 0) {
      float x, y;
      for (int g2 = 0; g2 < 100000; g2++) {
        x = (float)(-0.2904764 * (double)logf_ref(zuni(jsr), d));
        y = -logf_ref(zuni(jsr), d);
        if (x * x <= y + y) break;
      }
      return (hz <= 0) ? -r - x : r + x;
    }
    const float x = (float)hz * c_wn[iz];
    const float lhs = c_fn[iz] + zuni(jsr) * (c_fn[iz - 1] - c_fn[iz]);
    if ((double)lhs < exp(-0.5 * (double)x * (double)x)) return x;
    hz = (int)shr3(jsr);
    iz = (uint32_t)(hz & 127);
    if (fabs((double)hz) < (double)c_kn[iz]) return (float)hz * c_wn[iz];
  }
  if (d.err) atomicOr(d.err, 1);
  return 0.0f;
}
// jcong after k further congruential steps
__device__ __forceinline__ uint32_t jcong_jump(uint32_t x, uint32_t k) {
#pragma unroll 1
  for (int i = 0; k; i++, k >>= 1)
    if (k & 1) x = c_jump_a[i] * x + c_jump_c[i];
  return x;
}

// ---- firing (code/EqsGnl2.cpp:229-251) ----------------------------------
__device__ __forceinline__ void firing(float &V, int32_t &cnt, uint32_t &ns, int32_t rf, int32_t sd,
                                       float vreset) {
  if (cnt < rf) {
    V = (cnt == 0) ? 0.0f : vreset;
    if (cnt == sd) ns |= FS_NS_SPIKE;
    else ns &= ~FS_NS_SPIKE;
    cnt++;
  } else {
    cnt = 0;
    ns &= ~FS_NS_FIRE;
  }
}

constexpr uint32_t kCT = 256;       // threads of a k_compat block
constexpr uint32_t kUnit = 128;     // items of a work unit: four a lane
constexpr uint32_t kPassUnits = 56;
constexpr uint32_t kCTerms = kPassUnits * kUnit;  // terms of a pass in shared memory
constexpr int kSpans = 2 * FS_NREC;
constexpr uint32_t kBitWords = 1024;

// Arrays of a span from the tile's first entry on.
struct Span {
  const uint32_t *k;    // gates of the gather entries, or the records' presynaptic neurons
  const uint32_t *post;
  const uint8_t *loc;
  float *st, *xt, *g;   // records; a gather's gates: st (this step's buffer is par * n_gates on), g
  uint32_t n_gates;
};

// One tile (the posts a block advances together): its neurons' parameters and
// state (CompatDev::npar and nst, a word per neuron), the terms of a pass and
// the shape of its sequence of synaptic items (tile_items).
struct CompatSmem {
  float terms[kCTerms];
  uint32_t par[CP_N][kCompatTile], st[CS_N][kCompatTile];
  uint32_t off[kSpans][kCompatTile + 1];
  float2 inc[kCompatTile];
  bool spk[kCompatTile];
  uint32_t len[kSpans], cum[kSpans + 1], ucum[kSpans + 1];
  Span span[kSpans];
  uint32_t bits[kBitWords];  // the step's spike bitmap (networks it fits)
};

// ---- short-term plasticity (code/EqsGnl2.cpp:1048-1090) ------------------
__device__ __forceinline__ void plasticity(const CompatDev &d, uint32_t i, bool spk) {
  if (d.glob & FS_ACT_STP) {
    float Dv = d.D[i], Fv = d.F[i], Cp = d.Cap[i], Cr = d.Car[i];
    if (spk) {
      Cr = Cr + d.stp_aCar[i];
      Cp = Cp + d.stp_aCap[i];
      Fv = Fv + (Cp + Cr) * (1.0f - Fv) * d.stp_aF[i];
      Dv = Dv * (1.0f - d.stp_pv[i] * Fv);
    } else {
      Cr = d.stp_dfCar[i] * Cr + d.stp_efCar[i];
      Cp = d.stp_dfCap[i] * Cp;
      Fv = d.stp_dfF[i] * Fv + d.stp_efF[i] * (Cp + Cr) * (1.0f - Fv) * d.stp_aF[i];
      Dv = d.stp_dfD[i] * Dv + d.stp_efD[i];
    }
    d.D[i] = Dv; d.F[i] = Fv; d.Cap[i] = Cp; d.Car[i] = Cr;
  } else {
    if (spk) d.D[i] = d.D[i] * (1.0f - d.stp_pv[i]);
    else d.D[i] = d.stp_dfD[i] * d.D[i] + d.stp_efD[i];
  }
}

// ---- Activation ---------------------------------------------------------
// Neuron i = tile neuron q, step s of the launch, its random words from
// `base` on in the ring of len words; inc: what its gates take on a spike of
// this step, from D and F before the step's plasticity (x: single-target
// records and linear group gates, y: NMDA group gates).  Parameters and state
// are the tile's words in shared memory: read from global memory with the
// state stored between the loads, the receptors' loads waited for one another
// (11,000 cycles a step; L1 keeps nothing across the step's barrier).
// Returns whether it spiked.
__device__ __forceinline__ bool activate(const CompatDev &d, CompatSmem &B, uint32_t s, uint32_t i, uint32_t q,
                                         const uint32_t *ring, uint32_t base, uint32_t len, float2 &inc) {
  const uint32_t n = d.n;
  auto P = [&](int k) { return __uint_as_float(B.par[k][q]); };
  auto S = [&](int k) { return __uint_as_float(B.st[k][q]); };
  auto set = [&](int k, float v) { B.st[k][q] = __float_as_uint(v); };
  const uint32_t a = B.par[CP_ACT][q];
  uint32_t word[FS_NREC];
  {
    uint32_t pos = base + B.par[CP_DRAWOFF][q];
    pos = pos >= len ? pos - len : pos;
#pragma unroll
    for (int k = 0; k < FS_NREC; k++) {
      word[k] = ring[pos];
      pos = pos + 1 == len ? 0u : pos + 1;
    }
  }
  float g[FS_NREC];
#pragma unroll
  for (int r = 0; r < FS_NREC; r++) g[r] = S(CS_G + r);
  float isyn = S(CS_ISYN);
  // BgInit (code/EqsGnl2.cpp:284-337): one draw per enabled receptor
  int k = 0;
  auto draw = [&]() {
    const uint32_t w = k == 0 ? word[0] : k == 1 ? word[1] : k == 2 ? word[2] : k == 3 ? word[3] : word[4];
    k++;
    return u01(mt_temper(w));
  };
  const uint32_t bits[4] = {FS_ACT_AMPA, FS_ACT_GABA, FS_ACT_ACH, FS_ACT_GCL};
#pragma unroll
  for (int r = 0; r < 4; r++) {
    if (a & bits[r]) {
      const float u = draw();
      float st = S(CS_EST + r);
      if (P(CP_PB + r) > u) st = st + 1.0f;
      else st = st * P(CP_DFST + r);
      set(CS_EST + r, st);
      g[r] = g[r] + P(CP_EXTG + r) * st;
    }
  }
  if (a & FS_ACT_NMDA) {
    const float u = draw();
    float xt = S(CS_EXT), st = S(CS_ESTN);
    if (P(CP_PB + FS_NMDA) > u) xt = xt + 1.0f;
    else xt = xt * P(CP_NDFXT);
    st = P(CP_DFST + FS_NMDA) * st + P(CP_NEFST) * P(CP_NAS) * xt * (1.0f - st);
    set(CS_EXT, xt);
    set(CS_ESTN, st);
    g[FS_NMDA] = g[FS_NMDA] + P(CP_EXTG + FS_NMDA) * st;
  }
  if (a & FS_ACT_INJ) {
    const uint32_t j = s * d.inj_per_step + B.par[CP_INJOFF][q] + 1u;
    uint32_t jsr = jcong_jump(d.jcong_base, j);
    isyn = isyn + (P(CP_IMEAN) + P(CP_ISTD) * zig_nor(jsr, d));
  }
  // VmEul (code/EqsGnl2.cpp:152-225)
  float V = S(CS_V);
  int32_t cnt = (int32_t)B.st[CS_COUNT][q];
  uint32_t ns = B.st[CS_NS][q];
  const int32_t rf = (int32_t)B.par[CP_RF][q], sd = (int32_t)B.par[CP_SD][q];
  const float vreset = P(CP_VRESET);
  if (ns & FS_NS_FIRE) {
    firing(V, cnt, ns, rf, sd, vreset);
  } else {
    const float v = V;
    float Ir[5];
    Ir[0] = g[FS_AMPA] * (P(CP_VREV + FS_AMPA) - v);
    Ir[1] = g[FS_GABA] * (P(CP_VREV + FS_GABA) - v);
    Ir[2] = g[FS_NMDA] * (P(CP_VREV + FS_NMDA) - v) / (1.0f + P(CP_NMG) * expf_ref(-0.062f * v, d) / 3.57f);
    Ir[3] = g[FS_ACH] * (P(CP_VREV + FS_ACH) - v);
    Ir[4] = g[FS_GCL] * (P(CP_VREV + FS_GCL) - v);
    float I = Ir[0] + Ir[1] + Ir[2] + Ir[3] + Ir[4] + isyn * 1e3f + P(CP_GL) * P(CP_EL) * 1e3f;
    I = 1e-3f * I / P(CP_CM);
    const float dv = P(CP_DVMAX);
    if (I > dv) {
      I = dv;
      ns |= FS_NS_MEMDV_OVF;
      ns &= ~FS_NS_MEMDV_UDF;
    } else if (I < -dv) {
      I = -dv;
      ns &= ~FS_NS_MEMDV_OVF;
      ns |= FS_NS_MEMDV_UDF;
    } else {
      ns &= ~(FS_NS_MEMDV_OVF | FS_NS_MEMDV_UDF);
    }
    V = P(CP_DF) * v + P(CP_EF) * I;
#pragma unroll
    for (int r = 0; r < 5; r++) set(CS_IREP + r, Ir[r]);
    if (V > P(CP_VTH)) {
      ns |= FS_NS_FIRE;
      firing(V, cnt, ns, rf, sd, vreset);
      if (a & FS_ACT_LTP) ns |= FS_NS_LP_FIRE;
    }
  }
  if (a & FS_ACT_LTP) {  // firLP + ltpEul (code/EqsGnl2.cpp:254-280)
    int32_t clp = (int32_t)B.st[CS_CLP][q];
    if (ns & FS_NS_LP_FIRE) {
      if (clp == (int32_t)B.par[CP_SPILP][q]) {
        ns |= FS_NS_LP_SPIKE;
        ns &= ~FS_NS_LP_FIRE;
        clp = 0;
      } else {
        ns &= ~FS_NS_LP_SPIKE;
        clp++;
      }
    } else {
      ns &= ~FS_NS_LP_SPIKE;
    }
    B.st[CS_CLP][q] = (uint32_t)clp;
    set(CS_LP, (ns & FS_NS_LP_SPIKE) ? S(CS_LP) + 1.0f : P(CP_DFLP) * S(CS_LP));
  }
  // copies by step parity: what other blocks read of this step while their
  // owners advance the next
  const size_t o2 = (size_t)(s & 1u) * n + i;
  if (d.LP2) d.LP2[o2] = S(CS_LP);
  if (d.V2) d.V2[o2] = V;
  set(CS_V, V);
  B.st[CS_COUNT][q] = (uint32_t)cnt;
  B.st[CS_NS][q] = ns;
#pragma unroll
  for (int r = 0; r < FS_NREC; r++) set(CS_G + r, 0.0f);
  set(CS_ISYN, 0.0f);
  const bool spk = (ns & FS_NS_SPIKE) != 0;
  if (d.outV) d.outV[(size_t)s * n + i] = V;
  if (d.outNS) d.outNS[(size_t)s * n + i] = ns;
  if (d.outIrep)
#pragma unroll
    for (int r = 0; r < 5; r++) d.outIrep[(size_t)s * FS_NREC * n + (size_t)r * n + i] = S(CS_IREP + r);
  inc = make_float2(1.0f, 1.0f);
  if (d.glob & (FS_ACT_STP | FS_ACT_STD)) {
    const float D = d.D[i], DF = D * d.F[i];
    inc = (d.glob & FS_ACT_STP) ? make_float2(DF, DF) : make_float2(D, DF);
    d.inc2[(size_t)(s & 1u) * n + i] = inc.x;
    plasticity(d, i, spk);
  }
  return spk;
}

// The tile's words from and to global memory.
__device__ __forceinline__ void tile_load(const CompatDev &d, CompatSmem &B, uint32_t p0, uint32_t np) {
  const uint32_t q = threadIdx.x % kCompatTile;
  if (q >= np) return;
  for (uint32_t f = threadIdx.x / kCompatTile; f < CP_N + CS_N; f += kCT / kCompatTile) {
    if (f < CP_N) B.par[f][q] = __ldg(d.npar[f] + p0 + q);
    else B.st[f - CP_N][q] = __ldcg(d.nst[f - CP_N] + p0 + q);
  }
}
__device__ __forceinline__ void tile_store(const CompatDev &d, const CompatSmem &B, uint32_t p0, uint32_t np) {
  const uint32_t q = threadIdx.x % kCompatTile;
  if (q >= np) return;
  for (uint32_t f = threadIdx.x / kCompatTile; f < CS_N; f += kCT / kCompatTile) d.nst[f][p0 + q] = B.st[f][q];
}

// ---- group gates of a tile's neurons --------------------------------------
// The gates of presynaptic neurons [p0, p1) (gby: gates by presynaptic
// neuron, over all receptors' gates), advanced from the buffer of the step
// before into this step's: their posts' blocks still read the former.
__device__ __forceinline__ void tile_gates(const CompatDev &d, uint32_t p0, uint32_t p1, uint32_t par,
                                           const bool *spk, const float2 *inc) {
  if (!d.gby_row) return;
  const uint32_t n = d.n, e1 = d.gby_row[p1];
  for (uint32_t e = d.gby_row[p0] + threadIdx.x; e < e1; e += kCT) {
    const uint32_t ent = d.gby_ent[e];
    uint32_t r = 0;
#pragma unroll
    for (uint32_t q = 1; q < FS_NREC; q++)
      if (ent >= d.gate_off[q]) r = q;
    const uint32_t k = ent - d.gate_off[r];
    const RecDev &R = d.R[r];
    const uint32_t q = R.gate_pre[k] - p0, t0 = R.gate_post0[k];
    const size_t from = (size_t)(par ^ 1u) * R.n_gates + k, to = (size_t)par * R.n_gates + k;
    float st = R.gate_st[from];
    if (r != FS_NMDA) {
      st = spk[q] ? st + inc[q].x : st * d.dfst[(size_t)r * n + t0];
    } else {
      float xt = R.gate_xt[k];
      xt = spk[q] ? xt + inc[q].y : xt * d.nmda_dfxt[t0];
      st = d.dfst[(size_t)r * n + t0] * st + d.nmda_efst[t0] * d.nmda_as[t0] * xt * (1.0f - st);
      R.gate_xt[k] = xt;
    }
    R.gate_st[to] = st;
  }
}

// ---- a tile's synaptic terms ----------------------------------------------
// The tile's gather entries and records, receptor by receptor (gather before
// records, each by post), form one sequence of items; span j = 2r (gather) or
// 2r + 1 (records) holds items [cum[j], cum[j + 1]), those of tile post q at
// [off[j][q], off[j][q + 1]).  Work units of at most kUnit items, each within
// a span: units [ucum[j], ucum[j + 1]).
__device__ __forceinline__ void tile_items(const CompatDev &d, CompatSmem &B, uint32_t p0, uint32_t np) {
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < kSpans * (np + 1); i += kCT) {
    const uint32_t j = i / (np + 1), q = i - j * (np + 1);
    const uint32_t *row = (j & 1u) ? d.R[j >> 1].rrow : d.R[j >> 1].grow;
    const uint32_t f = row ? __ldg(row + p0) : 0u, e = row ? __ldg(row + p0 + q) - f : 0u;
    B.off[j][q] = e;
    if (q == 0) {
      const RecDev &R = d.R[j >> 1];
      B.span[j] = (j & 1u) ? Span{R.rpre + f, R.rpost + f, R.rloc + f, R.rst + f, R.rxt + f, R.rg + f, 0u}
                           : Span{R.ggate + f, nullptr, nullptr, R.gate_st, R.gate_xt, (float *)R.gate_g, R.n_gates};
    }
    if (q == np) B.len[j] = e;
  }
  __syncthreads();
  if (tid == 0) {
    uint32_t c = 0, u = 0;
    for (int j = 0; j < kSpans; j++) {
      B.cum[j] = c;
      B.ucum[j] = u;
      c += B.len[j];
      u += (B.len[j] + kUnit - 1) / kUnit;
    }
    B.cum[kSpans] = c;
    B.ucum[kSpans] = u;
  }
  __syncthreads();
  for (uint32_t i = tid; i < kSpans * (np + 1); i += kCT) {
    const uint32_t j = i / (np + 1), q = i - j * (np + 1);
    B.off[j][q] += B.cum[j];
  }
  __syncthreads();
}

__device__ __forceinline__ bool spiked(const uint32_t *bits, uint32_t i) { return (bits[i >> 5] >> (i & 31u)) & 1u; }

// The terms of unit u into terms[item - c0], four items in flight a lane.  The
// item streams pass by L1 (each is read once a step).  Records advance here
// (nobody else reads them); kLTP: the weight's long-term plasticity after its
// term.
template <bool kLTP>
__device__ __forceinline__ void unit_terms(const CompatDev &d, CompatSmem &B, uint32_t u, uint32_t lane, uint32_t s,
                                           uint32_t par, uint32_t c0, const uint32_t *bits) {
  uint32_t j = 0;
#pragma unroll
  for (int q = 1; q < kSpans; q++)
    if (u >= B.ucum[q]) j = q;
  const uint32_t done = (u - B.ucum[j]) * kUnit, cnt = min(kUnit, B.len[j] - done), r = j >> 1, n = d.n;
  float *out = B.terms + (B.cum[j] + done - c0);
  const Span &P = B.span[j];
  uint32_t k[4];
#pragma unroll
  for (int v = 0; v < 4; v++) k[v] = lane + 32u * v < cnt ? __ldcg(P.k + done + lane + 32u * v) : 0u;
  if (!(j & 1u)) {
    const float *st = P.st + (size_t)par * P.n_gates;
    float a[4], g[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
      a[v] = lane + 32u * v < cnt ? st[k[v]] : 0.0f;
      g[v] = lane + 32u * v < cnt ? __ldg(P.g + k[v]) : 0.0f;
    }
#pragma unroll
    for (int v = 0; v < 4; v++)
      if (lane + 32u * v < cnt) out[lane + 32u * v] = a[v] * g[v];
    return;
  }
  const bool nm = r == FS_NMDA, plastic = (d.glob & (FS_ACT_STP | FS_ACT_STD)) != 0;
  float st[4], xt[4], g[4];
  uint32_t loc[4];
#pragma unroll
  for (int v = 0; v < 4; v++) {
    const uint32_t e = done + lane + 32u * v;
    const bool ok = lane + 32u * v < cnt;
    st[v] = ok ? __ldcg(P.st + e) : 0.0f;
    xt[v] = ok && nm ? __ldcg(P.xt + e) : 0.0f;
    g[v] = ok ? __ldcg(P.g + e) : 0.0f;
    loc[v] = ok ? __ldcg(P.loc + e) : 0u;
  }
#pragma unroll
  for (int v = 0; v < 4; v++) {
    const uint32_t e = done + lane + 32u * v, q = loc[v];
    if (lane + 32u * v >= cnt) break;
    const bool spk = spiked(bits, k[v]);
    const float inc = (spk && plastic) ? d.inc2[(size_t)(s & 1u) * n + k[v]] : 1.0f;
    const float dfp = __uint_as_float(B.par[CP_DFST + r][q]);
    if (!nm) {
      st[v] = spk ? st[v] + inc : st[v] * dfp;
    } else {
      xt[v] = spk ? xt[v] + inc : xt[v] * __uint_as_float(B.par[CP_NDFXT][q]);
      st[v] = dfp * st[v] +
              __uint_as_float(B.par[CP_NEFST][q]) * __uint_as_float(B.par[CP_NAS][q]) * xt[v] * (1.0f - st[v]);
      __stcg(P.xt + e, xt[v]);
    }
    __stcg(P.st + e, st[v]);
    out[lane + 32u * v] = st[v] * g[v];
    if (kLTP) {  // code/EqsGnl2.cpp:1005-1044
      const uint32_t pre = k[v], post = __ldcg(P.post + e);
      const bool pspk = spiked(bits, post);
      if (spk || pspk) {
        const float *LP = d.LP2 + (size_t)(s & 1u) * n;
        float w = g[v];
        if (spk) {
          const float ni = d.ltp_Neg[pre];
          if (ni > 0) w = w + LP[post] * ni;
          else w = w * (1.0f + LP[post] * ni);
        }
        if (pspk) {
          const float pi = d.ltp_Pos[pre];
          if (pi > 0) w = w + LP[pre] * pi;
          else w = w * (1.0f + LP[pre] * pi);
        }
        __stcg(P.g + e, w);
      }
    }
  }
}

// acc plus the terms of items [a, b) of the pass [c0, c1), in order (the next
// eight in flight while eight are added).
__device__ __forceinline__ float ordered_sum(float acc, const float *terms, uint32_t a, uint32_t b, uint32_t c0,
                                             uint32_t c1) {
  uint32_t i = max(a, c0);
  const uint32_t hi = min(b, c1);
  const float *t = terms - c0;
  float v[8], w[8];
  if (i + 8 <= hi)
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = t[i + k];
  while (i + 8 <= hi) {
    i += 8;
    if (i + 8 <= hi)
#pragma unroll
      for (int k = 0; k < 8; k++) w[k] = t[i + k];
#pragma unroll
    for (int k = 0; k < 8; k++) acc = acc + v[k];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = w[k];
  }
  for (; i < hi; i++) acc = acc + t[i];
  return acc;
}

// The synaptic phase of a tile: its posts' G (and Isyn of the gap junctions)
// for the next step, into the tile's state (own) or global memory.
template <bool kLTP>
__device__ __forceinline__ void tile_synapses(const CompatDev &d, CompatSmem &B, uint32_t p0, uint32_t np, uint32_t s,
                                              uint32_t par, bool own, const uint32_t *bits) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, n = d.n;
  constexpr uint32_t kW = kCT / 32;
  const uint32_t units = B.ucum[kSpans], sums = FS_NREC * ((np + 31u) / 32u);
  float acc[2] = {0.0f, 0.0f};
  for (uint32_t u0 = 0, c0 = 0; u0 < units; u0 += kPassUnits) {
    const uint32_t u1 = min(units, u0 + kPassUnits);
    uint32_t c1 = B.cum[kSpans];
    if (u1 < units) {
      uint32_t j = 0;
      for (int q = 1; q < kSpans; q++)
        if (u1 >= B.ucum[q]) j = q;
      c1 = B.cum[j] + (u1 - B.ucum[j]) * kUnit;
    }
    for (uint32_t u = u0 + warp; u < u1; u += kW) unit_terms<kLTP>(d, B, u, lane, s, par, c0, bits);
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < 2; k++) {
      const uint32_t w = warp + k * kW, r = w % FS_NREC, q = w / FS_NREC * 32u + lane;
      if (w < sums && q < np) {
        acc[k] = ordered_sum(acc[k], B.terms, B.off[2 * r][q], B.off[2 * r][q + 1], c0, c1);
        acc[k] = ordered_sum(acc[k], B.terms, B.off[2 * r + 1][q], B.off[2 * r + 1][q + 1], c0, c1);
      }
    }
    __syncthreads();
    c0 = c1;
  }
#pragma unroll
  for (uint32_t k = 0; k < 2; k++) {
    const uint32_t w = warp + k * kW, r = w % FS_NREC, q = w / FS_NREC * 32u + lane;
    if (w < sums && q < np) {
      if (own) B.st[CS_G + r][q] = __float_as_uint(acc[k]);
      else d.nst[CS_G + r][p0 + q] = __float_as_uint(acc[k]);
    }
  }
  if (d.gap_row)
    for (uint32_t q = threadIdx.x; q < np; q += kCT) {
      const float *V = d.V2 + (size_t)(s & 1u) * n;
      const uint32_t p = p0 + q;
      const float vp = V[p];
      float a = 0.0f;
      for (uint32_t e = d.gap_row[p], e1 = d.gap_row[p + 1]; e < e1; e++) a = a + d.gap_g[e] * (V[d.gap_other[e]] - vp);
      if (own) B.st[CS_ISYN][q] = __float_as_uint(a);
      else d.nst[CS_ISYN][p] = __float_as_uint(a);
    }
}

// GatingVariable columns of step s (records of every tile; between two grid
// barriers).
__device__ __forceinline__ void gv_snapshot(const CompatDev &d, uint32_t s, uint32_t first, uint32_t stride) {
  for (uint32_t q = first; q < d.gv_n; q += stride) {
    const uint32_t code = d.gv_sel[q], r = code >> 28, e = code & 0x0fffffffu;
    d.gv_st[(size_t)s * d.gv_n + q] = __ldcg(d.R[r].rst + e);
    d.gv_xt[(size_t)s * d.gv_n + q] = __ldcg(d.R[r].rxt + e);
  }
}

// ---- VarInit (code/EqsGnl2.cpp:339-401) -----------------------------------
// Group gates are not reset here, as in the reference (they are zeroed only
// when the network is built).
__global__ void __launch_bounds__(256) k_varinit(const __grid_constant__ CompatDev d) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t n = d.n;
  if (t < n) {
    const uint32_t i = t, a = d.act[i];
    d.Isyn[i] = 0.0f;
    d.V[i] = -70.0f;
    d.Count[i] = 0;
    d.NS[i] = 0u;
    if (a & FS_ACT_STP) {
      d.D[i] = 1.0f; d.F[i] = 1.0f; d.Cap[i] = 0.0f; d.Car[i] = 20.0f;
    } else if (a & FS_ACT_STD) {
      d.D[i] = 1.0f;
    }
    if (a & FS_ACT_LTP) { d.LP[i] = 0.0f; d.CountLP[i] = 0; }
#pragma unroll
    for (int r = 0; r < FS_NREC; r++) {
      d.G[(size_t)r * n + i] = 0.0f;
      d.Irep[(size_t)r * n + i] = 0.0f;
    }
#pragma unroll
    for (int r = 0; r < 4; r++) d.ext_st[(size_t)r * n + i] = 0.0f;
    d.ext_xt_n[i] = 0.0f;
    d.ext_st_n[i] = 0.0f;
  }
  if (t < d.rec_off[FS_NREC]) {
    int r = 0;
#pragma unroll
    for (int q = 1; q < FS_NREC; q++)
      if (t >= d.rec_off[q]) r = q;
    const RecDev &R = d.R[r];
    const uint32_t e = t - d.rec_off[r];
    R.rst[e] = 0.0f;
    R.rxt[e] = 0.0f;
  }
}

cudaError_t compat_varinit(const CompatDev &d, cudaStream_t st) {
  const uint64_t work = d.n > d.rec_off[FS_NREC] ? d.n : d.rec_off[FS_NREC];
  if (work == 0) return cudaSuccess;
  k_varinit<<<(unsigned)((work + 255) / 256), 256, 0, st>>>(d);
  return cudaGetLastError();
}

// ---- mt19937 stream -------------------------------------------------------
// Generator of one block.  The recurrence is that of mt_twist; word k of the
// next 624 needs the new word k - 227 when k >= 227, so thread t < 227 makes
// words t, t + 227 and t + 454 one after the other, from old words only: one
// block barrier and at most three twists a thread for 624 words (370 cycles
// on an SM of its own; three dependent waves with a barrier each took 660).  The raw words go
// to a ring of nb blocks that the activations read and temper.
struct MtBlock {
  uint32_t (*buf)[624];  // buf[cur]: the last block
  uint32_t cur;
  uint32_t blk;          // its place in the ring
  uint64_t have;         // stream words in the ring, counted from its first block
  __device__ __forceinline__ void draw(uint32_t *ring, uint32_t nb, uint64_t need) {
    const uint32_t t = threadIdx.x;
    while (have < need) {
      const uint32_t *o = buf[cur];
      uint32_t *w = buf[cur ^ 1];
      blk = blk + 1 == nb ? 0u : blk + 1;
      uint32_t *out = ring + (size_t)blk * 624;
      if (t < 227) {
        const uint32_t w0 = o[t + 397] ^ mt_twist(o[t], o[t + 1]);
        const uint32_t w1 = w0 ^ mt_twist(o[t + 227], o[t + 228]);
        w[t] = w0;
        w[t + 227] = w1;
        out[t] = w0;
        out[t + 227] = w1;
        if (t < 170) {
          // word 623 is followed by the new word 0
          const uint32_t nx = t == 169 ? o[397] ^ mt_twist(o[0], o[1]) : o[t + 455];
          const uint32_t w2 = w1 ^ mt_twist(o[t + 454], nx);
          w[t + 454] = w2;
          out[t + 454] = w2;
        }
      }
      __syncthreads();
      cur ^= 1;
      have += 624;
    }
  }
};

// ---- the steps of a call ----------------------------------------------------
// One persistent launch: the last block draws the random stream, one step
// ahead of the others; every other block owns tiles of posts.  Step s: (A)
// activate the own neurons, advance the gates they are presynaptic to, set
// their bits of the step's spike bitmap; a grid barrier; (B) the tile's
// synaptic terms and ordered sums, for the next step.  What (B) reads from
// other blocks (spikes, gates, plasticity increments, LP, V of gap junctions)
// is kept by step parity, so the owners' next (A) does not disturb it and one
// barrier a step suffices.  Records are read and written by their post's
// block only.  A block
// with one tile (up to 28,352 neurons: 443 blocks of 64) keeps its neurons in shared memory for
// the launch; with more it loads and stores them every step.
//
// A step moves every record once through L2 (17 B a linear, 25 B an NMDA
// record); the three launches before this kernel walked a post's records with
// one warp and added its terms through a chain of warp shuffles, searched
// the expf exceptions in 18 dependent loads, and drew the stream in a launch
// of its own.
// Measured: 20,000 neurons with 4.1 M records 106 -> 42 us a step, now bounded by
// the random stream (160 blocks of 624 words a step, about 480 cycles each
// next to two other blocks of its SM); the two-population network of 1,000
// neurons 30 -> 9.7 us, latencies one after the other (activation 5,700
// cycles, barrier 3,500, terms 4,500, ordered sums 3,800).  Three blocks an SM:
// four spill (64 registers), and the spills and the tile leave L1 too little.
template <bool kLTP>
__global__ void __launch_bounds__(kCT, 3) k_compat(const __grid_constant__ CompatDev d,
                                                   const __grid_constant__ CompatRun R) {
  extern __shared__ __align__(16) unsigned char smc[];
  CompatSmem &B = *(CompatSmem *)smc;
  unsigned long long target = 0;
  const uint32_t tid = threadIdx.x, nblk = gridDim.x - 1u;
  const uint32_t D = d.draws_per_step, pos0 = *R.mt_pos, ring_len = R.ring_blocks * 624u;
  if (blockIdx.x == nblk) {  // the random stream
    uint32_t(*buf)[624] = (uint32_t(*)[624])B.terms;
    for (uint32_t k = tid; k < 624; k += kCT) R.ring[k] = buf[0][k] = R.mt_state[k];
    MtBlock mt{buf, 0u, 0u, 624u};
    __syncthreads();
    mt.draw(R.ring, R.ring_blocks, pos0 + D);
    if (!grid_sync(R.bar, d.err, gridDim.x, target)) return;
    for (uint32_t s = 0; s < R.nsteps; s++) {
      if (s + 1 < R.nsteps) mt.draw(R.ring, R.ring_blocks, pos0 + (uint64_t)(s + 2) * D);
      if (!grid_sync(R.bar, d.err, gridDim.x, target)) return;
      if (d.gv_n && !grid_sync(R.bar, d.err, gridDim.x, target)) return;
    }
    for (uint32_t k = tid; k < 624; k += kCT) R.mt_state[k] = mt.buf[mt.cur][k];
    if (tid == 0) *R.mt_pos = (uint32_t)(pos0 + (uint64_t)R.nsteps * D - (mt.have - 624u));
    return;
  }
  const bool own = R.tiles <= nblk;  // the block's one tile stays in shared memory
  uint32_t p0 = 0, np = 0;
  auto enter = [&](uint32_t t) {
    p0 = __ldg(R.tile_post + t);
    np = __ldg(R.tile_post + t + 1) - p0;
  };
  if (own) {
    enter(blockIdx.x);
    tile_load(d, B, p0, np);
    tile_items(d, B, p0, np);
  }
  if (!grid_sync(R.bar, d.err, gridDim.x, target)) return;
  for (uint32_t s = 0; s < R.nsteps; s++) {
    const uint32_t par = (R.gpar + s) & 1u;
    const uint32_t base = (uint32_t)((pos0 + (uint64_t)s * D) % ring_len);
    for (uint32_t t = blockIdx.x; t < R.tiles; t += nblk) {
      if (!own) {
        enter(t);
        tile_load(d, B, p0, np);
        __syncthreads();
      }
      for (uint32_t q = tid; q < np; q += kCT) {
        float2 inc;
        const bool spk = activate(d, B, s, p0 + q, q, R.ring, base, ring_len, inc);
        B.inc[q] = inc;
        B.spk[q] = spk;
        if (spk) atomicOr(d.spikebits + (size_t)s * d.words + ((p0 + q) >> 5), 1u << ((p0 + q) & 31u));
      }
      if (d.gby_row || !own) __syncthreads();
      if (d.gby_row) tile_gates(d, p0, p0 + np, par, B.spk, B.inc);
      if (!own) {
        tile_store(d, B, p0, np);
        __syncthreads();
      }
    }
    if (!grid_sync(R.bar, d.err, gridDim.x, target)) return;
    const uint32_t *bits = d.spikebits + (size_t)s * d.words;
    if (d.words <= kBitWords) {
      for (uint32_t w = tid; w < d.words; w += kCT) B.bits[w] = __ldcg(bits + w);
      bits = B.bits;
      __syncthreads();
    }
    for (uint32_t t = blockIdx.x; t < R.tiles; t += nblk) {
      if (!own) {
        enter(t);
        tile_load(d, B, p0, np);
        tile_items(d, B, p0, np);
      }
      tile_synapses<kLTP>(d, B, p0, np, s, par, own, bits);
    }
    if (d.gv_n) {
      if (!grid_sync(R.bar, d.err, gridDim.x, target)) return;
      gv_snapshot(d, s, blockIdx.x * kCT + tid, nblk * kCT);
    }
    __syncthreads();  // the tiles' G before the next step reads it
  }
  if (own) tile_store(d, B, p0, np);
}

static const void *compat_kernel(bool ltp) {
  return ltp ? (const void *)k_compat<true> : (const void *)k_compat<false>;
}

// Blocks of k_compat that are resident at once, the random stream's not counted.
cudaError_t compat_blocks(uint32_t sm_count, uint32_t *blocks) {
  int occ = 0;
  for (int ltp = 0; ltp < 2; ltp++) {
    const void *k = compat_kernel(ltp != 0);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CompatSmem));
    int o = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k, (int)kCT, sizeof(CompatSmem));
    if (e != cudaSuccess) return e;
    occ = ltp ? (o < occ ? o : occ) : o;
  }
  *blocks = sm_count * (uint32_t)(occ > 0 ? occ : 1) - 1u;
  return cudaSuccess;
}

cudaError_t compat_steps(const CompatDev &d, CompatRun R, cudaStream_t st, uint64_t *launches) {
  if (R.nsteps == 0) return cudaSuccess;
  R.ring_blocks = 2u * d.draws_per_step / 624u + 3u;
  CompatDev dd = d;
  void *args[] = {&dd, &R};
  cudaError_t e = cudaMemsetAsync(R.bar, 0, 8, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(d.spikebits, 0, (size_t)R.nsteps * d.words * 4, st);
  if (e == cudaSuccess)
    e = cudaLaunchCooperativeKernel(compat_kernel((d.glob & FS_ACT_LTP) && d.rec_off[FS_NREC]), R.blocks + 1u, kCT,
                                    args, sizeof(CompatSmem), st);
  if (launches) *launches += 1;
  return e;
}

// ---- ordered spike compaction ----------------------------------------------
// bits[s][w] are the warp ballots of step s.  k_count: one block per step sums
// the population counts.  k_write: one block per step computes a block-wide
// exclusive prefix of per-word counts and writes ascending neuron ids.
__global__ void __launch_bounds__(256) k_count(const uint32_t *bits, uint32_t words, uint32_t *counts) {
  const uint32_t s = blockIdx.x;
  uint32_t c = 0;
  for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) c += __popc(bits[(size_t)s * words + w]);
  for (int o = 16; o; o >>= 1) c += __shfl_down_sync(kFull, c, o);
  __shared__ uint32_t part[8];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t tot = 0;
    for (int k = 0; k < 8; k++) tot += part[k];
    counts[s] = tot;
  }
}
__global__ void k_scan_counts(const uint32_t *counts, uint32_t nsteps, uint32_t *offsets) {
  // single block, sequential over chunks of 1024
  __shared__ uint32_t sh[1024];
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t base = 0; base < nsteps; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = (i < nsteps) ? counts[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (uint32_t o = 1; o < 1024; o <<= 1) {
      const uint32_t a = (threadIdx.x >= o) ? sh[threadIdx.x - o] : 0;
      __syncthreads();
      sh[threadIdx.x] += a;
      __syncthreads();
    }
    if (i < nsteps) offsets[i] = carry + sh[threadIdx.x] - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += sh[1023];
    __syncthreads();
  }
  if (threadIdx.x == 0) offsets[nsteps] = carry;
}
__global__ void __launch_bounds__(256) k_write(const uint32_t *bits, uint32_t words, const uint32_t *offsets,
                                               uint32_t *idx) {
  const uint32_t s = blockIdx.x;
  __shared__ uint32_t warp_tot[8];
  __shared__ uint32_t run;
  if (threadIdx.x == 0) run = offsets[s];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (uint32_t base = 0; base < words; base += blockDim.x) {
    const uint32_t w = base + threadIdx.x;
    const uint32_t b = (w < words) ? bits[(size_t)s * words + w] : 0u;
    const uint32_t c = __popc(b);
    // warp inclusive scan of c
    uint32_t x = c;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t k = 0; k < wid; k++) before += warp_tot[k];
    uint32_t o0 = run + before + x - c;
    uint32_t bb = b;
    while (bb) {
      const int bit = __ffs(bb) - 1;
      idx[o0++] = w * 32u + (uint32_t)bit;
      bb &= bb - 1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t tot = 0;
      for (int k = 0; k < 8; k++) tot += warp_tot[k];
      run += tot;
    }
    __syncthreads();
  }
}

cudaError_t spikes_compact(const uint32_t *bits, uint32_t nsteps, uint32_t words, uint32_t *counts,
                           uint32_t *offsets, uint32_t *idx, cudaStream_t st, uint64_t *launches) {
  if (nsteps == 0) return cudaSuccess;
  k_count<<<nsteps, 256, 0, st>>>(bits, words, counts);
  k_scan_counts<<<1, 1024, 0, st>>>(counts, nsteps, offsets);
  k_write<<<nsteps, 256, 0, st>>>(bits, words, offsets, idx);
  if (launches) *launches += 3;
  return cudaGetLastError();
}

void compat_set_tables(const uint32_t kn[128], const float fn[128], const float wn[128],
                       const uint32_t jump_a[32], const uint32_t jump_c[32], cudaStream_t st) {
  cudaMemcpyToSymbolAsync(c_kn, kn, sizeof(uint32_t) * 128, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c_fn, fn, sizeof(float) * 128, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c_wn, wn, sizeof(float) * 128, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c_jump_a, jump_a, sizeof(uint32_t) * 32, 0, cudaMemcpyHostToDevice, st);
  cudaMemcpyToSymbolAsync(c_jump_c, jump_c, sizeof(uint32_t) * 32, 0, cudaMemcpyHostToDevice, st);
}

// test hook: the device expf used by the NMDA Mg block
__global__ void k_expf_eval(const float *x, float *y, uint64_t k, const uint32_t *keys, const float *vals,
                            uint32_t nk, const uint4 *tab) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k) return;
  CompatDev d{};
  d.expf_keys = keys;
  d.expf_vals = vals;
  d.expf_n = nk;
  d.expf_tab = tab;
  y[i] = expf_ref(x[i], d);
}
cudaError_t expf_ref_eval(const float *x, float *y, uint64_t k, const uint32_t *keys, const float *vals,
                          uint32_t nk, const uint4 *tab, cudaStream_t st) {
  if (k == 0) return cudaSuccess;
  k_expf_eval<<<(unsigned)((k + 255) / 256), 256, 0, st>>>(x, y, k, keys, vals, nk, tab);
  return cudaGetLastError();
}

}  // namespace fsd
