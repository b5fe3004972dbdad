// engine.cu -- the B200 engine: connectome build, bath producer, delivery,
// LIFCA update, spike compaction and STDP, behind the C ABI of
// include/dpsnn_b200.h.
//
// Arithmetic follows the reference operation by operation (compiled with
// --fmad=false so no multiply-add is contracted, like the reference's
// x86-64 SSE2 build); the comments cite the reference lines each kernel
// restates.  Data layout in HBM (N neurons, S synapses, D delays):
//   neuron state  SoA fp64 v, c, Tr, Te, nextBath (5*8 B/neuron)
//   connectome    CSR sorted by (pre, delay, generation order):
//                 row_ptr[N+1] u64, sub_off[N*(D+1)] u16 (per-delay offsets
//                 inside a row), post[S] u32, w16[S] i16 (6 B/synapse);
//                 with STDP also tderiv[S] f32, last_act[S] i32
//   spike ring    80 slots x N: ids u32, te f64 (one slot per step)
//   events        per target neuron `cap` slots of {u32 key, f32 weight};
//                 overflow list of {target, key, weight}
//   bath          per rank: the last 256 ran3 draws; per step per-neuron
//                 event lists
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <dlfcn.h>
#include <string>
#include <mutex>
#include <vector>

#include "dd_math.cuh"
#include "dpsnn_internal.h"

#define RING_SLOTS 80          // DSD__maxD: axonal delay ring length
#define MAX_SYN_PER_NEURON 7500  // DSD__maxM (Makefile miniM)
#define MAX_INPUTS_PER_STEP 6000 // DSD__maxSimultaneousSpikesOnSameTarget
#define MBIG 1000000000
#define MSEED 161803398
#define NEURON_BLOCK 256
#define LOCAL_EVENTS 16        // per-thread event buffer of the neuron kernel
#define NEURON_BATCH 8         // event loads in flight per thread
#define DEFAULT_EVENT_CAP 1024 // per-target event slots per step (capped by memory)

// ------------------------------------------------------------------ errors
static thread_local char g_err[1024];
int dpsnn_fail(int code, const char *fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
  return code;
}
extern "C" const char *dpsnn_last_error(void) { return g_err; }

const char *dpsnn_library_dir(void) {
  // initialised once, thread-safely (engines may be created from several threads)
  static const std::string dir = [] {
    Dl_info info;
    if (dladdr((void *)&dpsnn_library_dir, &info) && info.dli_fname) {
      std::string d = info.dli_fname;
      size_t p = d.rfind('/');
      return (p == std::string::npos) ? std::string(".") : d.substr(0, p);
    }
    return std::string(".");
  }();
  return dir.c_str();
}

#define CK(x)                                                                       \
  do {                                                                              \
    cudaError_t e_ = (x);                                                           \
    if (e_ != cudaSuccess)                                                          \
      return dpsnn_fail(DPSNN_E_CUDA, "%s: %s", #x, cudaGetErrorString(e_));        \
  } while (0)

// Error flags raised by kernels (bit set in Dev::flags[0]).
enum {
  F_TIME_WINDOW = 1,     // event time outside [t, t+1)  (DPSNN_neuron_sim.c:681-685)
  F_NO_TARGET = 2,       // spiking neuron without targets (DPSNN_localNet_sim.c:732-737)
  F_OVERFLOW = 4,        // overflow list full
  F_TOO_MANY_INPUTS = 8, // > miniSimSpikes inputs on one neuron in one step
  F_BATH_DRAWS = 16,     // bath draw ring exhausted
  F_GEN = 32,            // synapse generation error (see gen error code)
};

// ------------------------------------------------------------------ model
struct NetConst {
  uint32_t N, locN, P, D, nsub, npcm, cfx, cfy, nmod, mods_per_rank;
  uint32_t stencil, max_mod, stencil_dim, delay_min, delay_max;
  uint32_t offset[DPSNN_MAX_SUBPOP], count[DPSNN_MAX_SUBPOP];
  double Tau[DPSNN_MAX_SUBPOP], Theta[DPSNN_MAX_SUBPOP], H[DPSNN_MAX_SUBPOP];
  double Tarp[DPSNN_MAX_SUBPOP], AlphaC[DPSNN_MAX_SUBPOP], TauC[DPSNN_MAX_SUBPOP];
  double gC[DPSNN_MAX_SUBPOP], NuExt[DPSNN_MAX_SUBPOP];
  double r_tau[DPSNN_MAX_SUBPOP], r_tauC[DPSNN_MAX_SUBPOP];   // 1/Tau, 1/TauC (div_by)
  double J[DPSNN_MAX_SUBPOP * DPSNN_MAX_SUBPOP], DJ[DPSNN_MAX_SUBPOP * DPSNN_MAX_SUBPOP];
  double DMin[DPSNN_MAX_SUBPOP * DPSNN_MAX_SUBPOP], DMax[DPSNN_MAX_SUBPOP * DPSNN_MAX_SUBPOP];
  float f2w, w2f, min_w;
  uint32_t global_seed, start_pl, stop_pl, stdp_on;
  float causal_tab[128], anti_tab[128];
  float stdp_drift, stdp_tauDecay;
  uint32_t ev_cap, ovf_cap;
  uint32_t light_max;   // neurons with more synaptic events take the heavy path
  uint32_t delay_exp;  // getRandomDelay_EXP instead of _UNI
  float inv_log_tn;    // (float)(1.0 / log(0.05)), the EXP tail constant
  const uint32_t *fix_keys, *fix_vals;   // the logf fix-up table, where the bath searches it
  uint32_t fix_n;
};

// ------------------------------------------------------------------ ran3
// Numerical Recipes ran3 with the reference's |mj| tweak and seeding rules
// (randdev.c:116-196, :477-502).  Same code on host and device.
struct Ran3 {
  int32_t ma[56];
  int32_t inext, inextp, iff, idum;
};

__host__ __device__ static inline double r3_rand(Ran3 &g) {
  int32_t mj, mk;
  if (g.idum < 0 || g.iff == 0) {
    g.iff = 1;
    mj = MSEED - (g.idum < 0 ? -g.idum : g.idum);
    mj = (mj < 0 ? -mj : mj);
    mj %= MBIG;
    g.ma[55] = mj;
    mk = 1;
    for (int i = 1; i <= 54; i++) {
      int ii = (21 * i) % 55;
      g.ma[ii] = mk;
      mk = mj - mk;
      if (mk < 0) mk += MBIG;
      mj = g.ma[ii];
    }
    for (int k = 1; k <= 4; k++)
      for (int i = 1; i <= 55; i++) {
        g.ma[i] -= g.ma[1 + (i + 30) % 55];
        if (g.ma[i] < 0) g.ma[i] += MBIG;
      }
    g.inext = 0;
    g.inextp = 31;
    g.idum = 1;
  }
  if (++g.inext == 56) g.inext = 1;
  if (++g.inextp == 56) g.inextp = 1;
  mj = g.ma[g.inext] - g.ma[g.inextp];
  if (mj < 0) mj += MBIG;
  g.ma[g.inext] = mj;
  return mj * (1.0 / (double)MBIG);
}
__host__ __device__ static inline void r3_seed(Ran3 &g, int32_t s) {
  g.idum = -s;
  (void)r3_rand(g);
}
// The last 55 outputs (oldest first): the whole state of the lagged
// Fibonacci recurrence x[n] = x[n-55] - x[n-24] (mod 1e9) that ran3 runs.
__host__ __device__ static inline void r3_history(const Ran3 &g, uint32_t *hist55) {
  int k = 0;
  for (int i = g.inext + 1; i <= 55; i++) hist55[k++] = (uint32_t)g.ma[i];
  for (int i = 1; i <= g.inext; i++) hist55[k++] = (uint32_t)g.ma[i];
}

struct NormState {
  int32_t set;
  double cache;
};
// NormDev: polar Box-Muller with a one-value cache (randdev.c:584-606).
__device__ static inline double normdev(Ran3 &g, NormState &ns) {
  if (ns.set == 0) {
    double v1, v2, r, fac;
    do {
      v1 = (double)(2.0 * r3_rand(g) - 1.0);
      v2 = (double)(2.0 * r3_rand(g) - 1.0);
      r = v1 * v1 + v2 * v2;
    } while (r >= 1.0 || r == 0.0);
    fac = (double)sqrt(-2.0 * log_cr(r) / r);
    ns.cache = v1 * fac;
    ns.set = 1;
    return v2 * fac;
  }
  ns.set = 0;
  return ns.cache;
}

// erflib.c:172-181.  The reference converts a possibly negative double to
// uint32_t; its x86-64 build truncates to 64 bits and keeps the low 32 bits
// (so -1.0 gives 0xFFFFFFFF), which the two casts state explicitly (a plain
// device cast would saturate to 0).
__host__ __device__ static inline uint32_t roundr2i(double r) {
  double i = floor(r);
  if (i + 0.5 > r) return (uint32_t)(int64_t)i;
  return (uint32_t)(int64_t)(i + 1.0);
}

__device__ static inline uint32_t subpop_of(const NetConst *net, uint32_t in_cm) {
  for (uint32_t s = 0; s < net->nsub; s++)
    if (in_cm >= net->offset[s] && in_cm < net->offset[s] + net->count[s]) return s;
  return 0xFFFFFFFFu;
}

// ------------------------------------------------------------------ generation
// A cortical module's neurons consume its serial ran3 stream in order
// (simpleCM_invokeIndivSynGenerators, DPSNN_LIFCAcorticalModuleGen.cpp:62-220).
// Modules are independent streams (SetRandomSeed(module) at :96-107) except
// for NormDev's cached value, which carries from one module to the next
// inside a rank.  Two forms:
//  - where no weight can be rejected (below, and the rule in engine_build), a
//    warp per module finds every neuron's position in the stream
//    (gen_chain_kernel), and a warp per neuron then generates its synapses
//    (gen_fill_kernel);
//  - otherwise one thread walks one module (gen_kernel): a rejected weight
//    draws again, so that a neuron's draws depend on its weights.  Pass A runs
//    each module under both hypotheses for NormDev's cache (empty, or holding
//    a value that the module's first weight accepts) and pass B regenerates
//    the chosen one, writing synapses straight into their CSR slots.
struct GenRecord {
  uint32_t nsyn;
  int32_t used_normdev, set_out, err;
  double cache_out;
  float first_mean, first_sigma;
  uint32_t err_arg;
  uint32_t hist[55];
};

enum { GEN_ERR_TOO_MANY = 1, GEN_ERR_WEIGHT_RANGE = 2, GEN_ERR_PROB = 3, GEN_ERR_DELAY = 4,
       GEN_ERR_ZERO_MEAN = 5, GEN_ERR_DELAY_LEVEL = 6, GEN_ERR_DELAY_RANGE = 7 };

__device__ static inline uint32_t empty_random_synapses(Ran3 &g, float pf, uint32_t max_n) {
  // getEmptyRandomSynapses (DPSNN_LIFCAconnectome.cpp:1079-1133)
  double connectivity = (double)pf;
  double r = r3_rand(g);
  double P = connectivity, C = P;
  uint32_t n = 1;
  while ((C < r) && (n <= max_n)) {
    n++;
    P *= 1 - connectivity;
    C += P;
  }
  return n;
}

// Delay generators' error returns (the reference's exit(0) points).
#define DELAY_LEVEL_ERR 0xFFFFFFFFu   // level >= DSD__delayNum
#define DELAY_RANGE_ERR 0xFFFFFFFEu   // delay beyond the pair's DMax

__device__ static inline uint32_t random_delay_uni(const NetConst *net, double u, uint32_t s, uint32_t t) {
  // getRandomDelay_UNI (DPSNN_LIFCAcorticalModuleGen.cpp:299-338)
  float outF, DMin, DMax, DelayMin, DelayMax, DelayStep, DelayNum;
  DMin = (float)net->DMin[s * DPSNN_MAX_SUBPOP + t];
  DMax = (float)net->DMax[s * DPSNN_MAX_SUBPOP + t];
  DelayMin = (float)net->delay_min;
  DelayMax = (float)net->delay_max;
  DelayNum = 80;
  DelayStep = (DelayMax - DelayMin) / DelayNum;
  DelayMax -= DelayStep / 2;
  DelayMin += DelayStep / 2;
  DMax = roundr2i((DMax - DelayMin) / DelayStep) * DelayStep + DelayMin;
  DMin = roundr2i((DMin - DelayMin) / DelayStep) * DelayStep + DelayMin;
  outF = (float)((u * (DMax - DMin) + DMin - DelayMin) / DelayStep);
  (void)DelayMax;
  // the reference stops here: "delay level generated %f > %f max allowed
  // delay levels" (:322-326); the level goes back in the error argument
  if (outF >= DelayNum) return DELAY_LEVEL_ERR;
  const uint32_t outfunc = roundr2i(outF * DelayStep);
  if (outfunc > net->DMax[s * DPSNN_MAX_SUBPOP + t]) return DELAY_RANGE_ERR;   // :330-334
  return outfunc;
}

// getRandomDelay_EXP (DPSNN_LIFCAcorticalModuleGen.cpp:247-297), the
// reference Makefile's default: a truncated exponential over [DMin, DMax);
// DELAY_LEVEL_ERR / DELAY_RANGE_ERR where the reference stops with an error.
__device__ static inline uint32_t random_delay_exp(const NetConst *net, double u, uint32_t s, uint32_t t) {
  float outfuncF, DMin, DMax, DelayMin, DelayMax, DelayStep, DelayNum;
  const float InvLogTN = net->inv_log_tn;
  DMin = (float)net->DMin[s * DPSNN_MAX_SUBPOP + t];
  DMax = (float)net->DMax[s * DPSNN_MAX_SUBPOP + t];
  DelayMin = (float)net->delay_min;
  DelayMax = (float)net->delay_max;
  DelayNum = 80;
  DelayStep = (DelayMax - DelayMin) / DelayNum;
  DelayMax -= DelayStep / 2;
  DelayMin += DelayStep / 2;
  DMax = roundr2i((DMax - DelayMin) / DelayStep) * DelayStep + DelayMin;
  DMin = roundr2i((DMin - DelayMin) / DelayStep) * DelayStep + DelayMin;
  outfuncF = (float)((((double)DMin + (double)(DMax - DMin - DelayStep) *
                       log_cr(1.0 - u * (1.0 - 0.05)) * (double)InvLogTN) -
                      (double)DelayMin) / (double)DelayStep);
  if (outfuncF >= DelayNum) return DELAY_LEVEL_ERR;
  const uint32_t outfunc = roundr2i(outfuncF * DelayStep);
  if (outfunc >= net->DMax[s * DPSNN_MAX_SUBPOP + t]) return DELAY_RANGE_ERR;
  (void)DelayMax;
  return outfunc;
}

// The external bath rate of one neuron
// (ModuleGen.cpp:201-211, LIFCAconnectome.cpp:871-887).
__device__ static inline void gen_bath_rate(const NetConst *net, const uint32_t *__restrict__ bath_tmpl, uint32_t ssub,
                                            uint32_t cfx, uint32_t cfy, double &inv_nu, uint32_t &max_ext) {
  const float nu = (float)net->NuExt[ssub];
  uint32_t bx = cfx, by = cfy;
  if (bx >= net->cfx / 2) bx = 0u - (bx - net->cfx + 1u);   // unsigned, as the reference computes it
  if (by >= net->cfy / 2) by = 0u - (by - net->cfy + 1u);
  if (bx >= net->stencil_dim) bx = net->stencil_dim - 1;
  if (by >= net->stencil_dim) by = net->stencil_dim - 1;
  const float cext = (float)bath_tmpl[bx * net->stencil_dim + by];
  inv_nu = 0;
  max_ext = 0;
  if (cext != 0) {
    inv_nu = 1000.0 / (nu * cext);
    max_ext = (uint32_t)ceil(20 / inv_nu);
  }
}

#define GEN_THREADS 16          // generation streams per block
#define GEN_TL_SMEM 2048        // targets of a neuron held in shared memory
#define GEN_TL_STRIDE (GEN_TL_SMEM + 1)   // odd stride: threads' lists in different banks
#define GEN_SMEM ((size_t)GEN_THREADS * (sizeof(Ran3) + 4 * GEN_TL_STRIDE + 2 * RING_SLOTS))

// A neuron's target list: the first GEN_TL_SMEM entries in shared memory,
// the rest (rare: in-degrees are ~1100) in the thread's global scratch.
struct GenTargets {
  uint32_t *sh, *gl;
  __device__ uint32_t &operator[](uint32_t j) const { return j < GEN_TL_SMEM ? sh[j] : gl[j]; }
};

__global__ void gen_kernel(const NetConst *__restrict__ net, const float *__restrict__ prob, int pass,
                           GenRecord *rec, const int32_t *__restrict__ chosen_hyp,
                           const double *__restrict__ chosen_cache, uint16_t *cnt_out,
                           const uint64_t *__restrict__ row_ptr, const uint16_t *__restrict__ sub_off,
                           uint32_t *post, int16_t *w16, uint32_t *scratch,
                           const uint32_t *__restrict__ bath_tmpl, double *inv_nu,
                           uint32_t *max_ext, uint8_t *sub) {
  // Each thread's serial stream keeps its ran3 table, the current neuron's
  // target list (its first GEN_TL_SMEM entries; more go to the global
  // scratch) and the per-delay counts in shared memory: the stream is a long
  // chain of dependent table reads.
  extern __shared__ __align__(16) unsigned char gen_smem_raw[];
  Ran3 *s_rng = reinterpret_cast<Ran3 *>(gen_smem_raw);
  uint32_t *s_tl = reinterpret_cast<uint32_t *>(s_rng + blockDim.x);
  uint16_t *s_cnt = reinterpret_cast<uint16_t *>(s_tl + (size_t)blockDim.x * GEN_TL_STRIDE);
  uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t nthreads = (pass == 0) ? 2 * net->nmod : net->nmod;
  if (tid >= nthreads) return;
  uint32_t m = (pass == 0) ? (tid >> 1) : tid;
  int hyp = (pass == 0) ? (int)(tid & 1) : chosen_hyp[m];
  GenRecord *R = &rec[(pass == 0) ? tid : m];
  const uint32_t N = net->N, D = net->D, npcm = net->npcm, stencil = net->stencil;
  GenTargets tl{s_tl + (size_t)threadIdx.x * GEN_TL_STRIDE, scratch + (size_t)tid * MAX_SYN_PER_NEURON};
  uint16_t *cnt = s_cnt + (size_t)threadIdx.x * RING_SLOTS;

  Ran3 &g = s_rng[threadIdx.x];
  g.iff = 0;
  g.idum = 0;
  g.inext = g.inextp = 0;
  if (m % net->mods_per_rank == 0) r3_seed(g, (int32_t)net->global_seed);  // localNet_init.c:119
  r3_seed(g, (int32_t)m);  // module start (ModuleGen.cpp:96-107); m==0 does not re-initialise
  NormState ns;
  ns.set = hyp;
  ns.cache = (pass == 1 && hyp == 1) ? chosen_cache[m] : 0.0;
  int used = 0;
  uint32_t nsyn = 0;
  R->err = 0;
  for (uint32_t gi = m * npcm; gi < (m + 1) * npcm; gi++) {
    uint32_t mod = gi / npcm;
    uint32_t cfy = mod / net->cfx, cfx = mod % net->cfx;
    uint32_t ssub = subpop_of(net, gi % npcm);
    if (pass == 1) sub[gi] = (uint8_t)ssub;
    uint32_t tot = 0;
    for (uint32_t ts = 0; ts < net->nsub; ts++)
      for (uint32_t x = 0; x < stencil; x++)
        for (uint32_t y = 0; y < stencil; y++) {
          int32_t nx = (int32_t)cfx + (int32_t)x - (int32_t)net->max_mod;
          int32_t ny = (int32_t)cfy + (int32_t)y - (int32_t)net->max_mod;
          if (nx < 0 || nx >= (int32_t)net->cfx || ny < 0 || ny >= (int32_t)net->cfy) continue;
          float pf = prob[(((size_t)ssub * DPSNN_MAX_SUBPOP + ts) * stencil + x) * stencil + y];
          if (!(pf > 0)) continue;
          if (!(pf > 0.00001f)) { R->err = GEN_ERR_PROB; R->err_arg = gi; return; }
          uint32_t in_cm = net->offset[ts] - 1;
          uint32_t last = net->offset[ts] + net->count[ts];
          uint32_t avail = last - in_cm;
          while ((in_cm += empty_random_synapses(g, pf, avail)) < last) {
            if (tot >= MAX_SYN_PER_NEURON) { R->err = GEN_ERR_TOO_MANY; R->err_arg = gi; return; }
            tl[tot++] = in_cm + (uint32_t)nx * npcm + (uint32_t)ny * npcm * net->cfx;
          }
        }
    if (tot >= MAX_SYN_PER_NEURON) { R->err = GEN_ERR_TOO_MANY; R->err_arg = gi; return; }
    for (uint32_t d = 0; d < D; d++) cnt[d] = 0;
    for (uint32_t j = 0; j < tot; j++) {
      uint32_t tg = tl[j];
      uint32_t tsub = subpop_of(net, tg % npcm);
      const double u = r3_rand(g);
      uint32_t delay = net->delay_exp ? random_delay_exp(net, u, ssub, tsub) : random_delay_uni(net, u, ssub, tsub);
      if (delay == DELAY_LEVEL_ERR) { R->err = GEN_ERR_DELAY_LEVEL; R->err_arg = gi; return; }
      if (delay == DELAY_RANGE_ERR) { R->err = GEN_ERR_DELAY_RANGE; R->err_arg = gi; return; }
      if (delay >= D) { R->err = GEN_ERR_DELAY; R->err_arg = delay; return; }
      float mean = (float)net->J[ssub * DPSNN_MAX_SUBPOP + tsub];
      float sigma = (float)(net->DJ[ssub * DPSNN_MAX_SUBPOP + tsub] * (double)mean);
      if (!used) {
        used = 1;
        R->first_mean = mean;
        R->first_sigma = sigma;
      }
      float wf;
      if (mean > 0.0) {
        do { wf = (float)(mean + normdev(g, ns) * sigma); } while ((wf < 0.0) || (wf >= 2.0 * mean));
      } else {
        if (mean == 0.0f) { R->err = GEN_ERR_ZERO_MEAN; R->err_arg = gi; return; }
        do { wf = (float)(mean + normdev(g, ns) * sigma); } while ((wf <= 2.0 * mean) || (wf > 0));
      }
      if ((wf < net->min_w) || (wf > (-net->min_w))) { R->err = GEN_ERR_WEIGHT_RANGE; R->err_arg = gi; return; }
      int16_t w = (int16_t)(wf * net->f2w);
      if (pass == 0) {
        cnt[delay]++;
      } else {
        uint64_t pos = row_ptr[gi] + sub_off[(size_t)gi * (D + 1) + delay] + cnt[delay]++;
        post[pos] = tg;
        w16[pos] = w;
      }
      nsyn++;
    }
    if (pass == 0) {
      uint16_t *co = cnt_out + ((size_t)hyp * N + gi) * D;
      for (uint32_t d = 0; d < D; d++) co[d] = cnt[d];
    } else {
      gen_bath_rate(net, bath_tmpl, ssub, cfx, cfy, inv_nu[gi], max_ext[gi]);
    }
  }
  R->nsyn = nsyn;
  R->used_normdev = used;
  R->set_out = ns.set;
  R->cache_out = ns.cache;
  r3_history(g, R->hist);
}

// ---- the warp form
// One (target sub-population, stencil cell) of a source sub-population with
// a connection probability, in the reference's order.
struct GenRow {
  int32_t dx, dy;
  uint32_t ts, tab;   // tab: its probability's table
};
// A probability's table of getEmptyRandomSynapses (DPSNN_LIFCAconnectome.cpp:1079-1133):
// C[n] = the sum of the reference's first n terms, n = 1 .. len, so that a
// draw r gives the first n with C[n] >= r, len + 1 if there is none.
struct GenTab {
  float pf, inv_log2q;   // 1 / log2(1 - pf): the first guess at n
  uint32_t len;
  uint32_t off;          // C[1] at gen_c[off]
};
__global__ void gen_tab_kernel(const GenTab *__restrict__ tab, uint32_t n, double *__restrict__ gen_c) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double connectivity = (double)tab[i].pf;
  double P = connectivity, C = P;
  for (uint32_t k = 0; k < tab[i].len; k++) {
    gen_c[tab[i].off + k] = C;
    P *= 1 - connectivity;
    C += P;
  }
}

// A ran3 stream in a warp's shared ring: draw n at n % GEN_RING, drawn up to
// `end`, the 220 draws before it kept.
#define GEN_RING 512
#define GEN_HIST 55
struct GenStream {
  uint32_t *x;
  uint32_t end;
  __device__ uint32_t at(uint32_t n) const { return x[n % GEN_RING]; }
  __device__ double u(uint32_t n) const { return (__hiloint2double(0x43300000, (int)at(n)) - 0x1p52) * (1.0 / (double)MBIG); }
};
// The draws before n0 from their last 55 (already at n0-55 .. n0-1): the
// recurrence backwards, x[k] = x[k+55] + x[k+31] (mod MBIG), 31 at a time.
__device__ static inline void gen_backfill(GenStream &g, uint32_t n0, uint32_t lane) {
  __syncwarp();
  for (uint32_t hi = n0 - GEN_HIST; hi > n0 - 224; hi -= 31) {
    const uint32_t k = hi - 1 - lane;
    uint32_t v = g.at(k + 55) + g.at(k + 31);
    if (v >= MBIG) v -= MBIG;
    __syncwarp();
    if (lane < 31) g.x[k % GEN_RING] = v;
    __syncwarp();
  }
  g.end = n0;
}
// Draws up to n: x[n] = x[n-96] - 4 x[n-127] + 6 x[n-158] - 4 x[n-189] + x[n-220] (bath_kernel), 96 at a time.
__device__ static inline void gen_draw(GenStream &g, uint32_t n, uint32_t lane) {
  while ((int32_t)(n - g.end) > 0) {
    uint32_t x[3];
#pragma unroll
    for (int v = 0; v < 3; v++) {
      const uint32_t k = g.end + lane + 32 * v;
      const int32_t x3 = 2 * (int32_t)g.at(k - 158);
      int32_t y = (int32_t)(g.at(k - 96) + g.at(k - 220)) - x3, z = (int32_t)(g.at(k - 127) + g.at(k - 189)) - x3;
      if (y < 0) y += MBIG;
      if (y < 0) y += MBIG;
      if (y >= MBIG) y -= MBIG;
      if (z < 0) z += MBIG;
      if (z < 0) z += MBIG;
      z = 2 * (z >= MBIG ? z - MBIG : z);
      if (z >= MBIG) z -= MBIG;
      y -= 2 * z;
      if (y < 0) y += MBIG;
      if (y < 0) y += MBIG;
      x[v] = (uint32_t)y;
    }
    __syncwarp();
#pragma unroll
    for (int v = 0; v < 3; v++) g.x[(g.end + lane + 32 * v) % GEN_RING] = x[v];
    __syncwarp();
    g.end += 96;
  }
}

// getEmptyRandomSynapses for raw draw mj (u as ran3 returns it): a guess from
// the logarithm, then the table decides.
__device__ static inline uint32_t gen_skip(const GenTab &tb, const double *__restrict__ gen_c, uint32_t mj, double u) {
  int n = (int)ceilf(__log2f((float)(MBIG - mj) * 1e-9f) * tb.inv_log2q);
  const int len = (int)tb.len;
  n = max(1, min(n, len + 1));
  const double *C = gen_c + tb.off - 1;
  while (n <= len && __ldg(&C[n]) < u) n++;
  while (n > 1 && __ldg(&C[n - 1]) >= u) n--;
  return (uint32_t)n;
}

// One row's targets from draw pos on (K draws per lane at once): `emit`
// receives (index in the row's list, index in the sub-population).  Returns
// their number; pos moves past the row's draws.
template <int K, typename Emit>
__device__ static inline uint32_t gen_row(GenStream &g, const GenTab &tb, const double *__restrict__ gen_c, uint32_t count,
                                          uint32_t &pos, uint32_t lane, const Emit &emit) {
  int32_t at = -1;
  uint32_t tot = 0;
  for (;;) {
    gen_draw(g, pos + 32 * K, lane);
    int32_t s[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t n = pos + K * lane + k;
      s[k] = (int32_t)gen_skip(tb, gen_c, g.at(n), g.u(n));
    }
#pragma unroll
    for (int k = 1; k < K; k++) s[k] += s[k - 1];
    int32_t incl = s[K - 1];
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    const int32_t base = at + incl - s[K - 1];
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < K; k++)
      if (base + s[k] < (int32_t)count) {
        emit(tot + K * lane + k, (uint32_t)(base + s[k]));
        v++;
      }
    const uint32_t full = __popc(__ballot_sync(0xffffffffu, v == K));   // the lanes before the row's end
    if (full == 32) {
      tot += 32 * K;
      pos += 32 * K;
      at = __shfl_sync(0xffffffffu, base + s[K - 1], 31);
      continue;
    }
    const uint32_t last = full * K + __shfl_sync(0xffffffffu, v, full);
    pos += last + 1;
    return tot + last;
  }
}
template <typename Emit>
__device__ static inline uint32_t gen_row(GenStream &g, const GenTab &tb, const double *__restrict__ gen_c, uint32_t count,
                                          uint32_t &pos, uint32_t lane, const Emit &emit) {
  return tb.pf * (float)count > 48.0f ? gen_row<4>(g, tb, gen_c, count, pos, lane, emit)
                                      : gen_row<1>(g, tb, gen_c, count, pos, lane, emit);
}

// The weights' draws.  Without rejected weights two targets in a row draw
// one delay, pairs of uniforms until one lies in the unit circle (NormDev,
// randdev.c:584-606; its second value is cached) and the other's delay: in
// steps of two draws from the first target's, pair g is at draw 1 + 2 g, and
// after an accepted pair g the next unit starts at step g + 2.  So of a run
// of acceptable pairs every other one is accepted, starting with the first.
// gen_pairs: of the 64 pairs from draw p on, which are accepted; carry: the
// pair before them was (and the first of them is skipped).
__device__ static inline uint64_t gen_pairs(const GenStream &g, uint32_t p, bool carry, uint32_t lane) {
  bool ok[2];
#pragma unroll
  for (int v = 0; v < 2; v++) {
    const uint32_t n = p + 2 * (lane + 32 * v);
    const double v1 = 2.0 * g.u(n) - 1.0, v2 = 2.0 * g.u(n + 1) - 1.0, r = v1 * v1 + v2 * v2;
    ok[v] = !(r >= 1.0 || r == 0.0);
  }
  const uint64_t m0 = __ballot_sync(0xffffffffu, ok[0]) | ((uint64_t)__ballot_sync(0xffffffffu, ok[1]) << 32);
  const uint64_t m = m0 & ~(uint64_t)carry, E = 0x5555555555555555ull;
  // adding a run's first bit clears the run: the runs that start at even positions, then the others
  const uint64_t even = m & ~(m + (m & ~(m << 1) & E));
  return (even & E) | (m & ~even & ~E);
}

// What gen_chain_kernel leaves of a module's stream (2 per module: NormDev's
// cache empty, or full, as the module starts).
struct GenChain {
  uint64_t nsyn;
  uint32_t err, err_arg;
  uint32_t set_out, c_out[2];   // cache at the end, and the pair of draws it comes from
  uint32_t hist[GEN_HIST];
};
// Per neuron and hypothesis: the draws before its first, whether NormDev's
// cache is full (2: from before the module), and the pair it comes from.
struct GenStart {
  uint32_t hist[GEN_HIST];
  uint32_t set, c[2];
};

// A warp per stream: every neuron's first draw and number of synapses.
// What bounds it: the serial chain of a module's neurons, about 40 rows and 20
// windows of pairs each; a warp does 32 or 128 draws of a row, or 64 pairs,
// per step.  Measured: 20 ms for a module of 1250 neurons (16 us per neuron),
// 40 ms for the 576 modules of the 24x24 network under both hypotheses; a
// thread per module took 2 s per pass, and two passes.
__global__ void __launch_bounds__(32) gen_chain_kernel(const NetConst *__restrict__ net, const GenRow *__restrict__ rows,
                                                       const uint32_t *__restrict__ row_off, const GenTab *__restrict__ tabs,
                                                       const double *__restrict__ gen_c, GenChain *chain,
                                                       GenStart *__restrict__ start, uint32_t *__restrict__ tot_out) {
  __shared__ uint32_t ring[GEN_RING];
  const uint32_t lane = threadIdx.x, m = blockIdx.x >> 1, hyp = blockIdx.x & 1;
  GenChain *R = &chain[blockIdx.x];
  if (hyp && m % net->mods_per_rank == 0) return;   // a rank starts with an empty cache
  const uint32_t N = net->N, npcm = net->npcm, cfy = m / net->cfx, cfx = m % net->cfx, n0 = 256;
  GenStream g{ring, n0};
  if (lane == 0) {
    Ran3 r;
    r.iff = 0;
    r.idum = 0;
    r.inext = r.inextp = 0;
    if (m % net->mods_per_rank == 0) r3_seed(r, (int32_t)net->global_seed);  // localNet_init.c:119
    r3_seed(r, (int32_t)m);  // module start (ModuleGen.cpp:96-107); m==0 does not re-initialise
    r3_history(r, ring + n0 - GEN_HIST);
  }
  gen_backfill(g, n0, lane);
  uint32_t pos = n0, set = hyp ? 2u : 0u, c0 = 0, c1 = 0;
  uint64_t nsyn = 0;
  for (uint32_t k = 0; k < npcm; k++) {
    const uint32_t ssub = subpop_of(net, k), gi = m * npcm + k;
    GenStart &S = start[(size_t)hyp * N + gi];
    for (uint32_t i = lane; i < GEN_HIST; i += 32) S.hist[i] = g.at(pos - GEN_HIST + i);
    if (lane == 0) {
      S.set = set;
      S.c[0] = c0;
      S.c[1] = c1;
    }
    uint32_t tot = 0;
    for (uint32_t i = row_off[ssub]; i < row_off[ssub + 1]; i++) {
      const GenRow w = rows[i];
      const int32_t nx = (int32_t)cfx + w.dx, ny = (int32_t)cfy + w.dy;
      if (nx < 0 || nx >= (int32_t)net->cfx || ny < 0 || ny >= (int32_t)net->cfy) continue;
      tot += gen_row(g, tabs[w.tab], gen_c, net->count[w.ts], pos, lane, [](uint32_t, uint32_t) {});
      if (tot >= MAX_SYN_PER_NEURON) {
        if (lane == 0) {
          R->err = GEN_ERR_TOO_MANY;
          R->err_arg = gi;
        }
        return;
      }
    }
    if (lane == 0) tot_out[(size_t)hyp * N + gi] = tot;
    nsyn += tot;
    uint32_t rem = tot;
    if (rem && set) {   // the first target's weight comes from the cache
      set = 0;
      pos++;
      rem--;
    }
    uint32_t units = (rem + 1) / 2;
    bool carry = false;
    for (uint32_t p = pos; units; p += 128) {
      gen_draw(g, p + 1 + 128, lane);
      uint64_t acc = gen_pairs(g, p + 1, carry, lane);
      const uint32_t cnt = __popcll(acc);
      carry = acc >> 63;
      if (cnt < units) {
        units -= cnt;
        continue;
      }
      // the last unit's pair: the units-th set bit
      uint32_t at = 0, want = units;
      for (uint32_t w = 32; w > 0; w >>= 1) {
        const uint32_t c = __popcll(acc & ((1ull << w) - 1));
        if (c < want) {
          want -= c;
          acc >>= w;
          at += w;
        }
      }
      pos = p + 2 * at + ((rem & 1) ? 3 : 4);
      if (rem & 1) {
        set = 1;
        c0 = g.at(p + 1 + 2 * at);
        c1 = g.at(p + 2 + 2 * at);
      }
      units = 0;
    }
    gen_draw(g, pos, lane);
  }
  for (uint32_t i = lane; i < GEN_HIST; i += 32) R->hist[i] = g.at(pos - GEN_HIST + i);
  if (lane == 0) {
    R->nsyn = nsyn;
    R->set_out = set;
    R->c_out[0] = c0;
    R->c_out[1] = c1;
  }
}

#define GEN_FILL_WARPS 4
#define GEN_FILL_LIST 1536      // a neuron's synapses held in shared memory; more in the warp's global scratch
struct GenFillWarp {
  uint32_t ring[GEN_RING];
  uint32_t tg[GEN_FILL_LIST];
  int16_t w[GEN_FILL_LIST];
  uint8_t dl[GEN_FILL_LIST];
  uint32_t cnt[RING_SLOTS + 1];
  uint8_t pair[32];
};
struct GenFillScratch {   // per warp
  uint32_t tg[MAX_SYN_PER_NEURON];
  int16_t w[MAX_SYN_PER_NEURON];
  uint8_t dl[MAX_SYN_PER_NEURON];
};

// One synapse's delay and weight from its draws; GEN_ERR_* where the
// reference stops.
__device__ static inline uint32_t gen_synapse(const NetConst *net, uint32_t ssub, uint32_t tsub, double ud, double z,
                                              uint32_t &delay, int16_t &w) {
  delay = net->delay_exp ? random_delay_exp(net, ud, ssub, tsub) : random_delay_uni(net, ud, ssub, tsub);
  if (delay == DELAY_LEVEL_ERR) return GEN_ERR_DELAY_LEVEL;
  if (delay == DELAY_RANGE_ERR) return GEN_ERR_DELAY_RANGE;
  if (delay >= net->D) return GEN_ERR_DELAY;
  const float mean = (float)net->J[ssub * DPSNN_MAX_SUBPOP + tsub];
  const float sigma = (float)(net->DJ[ssub * DPSNN_MAX_SUBPOP + tsub] * (double)mean);
  if (mean == 0.0f) return GEN_ERR_ZERO_MEAN;
  const float wf = (float)(mean + z * sigma);
  if ((wf < net->min_w) || (wf > (-net->min_w))) return GEN_ERR_WEIGHT_RANGE;
  w = (int16_t)(wf * net->f2w);
  return 0;
}

// A warp per neuron: its targets, delays and weights from its first draw on
// (in shared memory), then its CSR row, sorted by delay and in generation
// order within one.  What bounds it: issue slots, the correctly rounded log
// of a pair's radius above all, which 28 of 32 lanes do at a time.  Measured:
// 37 ms for the 0.81 G synapses of the 24x24 network (a row's 1125 synapses in
// about 120 us of a warp's time, 16 warps per SM).
__global__ void __launch_bounds__(32 * GEN_FILL_WARPS)
    gen_fill_kernel(const NetConst *__restrict__ net, const GenRow *__restrict__ rows, const uint32_t *__restrict__ row_off,
                    const GenTab *__restrict__ tabs, const double *__restrict__ gen_c, const GenStart *__restrict__ start,
                    const int32_t *__restrict__ hyp, const uint2 *__restrict__ mod_cache,
                    const uint64_t *__restrict__ row_ptr, uint16_t *__restrict__ sub_off, uint32_t *__restrict__ post,
                    int16_t *__restrict__ w16, GenFillScratch *scratch, unsigned long long *err,
                    const uint32_t *__restrict__ bath_tmpl, double *__restrict__ inv_nu, uint32_t *__restrict__ max_ext,
                    uint8_t *__restrict__ sub) {
  extern __shared__ __align__(16) unsigned char gen_fill_raw[];
  const uint32_t lane = threadIdx.x & 31, wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  GenFillWarp &s = reinterpret_cast<GenFillWarp *>(gen_fill_raw)[threadIdx.x >> 5];
  const uint32_t N = net->N, D = net->D, npcm = net->npcm, n0 = 256;
  for (uint32_t gi = wid; gi < N; gi += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t m = gi / npcm, cfy = m / net->cfx, cfx = m % net->cfx, ssub = subpop_of(net, gi % npcm);
    const GenStart &S = start[(size_t)hyp[m] * N + gi];
    const uint64_t row = row_ptr[gi];
    const uint32_t tot = (uint32_t)(row_ptr[gi + 1] - row);
    const bool big = tot > GEN_FILL_LIST;   // scratch is there when a neuron has that many
    uint32_t *tg = big ? scratch[wid].tg : s.tg;
    int16_t *wl = big ? scratch[wid].w : s.w;
    uint8_t *dl = big ? scratch[wid].dl : s.dl;
    GenStream g{s.ring, n0};
    for (uint32_t i = lane; i < GEN_HIST; i += 32) s.ring[n0 - GEN_HIST + i] = S.hist[i];
    for (uint32_t i = lane; i <= D; i += 32) s.cnt[i] = 0;
    gen_backfill(g, n0, lane);
    // targets, with their sub-population in the top bits (a network has fewer than 2^25 neurons)
    uint32_t pos = n0, k0 = 0;
    for (uint32_t i = row_off[ssub]; i < row_off[ssub + 1]; i++) {
      const GenRow w = rows[i];
      const int32_t nx = (int32_t)cfx + w.dx, ny = (int32_t)cfy + w.dy;
      if (nx < 0 || nx >= (int32_t)net->cfx || ny < 0 || ny >= (int32_t)net->cfy) continue;
      const uint32_t first = net->offset[w.ts] + (uint32_t)nx * npcm + (uint32_t)ny * npcm * net->cfx, top = w.ts << 25;
      k0 += gen_row(g, tabs[w.tab], gen_c, net->count[w.ts], pos, lane, [&](uint32_t k, uint32_t at) {
        if (k0 + k < tot) tg[k0 + k] = top | (first + at);
      });
    }
    __syncwarp();
    auto synapse = [&](uint32_t k, double ud, double z) {
      uint32_t delay = 0;
      int16_t w = 0;
      const uint32_t e = gen_synapse(net, ssub, tg[k] >> 25, ud, z, delay, w);
      if (e) {
        atomicMin(err, ((unsigned long long)gi << 39) | ((unsigned long long)k << 26) | ((unsigned long long)e << 22) |
                           min(e == GEN_ERR_DELAY ? delay : 0u, 0x3FFFFFu));
        delay = 0;
      }
      dl[k] = (uint8_t)delay;
      wl[k] = w;
      atomicAdd(&s.cnt[delay], 1u);
    };
    auto polar = [&](uint32_t a, uint32_t b, double &z2, double &z1) {   // NormDev of the pair of draws (a, b)
      const double v1 = 2.0 * ((double)a * (1.0 / (double)MBIG)) - 1.0;
      const double v2 = 2.0 * ((double)b * (1.0 / (double)MBIG)) - 1.0;
      const double r = v1 * v1 + v2 * v2, fac = sqrt(-2.0 * log_cr(r) / r);
      z1 = v1 * fac;
      z2 = v2 * fac;
    };
    uint32_t done = 0;
    if (tot && S.set) {   // the first target's weight comes from the cache
      if (lane == 0) {
        double z2, z1;
        if (S.set == 2) polar(mod_cache[m].x, mod_cache[m].y, z2, z1);
        else polar(S.c[0], S.c[1], z2, z1);
        synapse(0, g.u(pos), z1);
      }
      pos++;
      done = 1;
    }
    bool carry = false;
    int32_t prev = -2;   // pair of the last unit, from this window's first: the next unit starts two on
    for (uint32_t p = pos; done < tot; p += 128) {
      gen_draw(g, p + 130, lane);   // the last pair's unit ends with the draw after it
      const uint64_t acc = gen_pairs(g, p + 1, carry, lane);
      carry = acc >> 63;
      // the window's accepted pairs (at most 32, no two adjacent), a lane each
#pragma unroll
      for (int v = 0; v < 2; v++) {
        const uint32_t b = lane + 32 * v;
        if ((acc >> b) & 1ull) s.pair[__popcll(acc & ((1ull << b) - 1))] = (uint8_t)b;
      }
      __syncwarp();
      const uint32_t cnt = __popcll(acc), k = done + 2 * lane;
      if (lane < cnt && k < tot) {
        const int32_t pr = s.pair[lane], before = lane ? (int32_t)s.pair[lane - 1] : prev;
        double z2, z1;
        polar(g.at(p + 1 + 2 * pr), g.at(p + 2 + 2 * pr), z2, z1);
        synapse(k, g.u(p + 2 * (before + 2)), z2);
        if (k + 1 < tot) synapse(k + 1, g.u(p + 2 * pr + 3), z1);
      }
      prev = (cnt ? (int32_t)s.pair[cnt - 1] : prev) - 64;
      done += 2 * cnt;
      __syncwarp();
    }
    __syncwarp();
    // offsets of the delays, then the row: each synapse after those of its
    // delay generated before it
    uint32_t acc = 0;
    for (uint32_t d0 = 0; d0 <= D; d0 += 32) {
      const uint32_t d = d0 + lane, c = d < D ? s.cnt[d] : 0u;
      uint32_t incl = c;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
      }
      if (d <= D) {
        s.cnt[d] = acc + incl - c;
        sub_off[(size_t)gi * (D + 1) + d] = (uint16_t)(acc + incl - c);
      }
      acc += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncwarp();
    for (uint32_t k = lane; k - lane < tot; k += 32) {
      const uint32_t d = k < tot ? dl[k] : 0xFFu;
      const uint32_t same = __match_any_sync(0xffffffffu, d), before = __popc(same & ((1u << lane) - 1));
      uint32_t at = 0;
      if (k < tot) at = s.cnt[d] + before;
      __syncwarp();
      if (k < tot) {
        if (before == 0) s.cnt[d] += __popc(same);
        post[row + at] = tg[k] & ((1u << 25) - 1);
        w16[row + at] = wl[k];
      }
      __syncwarp();
    }
    if (lane == 0) {
      double inv;
      uint32_t mx;
      gen_bath_rate(net, bath_tmpl, ssub, cfx, cfy, inv, mx);
      inv_nu[gi] = inv;
      max_ext[gi] = mx;
      sub[gi] = (uint8_t)ssub;
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------ step kernels
struct Dev {
  NetConst *net;
  double *lut;              // [nsub*256]
  // neurons
  double *v, *c, *tr, *te, *nb, *inv_nu;
  const double *nb_prev;    // nextBath before this step's bath (bath_kernel input)
  uint32_t *max_ext;
  uint8_t *sub, *fired;
  int32_t *last_spike_ms;
  uint32_t *block_fired;    // per NEURON_BLOCK block
  uint32_t *fired_bits;     // [N/32] a small network's form of both: a bit per neuron
  uint32_t *ticket;         // blocks of tail_small_kernel that are done
  // connectome
  uint64_t *row_ptr;
  uint16_t *sub_off;
  uint32_t *post;
  int16_t *w16;
  float *tderiv;
  int32_t *last_act;
  // LTP probe (null unless enabled): weight and trace before the update,
  // and the trace after it before its decay
  int16_t *probe_w;
  float *probe_td, *probe_td_mid;
  // STDP event log of one step (null unless enabled): {synapse index lo/hi,
  // post | anti-causal << 31, contribution bits} of rank 0's synapses from
  // rank-0 neurons with a non-zero contribution
  uint4 *stdp_log;
  uint32_t *stdp_log_cnt;
  uint64_t *in_ptr;
  uint32_t *in_idx;
  // ring
  uint32_t *ring_ids, *ring_cnt;
  double *ring_te;
  // events
  uint32_t *ev_cnt;
  uint2 *ev;
  uint32_t *ovf_cnt;
  uint4 *ovf;
  double *huge_tau;                   // huge_kernel's scratch: HEAVY_MAX events per block
  uint32_t *huge_key;
  float *huge_val;
  uint32_t *heavy_list, *heavy_cnt;   // [4N]: neuron, event count of the warp path, then of
                                      // the block path; heavy_cnt[0..1]: their lengths
  // bath
  uint32_t *bath_hist;      // [P][BATH_KEEP] the BATH_HIST draws before each rank's next one, and some after
  uint32_t *bath_kept;      // [P] their number
  uint64_t *bath_rank_base; // [P+1]
  uint2 *bath_at;           // [N] first bath event of this step, and their number
  double2 *bath_ev;         // {time, input} per bath event
  const uint32_t *fix_bitmap; // one bit per float in [0x30000000, 0x3F800000]: key has a fix-up
  const double *fix_near;     // [256] by the result's exponent: a fix-up input's exact log lies at least
                              // this far from the float it rounds to
  const double2 *log_tab;     // [LOG_TAB_N] i = LOG_TAB_0 + k: 64/i, log(i/64)
  // control
  uint32_t *t;              // current step
  uint32_t *bath_t;         // [P] step of the rank's next bath (the bath runs one step ahead)
  uint32_t *flags;
  unsigned long long *events;  // synaptic events delivered
};

// Step 1: ordered spike compaction (compressNeuralSpikesInThisTimeStep,
// DPSNN_localNet_sim.c:103-132, :620-664): the neurons that fired during the
// previous step, ascending index, with their emission time Te, into ring slot
// t mod 80.  Also sets lastNeuralEmittedSpikeTime_ms = t.
__global__ void compact_kernel(Dev d) {
  const NetConst *net = d.net;
  const uint32_t N = net->N, t = *d.t, slot = t % RING_SLOTS;
  const uint32_t b = blockIdx.x, nb = gridDim.x;
  __shared__ uint32_t s_red[NEURON_BLOCK / 32];
  __shared__ uint32_t s_prefix;
  uint32_t part = 0;
  for (uint32_t k = threadIdx.x; k < b; k += blockDim.x) part += d.block_fired[k];
  for (int o = 16; o > 0; o >>= 1) part += __shfl_down_sync(0xffffffffu, part, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = part;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t s = 0;
    for (int w = 0; w < NEURON_BLOCK / 32; w++) s += s_red[w];
    s_prefix = s;
  }
  __syncthreads();
  uint32_t i = b * NEURON_BLOCK + threadIdx.x;
  uint32_t f = (i < N) ? d.fired[i] : 0;
  uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t bal = __ballot_sync(0xffffffffu, f);
  __shared__ uint32_t s_wcnt[NEURON_BLOCK / 32];
  if (lane == 0) s_wcnt[warp] = __popc(bal);
  __syncthreads();
  uint32_t woff = 0;
  for (uint32_t w = 0; w < warp; w++) woff += s_wcnt[w];
  if (f) {
    uint32_t q = s_prefix + woff + __popc(bal & ((1u << lane) - 1));
    d.fired[i] = 0;
    d.ring_ids[(size_t)slot * N + q] = i;
    d.ring_te[(size_t)slot * N + q] = d.te[i];
    d.last_spike_ms[i] = (int32_t)t;
    if (d.row_ptr[i + 1] == d.row_ptr[i]) atomicOr(d.flags, F_NO_TARGET);
  }
  if (b == nb - 1 && threadIdx.x == 0) {
    uint32_t tot = s_prefix;
    for (int w = 0; w < NEURON_BLOCK / 32; w++) tot += s_wcnt[w];
    d.ring_cnt[slot] = tot;
  }
}

#define STDP_LOG_CAP DPSNN_STDP_LOG_CAP   // STDP event records per step

// One record of the STDP event log (the statSTDPevent.write calls of
// DPSNN_neuron_sim.c:152-166 and :230-246, which report rank 0's synapses
// whose both ends are rank-0 neurons); the host restores the reference's order.
__device__ static inline void stdp_log_append(const Dev &d, uint64_t k, uint32_t post, uint32_t anti, float c) {
  const uint32_t o = atomicAdd(d.stdp_log_cnt, 1u);
  if (o < STDP_LOG_CAP)
    d.stdp_log[o] = make_uint4((uint32_t)k, (uint32_t)(k >> 32), post | (anti << 31), __float_as_uint(c));
  else
    atomicOr(d.flags, F_OVERFLOW);
}

// The anti-causal records of the STDP event log, after delivery: a synapse
// delivered at step t carries last_act == t (one delivery per synapse and
// step, none at step 0), and its contribution is the one delivery added.
__global__ void stdp_anti_log_kernel(Dev d) {
  const NetConst *net = d.net;
  const uint32_t t = *d.t;
  if (t == 0 || !(t >= net->start_pl && t <= net->stop_pl)) return;
  const uint64_t end = d.row_ptr[net->locN];
  for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < end; k += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t j = d.post[k];
    if (j >= net->locN || d.last_act[k] != (int32_t)t) continue;
    const int td = (int)t - d.last_spike_ms[j];
    const float a = (td < 128) ? net->anti_tab[td] : 0.0f;
    if (a != 0.0f) stdp_log_append(d, k, j, 1u, a);
  }
}

// Causal STDP at detection (causalSTDP_ms_ofBackwardSynapses,
// DPSNN_neuron_sim.c:94-177): one warp per spiking neuron walks its incoming
// synapses.
__global__ void causal_stdp_kernel(Dev d) {
  const NetConst *net = d.net;
  const uint32_t t = *d.t;
  if (!(t >= net->start_pl && t <= net->stop_pl)) return;
  const uint32_t slot = t % RING_SLOTS, cnt = d.ring_cnt[slot], N = net->N;
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < cnt;
       w += (gridDim.x * blockDim.x) >> 5) {
    uint32_t i = d.ring_ids[(size_t)slot * N + w];
    for (uint64_t k = d.in_ptr[i] + lane; k < d.in_ptr[i + 1]; k += 32) {
      uint32_t s = d.in_idx[k];
      int32_t la = d.last_act[s];
      int td = (int)t - 1 - la;
      float fc = (la != 0 && td < 128) ? net->causal_tab[td] : 0.0f;
      // the reference adds the term even when it is zero
      // (DPSNN_neuron_sim.c:171); a time derivative is never -0.0 (it starts
      // at +0.0 and no step of the plasticity makes a -0.0 from other
      // values), so skipping the zero terms changes no bit
      if (fc != 0.0f) d.tderiv[s] = d.tderiv[s] + fc;
      if (d.stdp_log && fc != 0.0f && t != 0 && i < net->locN && s < d.row_ptr[net->locN])
        stdp_log_append(d, s, i, 0u, fc);
    }
  }
}

// Step 2: delivery (axonalSpikeSchedulersToSynapticSpikeSchedulers,
// DPSNN_localNet_sim.c:837-999, and findAndGetNextSyn, DPSNN_synapse.c:179-267).
// Work item = (delay d, spike q of the slot written d steps ago), i.e. the CSR
// segment (pre, d).  A warp takes 32 work items at a time: each lane fetches
// one item's segment bounds, then the warp walks the concatenation of the 32
// segments with every lane on a different synapse, appending {key, weight}
// to each target's event list: per lane a batch of DELIVER_UNROLL synapses
// takes its slots (atomics) while the next batch's synapse loads are in
// flight.
// key = (D-1-d) << 25 | q orders a target's events as the reference delivers
// them (delay descending, then source ascending), which breaks ties between
// equal arrival times.
#define DELIVER_THREADS 256
#define DELIVER_UNROLL 2

// Stores one event in slot s of target j's list (taken by the caller's
// atomicAdd on ev_cnt[j]), or in the overflow list past the bucket.
__device__ static inline void deliver_event(const Dev &d, const NetConst *net, uint64_t k, uint32_t key,
                                            uint32_t t, bool stdp, uint32_t cap, uint32_t j, float wf,
                                            uint32_t s) {
  if (s < cap) {
    d.ev[(size_t)j * cap + s] = make_uint2(key, __float_as_uint(wf));
  } else {
    const uint32_t o = atomicAdd(d.ovf_cnt, 1u);
    if (o < net->ovf_cap)
      d.ovf[o] = make_uint4(j, key, __float_as_uint(wf), 0u);
    else
      atomicOr(d.flags, F_OVERFLOW);
  }
  if (stdp) {  // synapseSetLastActiveTime_antiCausalSTDP (DPSNN_neuron_sim.c:179-277)
    d.last_act[k] = (int32_t)t;
    const int td = (int)t - d.last_spike_ms[j];
    const float a = (td < 128) ? net->anti_tab[td] : 0.0f;
    if (a != 0.0f) d.tderiv[k] = d.tderiv[k] + a;   // zero terms change no bit (causal_stdp_kernel)
  }
}

// A small network's compaction (step 1), by every block of the kernel that
// needs the list: its fired bits are at most SMALL_N / 32 words, so each block
// counts them all and knows every spike's place without a launch or a wait;
// the blocks share the ring's writes.
#define SMALL_N 32768
#define SMALL_WORDS (SMALL_N / 32)
struct SmallSpikes {
  uint32_t bits[SMALL_WORDS];   // neurons that fired, a bit each
  uint32_t pre[SMALL_WORDS];    // spikes in the words before
  uint32_t warp_sum[DELIVER_THREADS / 32];
  uint32_t cnt;
  // the q-th spike's neuron
  __device__ uint32_t id(uint32_t q, uint32_t words) const {
    uint32_t lo = 0, hi = words - 1;   // the last word with pre <= q (empty words share their successor's pre)
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (pre[mid] <= q) lo = mid; else hi = mid - 1;
    }
    uint32_t k = q - pre[lo], w = bits[lo], at = 0;
    for (uint32_t h = 16; h > 0; h >>= 1) {   // the k-th set bit
      const uint32_t c = __popc(w & ((1u << h) - 1));
      if (k >= c) {
        k -= c;
        w >>= h;
        at += h;
      }
    }
    return 32 * lo + at;
  }
};
static_assert(SMALL_WORDS == 4 * DELIVER_THREADS, "four words per thread");

__device__ static inline void compact_small(const Dev &d, SmallSpikes &s, uint32_t t) {
  const uint32_t N = d.net->N, slot = t % RING_SLOTS, words = (N + 31) / 32;
  const uint32_t tid = threadIdx.x, lane = tid & 31, w0 = 4 * tid;
  uint32_t b[4], c = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    b[k] = w0 + k < words ? d.fired_bits[w0 + k] : 0u;
    c += __popc(b[k]);
  }
  uint32_t incl = c;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  if (lane == 31) s.warp_sum[tid >> 5] = incl;
  __syncthreads();
  uint32_t acc = incl - c;
  for (uint32_t w = 0; w < (tid >> 5); w++) acc += s.warp_sum[w];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    s.bits[w0 + k] = b[k];
    s.pre[w0 + k] = acc;
    acc += __popc(b[k]);
  }
  if (tid == DELIVER_THREADS - 1) {
    s.cnt = acc;
    if (blockIdx.x == 0) d.ring_cnt[slot] = acc;
  }
  __syncthreads();
  for (uint32_t w = blockIdx.x + gridDim.x * tid; w < words; w += gridDim.x * DELIVER_THREADS) {
    uint32_t q = s.pre[w];
    for (uint32_t m = s.bits[w]; m; m &= m - 1, q++) {
      const uint32_t i = 32 * w + __ffs(m) - 1;
      d.ring_ids[(size_t)slot * N + q] = i;
      d.ring_te[(size_t)slot * N + q] = d.te[i];
      d.last_spike_ms[i] = (int32_t)t;
      if (d.row_ptr[i + 1] == d.row_ptr[i]) atomicOr(d.flags, F_NO_TARGET);
    }
  }
}

// The compaction alone, where plasticity reads the last spike times before
// and in the delivery.
__global__ void __launch_bounds__(DELIVER_THREADS) compact_small_kernel(Dev d) {
  __shared__ SmallSpikes s;
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  compact_small(d, s, *d.t);
}

// FUSED: the step's compaction is done here (compact_small).
template <bool FUSED>
__device__ static inline void deliver(const Dev &d, SmallSpikes *sp) {
  const NetConst *net = d.net;
  const uint32_t t = *d.t, N = net->N, D = net->D, cap = net->ev_cap;
  __shared__ uint32_t s_pre[RING_SLOTS + 1];
  __shared__ uint32_t s_off[DELIVER_THREADS / 32][33];     // per warp: exclusive prefix of lengths
  __shared__ unsigned long long s_beg[DELIVER_THREADS / 32][32];
  __shared__ uint32_t s_key[DELIVER_THREADS / 32][32];
  if (threadIdx.x < 32) {   // counts of the slots, then their prefix
    for (uint32_t dd = threadIdx.x; dd < D; dd += 32)
      s_pre[dd + 1] = FUSED && dd == 0 ? 0u : d.ring_cnt[(t + RING_SLOTS - dd) % RING_SLOTS];
  }
  if (FUSED) compact_small(d, *sp, t);
  else __syncthreads();
  if (threadIdx.x == 0) {
    if (FUSED) s_pre[1] = sp->cnt;
    uint32_t acc = 0;
    s_pre[0] = 0;
    for (uint32_t dd = 1; dd <= D; dd++) s_pre[dd] = acc += s_pre[dd];
  }
  __syncthreads();
  const uint32_t total = s_pre[D];
  const uint32_t lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
  const bool stdp = net->stdp_on && t >= net->start_pl && t <= net->stop_pl;
  const float w2f = net->w2f;
  uint32_t *off = s_off[wb];
  unsigned long long *bg = s_beg[wb];
  uint32_t *ky = s_key[wb];
  unsigned long long my_events = 0;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  // items per warp at a time: 32, or fewer when they would leave warps idle
  const uint32_t ipw = max(1u, min(32u, (total + nwarps - 1) / nwarps));
  for (uint32_t w0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * ipw; w0 < total; w0 += nwarps * ipw) {
    const uint32_t w = w0 + lane;
    uint64_t beg = 0;
    uint32_t len = 0, key = 0;
    // the delay level of item w: the first dl with s_pre[dl + 1] > w.  The
    // warp finds w0's by a binary search over the D levels (some of them
    // empty), the same for every lane; each lane steps on from there (its 32
    // items span few levels)
    uint32_t dl = 0, hi = D - 1;
    while (dl < hi) {
      const uint32_t mid = (dl + hi) >> 1;
      if (s_pre[mid + 1] <= w0) dl = mid + 1; else hi = mid;
    }
    if (w < total && lane < ipw) {
      while (s_pre[dl + 1] <= w) dl++;
      const uint32_t q = w - s_pre[dl];
      const uint32_t slot = (t + RING_SLOTS - dl) % RING_SLOTS;
      const uint32_t P = FUSED && dl == 0 ? sp->id(q, (N + 31) / 32) : d.ring_ids[(size_t)slot * N + q];
      const uint16_t *so = d.sub_off + (size_t)P * (D + 1);
      const uint32_t a = so[dl], b = so[dl + 1];
      beg = d.row_ptr[P] + a;
      len = b - a;
      key = ((D - 1 - dl) << 25) | q;
    }
    uint32_t incl = len;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
    const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
    __syncwarp();
    off[lane] = incl - len;
    if (lane == 31) off[32] = tot;
    bg[lane] = beg;
    ky[lane] = key;
    my_events += len;
    __syncwarp();
    // the concatenated segments, element e = lane + 32 * i, in batches of
    // DELIVER_UNROLL per lane: the next batch's synapse loads are issued
    // while this batch's slot atomics are in flight
    uint32_t sg = 0;
    uint64_t k[DELIVER_UNROLL];
    uint32_t kk[DELIVER_UNROLL], jj[DELIVER_UNROLL];
    float wf[DELIVER_UNROLL];
#define DELIVER_FETCH(E0, K, KK, JJ, WF)                       \
  _Pragma("unroll") for (int u = 0; u < DELIVER_UNROLL; u++) { \
    const uint32_t e = (E0) + 32u * u + lane;                 \
    KK[u] = 0xFFFFFFFFu;                                      \
    if (e < tot) {                                            \
      while (off[sg + 1] <= e) sg++;                          \
      K[u] = bg[sg] + (e - off[sg]);                          \
      KK[u] = ky[sg];                                         \
      JJ[u] = __ldg(&d.post[K[u]]);                           \
      WF[u] = ((float)__ldg(&d.w16[K[u]])) * w2f;             \
    }                                                         \
  }
    DELIVER_FETCH(0u, k, kk, jj, wf);
    for (uint32_t e0 = 0; e0 < tot; e0 += 32u * DELIVER_UNROLL) {
      uint32_t sl[DELIVER_UNROLL];
#pragma unroll
      for (int u = 0; u < DELIVER_UNROLL; u++)
        if (kk[u] != 0xFFFFFFFFu) sl[u] = atomicAdd(&d.ev_cnt[jj[u]], 1u);
      uint64_t nk[DELIVER_UNROLL];
      uint32_t nkk[DELIVER_UNROLL], njj[DELIVER_UNROLL];
      float nwf[DELIVER_UNROLL];
      DELIVER_FETCH(e0 + 32u * DELIVER_UNROLL, nk, nkk, njj, nwf);
#pragma unroll
      for (int u = 0; u < DELIVER_UNROLL; u++)
        if (kk[u] != 0xFFFFFFFFu) deliver_event(d, net, k[u], kk[u], t, stdp, cap, jj[u], wf[u], sl[u]);
#pragma unroll
      for (int u = 0; u < DELIVER_UNROLL; u++) {
        k[u] = nk[u];
        kk[u] = nkk[u];
        jj[u] = njj[u];
        wf[u] = nwf[u];
      }
    }
#undef DELIVER_FETCH
    __syncwarp();
  }
  for (int o = 16; o > 0; o >>= 1) my_events += __shfl_down_sync(0xffffffffu, my_events, o);
  if (lane == 0 && my_events) atomicAdd(d.events, my_events);
}

__global__ void __launch_bounds__(DELIVER_THREADS) deliver_kernel(Dev d) {
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  deliver<false>(d, nullptr);
}
__global__ void __launch_bounds__(DELIVER_THREADS) deliver_small_kernel(Dev d) {
  __shared__ SmallSpikes s;
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  deliver<true>(d, &s);
}

// Step 3: the Poisson bath (regularDynamicTimeStep, DPSNN_neuron_sim.c:604-640,
// getPoissonLapse :844-865).  Each rank owns one serial ran3 stream that its
// neurons consume in index order: a neuron whose next bath time is before
// t+1 takes one pair of draws (LUT index, lapse) per event, the first c pairs
// at which nextBath + sum of c lapses * invNuExt reaches t+1.  Where a
// neuron's pairs start is known only once every earlier neuron of the rank is
// decided: a chain over the rank's neurons, which bounds the kernel.
//
// One block per rank.  The block meets at one barrier per round; in a round
//   mappers     (warps 0-7) decide up to 128 neurons, 16 each: a mapper walks
//               its 16 neurons from each of 32 candidate starts around the
//               predicted one, a candidate per lane (bath_map).  The chain is
//               then eight lookups (bath_compose, by every mapper for
//               itself): each segment's end for its actual start.  A start outside a segment's window
//               ends the round there;
//   preparers   (8, 13) read the next neurons, turn each one's budget (t+1 -
//               nextBath)/invNuExt into integer bounds, and queue those with
//               an event this step (the others pass at once);
//   converters  (9-11) turn 192 pairs of raw draws at a time into (LUT index,
//               lapse) and extend q[], the running sum of the lapses in
//               2^-20 units (integers mod 2^32);
//   emitters    (12, 14) write the events of the neurons decided in the round
//               before, a lane per neuron, each replaying its neuron in the
//               reference's arithmetic;
//   generator   (15) extends the stream's raw draws, 96 at a time.
// Warps go to the SM's four schedulers by index: the roles are spread so that
// each scheduler has two mappers and about the same instructions beside them.
// Starts are predicted in time, not in pairs: a neuron's last event
// overshoots its budget by a lapse of mean and deviation 1, so after n
// neurons the start's q is the sum of the budgets and n, to within sqrt(n).
// The pairs' parity is that of the launch's first draw (only draws past a
// neuron's maxExternCurrentCount cap are single; after one the pairs start
// afresh at the new position), so only every other draw becomes a lapse.
// What bounds it: the latency of a round (a mapper's 16 dependent steps, then
// the chain), not issue slots (less than half used).  Segments of 16: a round costs
// about 3000 cycles beside its steps, and at more neurons per segment the last
// windows miss too often.  Measured per step (one B200), against the form
// before, in which ten warps built tables of 64 candidate starts for every
// neuron and every draw of both parities was converted: 53 us from 173 for one
// rank of 1600 neurons, 87 from 300 for 11 ranks of 2743, 207 from 679 for 192
// ranks of 3750 beside the update (44 of the 148 SMs hold two ranks), 16 from
// 67 for one of 100.  At lower rates a step of 1600 neurons takes 24, 31, 31, 31
// and 32 us for 0.01, 0.06, 0.25, 0.5 and 0.7 events per neuron and ms; with the
// caps below 16 that go with them left to the walk it took 29, 45, 126, 217 and
// 275.  One warp deciding neuron by neuron (a shared read, a vote
// and a count each) took 85 cycles per neuron alone and 215 beside the other
// warps; this takes about 60.
#define BATH_THREADS 512       // 16 warps: roles above
#define BATH_SEG 16            // neurons per mapper
#define BATH_SEGS 8            // mappers
#define BATH_SB (BATH_SEG * BATH_SEGS)
#define BATH_NC 32             // candidate starts of a segment: 4 deviations on either side of the second
                               // one's, 1.5 of the last one's (a third of the rounds lose a segment or two)
#define BATH_PAIRS 2048        // pairs resident: two rounds behind (the emitters' and the walk's own), and ahead
#define BATH_MIRROR 1024       // the ring's first words again past its end: a round's reads do not wrap
#define BATH_RAW (2 * BATH_PAIRS)   // raw draws resident
#define BATH_HIST 256          // raw draws kept between launches (the generator reads 220 back),
#define BATH_KEEP 640          // and as many of those ahead as there are, up to 384: the first round converts them
#define BATH_ACT 512           // queued neurons: those being emitted, decided and prepared
#define BATH_CONV 192          // pairs converted at a time: 2 per lane of three warps
#define BATH_AHEAD 960         // pairs converted ahead of the decided ones, at most
#define BATH_MAX_EXT 121       // largest maxExternCurrentCount supported
#define BATH_UNDECIDED 0xFFFFu // a segment's entry: to be walked
#define BATH_NOT_YET 0xFFFEu   // or to be mapped in the next round
static_assert(BATH_AHEAD + BATH_CONV + BATH_MAX_EXT + 64 < BATH_PAIRS,
              "the walk always finds its next neuron's pairs converted or room for them");
static_assert(BATH_SEG == 16 && BATH_NC == 32, "packed counts are 16 nibbles; a candidate per lane");
static_assert(3 * BATH_SB + 64 <= BATH_ACT, "room to queue 64 neurons while two rounds' are held and one is ahead");

// What a round starts from; each field is written during the round before by
// one warp, into the other copy.
struct BathCtl {
  uint32_t m, a;        // walk: next pair, next queued neuron
  uint32_t rebase;      // walk: the pairs start afresh at this draw after this round (0: no)
  uint32_t done;        // walk: nothing is left to decide or to emit
  uint32_t act_end;     // preparers: queued neurons
  uint32_t prep_done;   // preparers: every neuron of the rank seen
  uint32_t conv_end;    // converters: pairs [0, conv_end) converted, from draw `base`
  uint32_t raw_end;     // generator: raw draws [.., raw_end)
  uint32_t sb_a, sb_n;  // walk: the neurons to emit
  uint32_t slow;        // walk: its segments walked neuron by neuron (bits)
  uint32_t keep;        // walk: first pair of the neurons being emitted
  uint32_t base, out;   // walk: first draw of pair 0, events before it
};

#define LOG_TAB_0 48
#define LOG_TAB_N 49
struct BathSmem {
  uint32_t raw[BATH_RAW];           // draw n at n % BATH_RAW
  uint32_t q[BATH_PAIRS + BATH_MIRROR];   // sum of the lapses of the pairs before k, at k % BATH_PAIRS
  float lap[BATH_PAIRS];
  uint8_t idx[BATH_PAIRS];
  double a_nb[BATH_ACT], a_inv[BATH_ACT];   // queued neuron a at a % BATH_ACT
  uint4 a_b[BATH_ACT + BATH_SEG];   // bounds lo and hi - lo, cap; mirrored at the end
  uint32_t a_id[BATH_ACT];          // neuron of the rank, its sub-population in the top bits
  uint32_t a_t[BATH_ACT];           // expected q advance of the queued neurons before a (2^-20 units)
  uint2 pack[BATH_SEGS][BATH_NC];   // a segment's counts less one, a nibble per neuron, by candidate
  uint16_t end[BATH_SEGS][BATH_NC + 2];   // its end, from win[], or BATH_UNDECIDED, BATH_NOT_YET
  uint4 win[BATH_SEGS / 4];         // pair of candidate 0
  uint2 e_pack[2][BATH_SEGS];       // decided segments by round parity: counts, first pairs
  uint32_t e_start[2][BATH_SEGS];
  uint32_t prep_n[2], prep_t[2];    // preparers: each one's queued neurons and their expected advance
  uint32_t start[2][BATH_SB + 1];   // first pairs of the neurons of the slow segments, then their end
  double near[256];                 // Dev::fix_near
  double2 log_tab[LOG_TAB_N];       // Dev::log_tab
  uint32_t conv_tot[3];             // converters: lapse sums of the warps' pairs
  uint32_t slots;                   // the rank's event slots (bath_slots)
  BathCtl ctl[2];
};

// The correctly rounded float log in the rare case that the double one does
// not decide it.  Inlined: out of line the kernel spills more (68 bytes from
// 52), and one rank of 1600 neurons takes 55.9 us per step against 53.1.
__device__ __forceinline__ static float logf_cr_undecided(float x) { return (float)log_cr((double)x); }

// The double of a normal float's bits (no conversion instruction: those have a
// quarter of the rate).
__device__ __forceinline__ double double_of_bits(uint32_t fb) {
  return __hiloint2double((int)((fb & 0x80000000u) | (((fb & 0x7FFFFFFFu) >> 3) + 0x38000000u)), (int)(fb << 29));
}

// Lapses of K raw draws (getPoissonLapse, DPSNN_neuron_sim.c:844-865): -logf
// of the host C library on (0,1].
//  - The double log: x = 2^e m, m in [0.75,1.5), i = round(64 m), log x =
//    e ln 2 + log(i/64) + log1p(r), r = m (64/i) - 1 in one rounding, |r| <=
//    1/96, by the series through r^8; an error below 2^-49 of the result (for
//    x near 1, i = 64 and the first two terms are zero).
//  - Inputs where the C library differs from the correctly rounded float all
//    have a logarithm close to a rounding midpoint: nearer than the furthest
//    of them in the result's binade (near) a bit per float says whether x is
//    one.  Its value is then the float on the midpoint's other side, as that of
//    any library with an error below one ulp is (a search of the table here took
//    up to eight dependent loads, in half of a warp's conversions); where the
//    table loaded has another value, SEARCH finds it.
// Each step is done for all K draws before the next, so that their loads are
// in flight together.  Run over all 10^9 draws, its lapses are the C library's,
// bit for bit.
template <int K, bool SEARCH>
__device__ static inline void bath_lapse(const Dev &d, const BathSmem &s, const uint32_t (&mj)[K], float (&lap)[K]) {
  uint32_t fb[K], key[K], bw[K];
  double r[K];
#pragma unroll
  for (int i = 0; i < K; i++) {
    // u = mj / MBIG as the reference rounds it; x = (float)(1 - u)
    const double u = (__hiloint2double(0x43300000, (int)mj[i]) - 0x1p52) * (1.0 / (double)MBIG);
    key[i] = __float_as_uint((float)(1.0 - u));
    const int e = (int)(key[i] - 0x3F400000u) >> 23;
    const uint32_t mb = key[i] - ((uint32_t)e << 23);
    const double2 c = s.log_tab[(int)(__uint_as_float(mb) * 64.0f + 0.5f) - LOG_TAB_0];
    const double z = fma(double_of_bits(mb), c.x, -1.0);
    double q = fma(z, -1.0 / 8, 1.0 / 7);
    q = fma(z, q, -1.0 / 6);
    q = fma(z, q, 1.0 / 5);
    q = fma(z, q, -1.0 / 4);
    q = fma(z, q, 1.0 / 3);
    q = fma(z, q, -1.0 / 2);
    const double ef = __hiloint2double(0x43300000, (int)(0x80000000u + (uint32_t)e)) - (0x1p52 + 0x1p31);
    const double y = fma(ef, 0x1.62e42fefa39efp-1, c.y) + fma(z * z, q, z);
    fb[i] = __float_as_uint((float)y);
    r[i] = y - double_of_bits(fb[i]);
  }
#pragma unroll
  for (int i = 0; i < K; i++) {
    bw[i] = 0;
    if (fabs(r[i]) >= s.near[(fb[i] >> 23) & 0xFFu] || (fb[i] & 0x7FFFFFu) == 0)
      bw[i] = __ldg(&d.fix_bitmap[(key[i] - 0x30000000u) >> 5]);   // 1e-9 <= x <= 1
  }
#pragma unroll
  for (int i = 0; i < K; i++) {
    // within 2^-18 of a midpoint (2^-24 of the binade, or 2^-25 below a power
    // of two): the rounding needs more digits
    const uint32_t E = (fb[i] >> 23) & 0xFFu;
    const double half = __hiloint2double((int)((E - 24 + 896) << 20), 0);
    if (fabs(r[i]) > half * (1.0 - 0x1p-18) ||
        ((fb[i] & 0x7FFFFFu) == 0 && fabs(r[i]) > 0.5 * half * (1.0 - 0x1p-18))) {
      if (E) {
        const float f = logf_cr_undecided(__uint_as_float(key[i]));
        r[i] += double_of_bits(fb[i]) - double_of_bits(__float_as_uint(f));
        fb[i] = __float_as_uint(f);
      }
    }
    if ((bw[i] >> ((key[i] - 0x30000000u) & 31)) & 1u) {
      if (SEARCH) {
        const NetConst *net = d.net;
        uint32_t lo = 0, hi = net->fix_n - 1;   // the key is listed
        while (lo < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (net->fix_keys[mid] < key[i]) lo = mid + 1; else hi = mid;
        }
        fb[i] = net->fix_vals[lo];
      } else {
        fb[i] += r[i] < 0 ? 1u : 0xFFFFFFFFu;   // f < 0: the next float below has the next bit pattern
      }
    }
    lap[i] = -__uint_as_float(fb[i]);
  }
}

__device__ static inline uint32_t lap_fixed(float lap) {
  return __float2uint_rn(lap * 0x1p20f);   // an exact product; lap < 2^11: no overflow
}

// Integer bounds on the lapse sum, in 2^-20 units, for one neuron with an
// event this step (inv > 0, nb < T1): a fixed-point sum F of c lapses below
// lo means the reference's sequential nextBath after c events is certainly <
// t+1, at or above hi1 certainly >= t+1.  E1 bounds the rounding of that
// sequential sum (c <= 32 additions, |values| < |T1| + 42 invNuExt, and t+1 -
// nextBath); 2^-16 bounds the rounding of F (32 terms of at most 2^-21); the
// 2^-30 relative margin covers the bound's own arithmetic.  Both are clamped
// to 32 bits (F < 2^30).
__device__ static inline void bath_bounds(double T1, double nb, double inv, uint32_t &lo, uint32_t &hi1) {
  const double E1 = 0x1p-44 * (fabs(T1) + fabs(nb) + 1.0 + 32.0 * inv);
  const double bud = (T1 - nb) / inv;
  const double mg = 1.001 * (double)((float)E1 / (float)inv) + 0x1p-16 + 0x1p-30 * (bud + 1.0);
  lo = __double2uint_rd(fmax((bud - mg) * 0x1p20, 0.0));   // the conversions clamp at 2^32 - 1
  hi1 = __double2uint_ru((bud + mg) * 0x1p20);
  hi1 += hi1 != 0xFFFFFFFFu;
}

// Draws past a neuron's cap, single ones (rare): from draw n on, until
// nextBath reaches T1; returns the position after them, 0 when a draw that
// is not generated yet is needed.
template <bool SEARCH>
__device__ static inline uint32_t bath_singles(const Dev &d, const BathSmem &s, uint32_t n, uint32_t raw_end,
                                               double inv, double T1, double &v) {
  do {
    if (n >= raw_end) return 0;
    const uint32_t mj[1] = {s.raw[n % BATH_RAW]};
    float lp[1];
    bath_lapse<1, SEARCH>(d, s, mj, lp);
    v += (double)lp[0] * inv;
    n++;
  } while (v < T1);
  return n;
}

// One neuron of a mapper's segment from its lane's candidate (pair p, whose
// q is qm): 1 + the number of sums of 1..16 lapses below lo, by fours, then
// within the four.  Returns the count less one.  LOW: a neuron's cap may be below
// sixteen.
template <bool LOW>
__device__ __forceinline__ uint32_t bath_count(const BathSmem &s, const uint4 &k, uint32_t &p, uint32_t &qm,
                                               uint32_t &bad) {
  const uint32_t T = qm + k.x;
  const uint32_t x =
      p + 4 * (((s.q[p + 4] - T) >> 31) + ((s.q[p + 8] - T) >> 31) + ((s.q[p + 12] - T) >> 31));
  const uint32_t y1 = s.q[x + 1] - T, y2 = s.q[x + 2] - T, y3 = s.q[x + 3] - T, y4 = s.q[x + 4] - T;
  const uint32_t e = x + (y1 >> 31) + (y2 >> 31) + (y3 >> 31) + (y4 >> 31), c = e - p;
  // the first sum not below lo, less lo: the negative ones are large unsigned
  const uint32_t over = min(min(y1, y2), min(y3, y4));
  // undecided, in bad's top bit: the sum lies between lo and hi, none of the
  // sixteen reaches lo (over is then a negative number), or the count is past
  // the neuron's cap (k.z)
  bad |= over - k.y;
  if (LOW) bad |= ~(c - k.z);
  qm = T + over;
  p = e + 1;
  return c;
}

// Mapper w: its segment's end and counts from every candidate start.
template <bool LOW>
__device__ static inline void bath_map(BathSmem &s, const BathCtl &cur, uint32_t w, uint32_t lane) {
  const uint32_t A = BATH_ACT - 1, a0 = cur.a + BATH_SEG * w;
  if (a0 >= cur.act_end || cur.rebase) return;
  const uint32_t n = min(cur.act_end - a0, (uint32_t)BATH_SEG);
  const uint32_t b = cur.m & (BATH_PAIRS - 1), lim = cur.conv_end - cur.m;   // q[b + i]: pair m + i; stale past lim
  uint32_t win = 0;   // candidate 0, from m
  if (w) {
    // the pair at the predicted time, to within two: pairs have density 1, so
    // it lies within a few sqrt(dt) of dt pairs on
    const uint32_t dt = s.a_t[a0 & A] - s.a_t[cur.a & A], T = s.q[b] + dt;
    const uint32_t first = max(min(dt >> 20, 600u), 64u) - 64, at = first + 4 * lane;
    const uint32_t pred =
        first + 4 * __popc(__ballot_sync(0xffffffffu, at <= lim && (int32_t)(s.q[b + at] - T) < 0)) - 2;
    win = max(pred, (uint32_t)BATH_NC / 2) - BATH_NC / 2;
  }
  uint32_t p = b + win + lane, qm = s.q[p], bad = 0;
  uint2 pk = make_uint2(0, 0);
  const uint4 *k = &s.a_b[a0 & A];   // mirrored past the ring's end
  if (n == BATH_SEG) {
#pragma unroll
    for (int j = 0; j < 8; j++) pk.x += bath_count<LOW>(s, k[j], p, qm, bad) << (4 * j);
#pragma unroll
    for (int j = 0; j < 8; j++) pk.y += bath_count<LOW>(s, k[8 + j], p, qm, bad) << (4 * j);
  } else {
#pragma unroll 1
    for (uint32_t j = 0; j < n; j++) {
      const uint32_t c = bath_count<LOW>(s, k[j], p, qm, bad) << (4 * (j & 7));
      if (j < 8) pk.x += c; else pk.y += c;
    }
  }
  // an end within 16 pairs of the converted ones may rest on stale words
  const uint32_t e = p - b;
  s.end[w][lane] = (uint16_t)(e + 16 > lim ? BATH_NOT_YET : (int32_t)bad < 0 ? BATH_UNDECIDED : e - win);
  s.pack[w][lane] = pk;
  if (lane == 0) {
    reinterpret_cast<uint32_t *>(s.win)[w] = cur.m + win;
    s.end[w][BATH_NC] = BATH_NOT_YET;
  }
}

// Every mapper, the segments mapped: the chain over them.  Each hands its own
// segment over if the chain reaches it decided; warp 0 also writes the next
// round's start.  A segment with no decided entry at its start runs neuron
// by neuron (warp 0) and ends the round: the sums of 1..32 lapses by lane and
// a vote, or the reference's loop.
template <bool SEARCH>
__device__ static inline void bath_compose(const Dev &d, BathSmem &s, const BathCtl &cur, BathCtl &nxt, uint32_t par,
                                           double T1, uint32_t w, uint32_t lane) {
  const uint32_t M = BATH_PAIRS - 1, A = BATH_ACT - 1;
  const uint32_t left = cur.rebase ? 0u : min(cur.act_end - cur.a, (uint32_t)BATH_SB);
  const uint32_t nseg = (left + BATH_SEG - 1) / BATH_SEG;
  const uint4 wa = s.win[0], wb = s.win[1];
  const uint32_t win[BATH_SEGS] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
  // a start outside a segment's window finds the sentinel, and so does, from
  // there on, every later segment
  uint32_t st[BATH_SEGS + 1], undec = 0;
  st[0] = cur.m;
#pragma unroll
  for (uint32_t g = 0; g < BATH_SEGS; g++) {
    const uint32_t e = s.end[g][min(st[g] - win[g], (uint32_t)BATH_NC)];
    undec |= (uint32_t)(e >= BATH_NOT_YET) << g;
    st[g + 1] = win[g] + e;
  }
  const uint32_t stop_g = min((uint32_t)__ffs(undec) - 1u, nseg);
  uint32_t m = st[0], my_m = st[0];
#pragma unroll
  for (uint32_t g = 1; g <= BATH_SEGS; g++) {
    if (g == stop_g) m = st[g];
    if (g == w) my_m = st[g];
  }
  if (w < stop_g && lane == 0) {
    s.e_start[par][w] = my_m;
    s.e_pack[par][w] = s.pack[w][my_m - reinterpret_cast<const uint32_t *>(s.win)[w]];
  }
  if (w) return;
  uint32_t n_done = min(stop_g * BATH_SEG, left), rebase = 0, slow = 0;
  if (stop_g < nseg && s.end[stop_g][min(m - reinterpret_cast<const uint32_t *>(s.win)[stop_g], (uint32_t)BATH_NC)] == BATH_UNDECIDED) {
    slow = 1u << stop_g;
    const uint32_t n_end = min(n_done + BATH_SEG, left), lim = cur.conv_end;
    while (n_done < n_end && !rebase) {
      const uint32_t a = (cur.a + n_done) & A, mx = s.a_b[a].z, lo = s.a_b[a].x;
      if (m + max(33u, mx + 1) > lim) break;   // its pairs are not converted yet
      uint32_t c = 0;
      const uint32_t F = s.q[(m + 1 + lane) & M] - s.q[m & M];
      const uint32_t mm = __popc(__ballot_sync(0xffffffffu, F < lo));
      if (mm < min(32u, mx) && __shfl_sync(0xffffffffu, F, mm) - lo >= s.a_b[a].y) c = mm + 1;
      if (!c) {   // the reference's loop (DPSNN_neuron_sim.c:604-640)
        const double inv = s.a_inv[a];
        double v = s.a_nb[a];
        do {
          v += (double)s.lap[(m + c) & M] * inv;
          c++;
        } while (v < T1 && c < mx);
        if (v < T1) {
          rebase = bath_singles<SEARCH>(d, s, cur.base + 2 * (m + c), cur.raw_end, inv, T1, v);
          if (!rebase) break;   // draws not generated yet
        }
      }
      if (lane == 0) {
        s.start[par][n_done] = m;
        s.start[par][n_done + 1] = m + c;
      }
      m += c;
      n_done++;
    }
  }
  const uint32_t a = cur.a + n_done;
  if (lane == 0) {
    nxt.sb_a = cur.a;
    nxt.sb_n = a - cur.a;
    if (cur.out + m > s.slots) {   // pairs and events have the same count: no room for this round's
      atomicOr(d.flags, F_BATH_DRAWS);
      nxt.sb_n = 0;
    }
    nxt.slow = slow;
    nxt.a = a;
    nxt.rebase = rebase;
    nxt.done = cur.prep_done && a == cur.act_end && n_done == 0 && !cur.rebase;
    if (cur.rebase) {   // the neurons before it are emitted in this round
      nxt.m = nxt.keep = 0;
      nxt.base = cur.rebase;
      nxt.out = cur.out + cur.m;
    } else {
      nxt.m = m;
      nxt.keep = cur.m;
      nxt.base = cur.base;
      nxt.out = cur.out;
    }
  }
}

// Sum of the nibbles of x (at most 8 x 15).
__device__ static inline uint32_t nibble_sum(uint32_t x) {
  return (((x & 0x0F0F0F0Fu) + ((x >> 4) & 0x0F0F0F0Fu)) * 0x01010101u) >> 24;
}

// SEARCH: the logf table has values to search for (bath_lapse).  LOW: a neuron's
// cap is below sixteen (rates below 0.75); the comparison that goes with it makes
// 24x24 steps of 6 events per neuron 1.2 % longer, so that others go without.
template <bool SEARCH, bool LOW>
__global__ void __launch_bounds__(BATH_THREADS, 2) bath_kernel(Dev d) {
  extern __shared__ __align__(16) unsigned char bath_smem_raw[];
  BathSmem &s = *reinterpret_cast<BathSmem *>(bath_smem_raw);
  const NetConst *net = d.net;
  const uint32_t h = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t M = BATH_PAIRS - 1, A = BATH_ACT - 1;
  const uint32_t t = d.bath_t[h], locN = net->locN, i0 = h * locN;
  const double T1 = (double)((double)t + 1.0);
  const uint32_t ev_base = (uint32_t)d.bath_rank_base[h];
  // draws of this launch are numbered from BATH_HIST; the ones before are the
  // rank's kept history
  const uint32_t kept = d.bath_kept[h];
  for (uint32_t n = tid; n < kept; n += BATH_THREADS) s.raw[n] = d.bath_hist[(size_t)h * BATH_KEEP + n];
  for (uint32_t r = tid; r < 256; r += BATH_THREADS) s.near[r] = d.fix_near[r];
  for (uint32_t r = tid; r < LOG_TAB_N; r += BATH_THREADS) s.log_tab[r] = d.log_tab[r];
  if (tid == 0) {
    s.q[0] = s.q[BATH_PAIRS] = 0;
    s.a_t[0] = 0;
    s.slots = (uint32_t)(d.bath_rank_base[h + 1] - d.bath_rank_base[h]);
    BathCtl c = {};
    c.base = BATH_HIST;
    c.raw_end = kept;
    s.ctl[0] = c;
  }
  // the preparers' next neurons, loaded an iteration ahead
  uint32_t p_i = 0, p_t = 0, x_mx = 0, x_sub = 0;
  double x_nb = 0, x_inv = 0;
  if (warp == 8 || warp == 13) {
    const uint32_t i = lane + (warp == 8 ? 0 : 32);
    if (i < locN) {
      x_nb = d.nb_prev[i0 + i];
      x_inv = d.inv_nu[i0 + i];
      x_mx = d.max_ext[i0 + i];
      x_sub = d.sub[i0 + i];
    }
  }
  __syncthreads();
  // a round decides a neuron, or brings its draws closer; the limit is far
  // beyond what a launch takes
  const uint32_t max_rounds = 64 + 16 * locN;
  uint32_t r = 0;
  for (;; r++) {
    const BathCtl &cur = s.ctl[r & 1];
    BathCtl &nxt = s.ctl[(r + 1) & 1];
    if (cur.done || r == max_rounds) break;
    if (warp < BATH_SEGS) {
      bath_map<LOW>(s, cur, warp, lane);
      asm volatile("bar.sync 1, 256;" ::: "memory");   // the mappers
      bath_compose<SEARCH>(d, s, cur, nxt, r & 1, T1, warp, lane);
    } else if (warp == 15) {
      // x[n] = x[n-55] - x[n-24] mod 1e9, applied four times over: x[n] = x[n-96] - 4 x[n-127] + 6 x[n-158]
      // - 4 x[n-189] + x[n-220], so that 96 draws follow from the ones before them at once; keeping BATH_HIST
      // draws behind the neurons being emitted
      uint32_t n = cur.raw_end;
      const uint32_t room =
          min(cur.base + 2 * (cur.m + BATH_AHEAD + BATH_CONV), cur.base + 2 * cur.keep + BATH_RAW - BATH_HIST);
      for (int g = 0; g < 8 && n + 96 <= room; g++, n += 96) {
        uint32_t x[3];
#pragma unroll
        for (int v = 0; v < 3; v++) {
          const uint32_t k = n + lane + 32 * v;
          const int32_t x3 = 2 * (int32_t)s.raw[(k - 158) % BATH_RAW];   // every term below is within 2 MBIG of 0
          int32_t y = (int32_t)(s.raw[(k - 96) % BATH_RAW] + s.raw[(k - 220) % BATH_RAW]) - x3;
          int32_t z = (int32_t)(s.raw[(k - 127) % BATH_RAW] + s.raw[(k - 189) % BATH_RAW]) - x3;
          if (y < 0) y += MBIG;
          if (y < 0) y += MBIG;
          if (y >= MBIG) y -= MBIG;
          if (z < 0) z += MBIG;
          if (z < 0) z += MBIG;
          z = 2 * (z >= MBIG ? z - MBIG : z);
          if (z >= MBIG) z -= MBIG;
          y -= 2 * z;   // x = y - 4 z
          if (y < 0) y += MBIG;
          if (y < 0) y += MBIG;
          x[v] = (uint32_t)y;
        }
#pragma unroll
        for (int v = 0; v < 3; v++) s.raw[(n + lane + 32 * v) % BATH_RAW] = x[v];
        __syncwarp();
      }
      if (lane == 0) nxt.raw_end = n;
    } else if (warp == 8 || warp == 13) {
      // ---- preparers, a warp per 32 neurons: enough queued for the next two rounds
      const uint32_t pw = warp == 8 ? 0 : 1;
      uint32_t e = cur.act_end;
      for (int g = 0; g < 4 && p_i < locN && e < cur.a + 2 * BATH_SB && e + 64 <= cur.sb_a + BATH_ACT; g++, p_i += 64) {
        const double nb = x_nb, inv = x_inv;
        const uint32_t mx = x_mx, sub = x_sub, i = p_i + 32 * pw + lane;
        if (i + 64 < locN) {
          x_nb = d.nb_prev[i0 + i + 64];
          x_inv = d.inv_nu[i0 + i + 64];
          x_mx = d.max_ext[i0 + i + 64];
          x_sub = d.sub[i0 + i + 64];
        }
        // a bath of rate zero (invNuExt infinite) asks for an event and has no slot for one
        const bool due = i < locN && inv > 0 && nb < T1, act = due && mx > 0;
        if (due && !act) atomicOr(d.flags, F_BATH_DRAWS);
        const uint32_t bal = __ballot_sync(0xffffffffu, act);
        uint32_t lo = 0, hi1 = 0;
        if (act) bath_bounds(T1, nb, inv, lo, hi1);
        const uint32_t tv = act ? min(lo, 64u << 20) + (1u << 20) : 0u;
        uint32_t incl = tv;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t sum = __shfl_sync(0xffffffffu, incl, 31);
        s.prep_n[pw] = __popc(bal);
        s.prep_t[pw] = sum;
        asm volatile("bar.sync 3, 64;" ::: "memory");   // the two preparers
        const uint32_t n0 = s.prep_n[0], n1 = s.prep_n[1], t0 = s.prep_t[0], t1 = s.prep_t[1];
        if (act) {
          const uint32_t k = (e + pw * n0 + __popc(bal & ((1u << lane) - 1))) & A;
          s.a_nb[k] = nb;
          s.a_inv[k] = inv;
          const uint4 ab = make_uint4(lo, hi1 - lo, mx, 0u);
          s.a_b[k] = ab;
          if (k < BATH_SEG) s.a_b[k + BATH_ACT] = ab;
          s.a_id[k] = i | (sub << 25);
          s.a_t[k] = p_t + pw * t0 + incl - tv;
        } else if (i < locN) {
          d.nb[i0 + i] = nb;
          d.bath_at[i0 + i] = make_uint2(0, 0);
        }
        p_t += t0 + t1;
        e += n0 + n1;
        asm volatile("bar.sync 3, 64;" ::: "memory");
      }
      if (pw == 0 && lane == 0) {
        s.a_t[e & A] = p_t;
        nxt.act_end = e;
        nxt.prep_done = p_i >= locN;
      }
    } else if (warp >= 9 && warp < 12) {
      // ---- converters: up to BATH_AHEAD pairs ahead, and no further than the last neurons need
      const uint32_t cw = warp - 9;
      uint32_t k0 = cur.conv_end;
      uint32_t want = cur.m + BATH_AHEAD;
      if (cur.prep_done) {
        const float left = (float)((s.a_t[cur.act_end & A] - s.a_t[cur.a & A]) >> 20);
        want = min(want, cur.m + 160 + (uint32_t)(left + 4.0f * sqrtf(left)));
      }
      const uint32_t room = min(cur.keep + BATH_PAIRS - 1, (cur.raw_end - cur.base) / 2);
      for (int g = 0; g < 3 && k0 < want && k0 + BATH_CONV <= room && !cur.rebase; g++, k0 += BATH_CONV) {
        const uint32_t kl = k0 + cw * 64 + 2 * lane, n = cur.base + 2 * kl;
        const uint32_t mi0 = s.raw[n % BATH_RAW], mi1 = s.raw[(n + 2) % BATH_RAW];
        const uint32_t mj[2] = {s.raw[(n + 1) % BATH_RAW], s.raw[(n + 3) % BATH_RAW]};
        float lp[2];
        bath_lapse<2, SEARCH>(d, s, mj, lp);
        const uint32_t f0 = lap_fixed(lp[0]), f1 = lap_fixed(lp[1]);
        uint32_t incl = f0 + f1;
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) s.conv_tot[cw] = incl;
        asm volatile("bar.sync 2, 96;" ::: "memory");   // the converters
        uint32_t qb = s.q[k0 & M] + incl;
        for (uint32_t w = 0; w < cw; w++) qb += s.conv_tot[w];
        const uint32_t k1 = (kl + 1) & M, k2 = (kl + 2) & M;
        s.lap[kl & M] = lp[0];
        s.lap[k1] = lp[1];
        // the LUT index draw (:617-619): (uint32_t)(u * 256) is mj / (MBIG / 256) for every draw
        s.idx[kl & M] = (uint8_t)(mi0 / (MBIG / 256));
        s.idx[k1] = (uint8_t)(mi1 / (MBIG / 256));
        s.q[k1] = qb - f1;
        s.q[k2] = qb;
        if (k1 < BATH_MIRROR) s.q[k1 + BATH_PAIRS] = qb - f1;
        if (k2 < BATH_MIRROR) s.q[k2 + BATH_PAIRS] = qb;
        asm volatile("bar.sync 2, 96;" ::: "memory");
      }
      if (cw == 0 && lane == 0) nxt.conv_end = cur.rebase ? 0u : k0;
    } else {
      // ---- emitters: the neurons of the last round
      const uint32_t par = (r + 1) & 1;
      for (uint32_t j = lane + (warp == 12 ? 0 : 32); j < cur.sb_n; j += 64) {
        const uint32_t a = (cur.sb_a + j) & A, g = j / BATH_SEG, jj = j % BATH_SEG;
        uint32_t m0, cnt;
        if ((cur.slow >> g) & 1u) {
          m0 = s.start[par][j];
          cnt = s.start[par][j + 1] - m0;
        } else {
          const uint2 pk = s.e_pack[par][g];
          const uint32_t word = jj < 8 ? pk.x : pk.y, sh = 4 * (jj & 7);
          m0 = s.e_start[par][g] + jj + nibble_sum(word & ((1u << sh) - 1)) + (jj < 8 ? 0u : nibble_sum(pk.x));
          cnt = ((word >> sh) & 15u) + 1;
        }
        const uint32_t id = s.a_id[a], i = i0 + (id & ((1u << 25) - 1)), at = ev_base + cur.out + m0;
        const double *lut = d.lut + 256 * (id >> 25);
        const double inv = s.a_inv[a];
        double v = s.a_nb[a];
        double2 *ev = d.bath_ev + at;
        for (uint32_t c = 0; c < cnt; c++) {
          ev[c] = make_double2(v, __ldg(&lut[s.idx[(m0 + c) & M]]));
          v += (double)s.lap[(m0 + c) & M] * inv;
        }
        if (v < T1) bath_singles<SEARCH>(d, s, cur.base + 2 * (m0 + cnt), cur.raw_end, inv, T1, v);
        d.nb[i] = v;
        d.bath_at[i] = make_uint2(at, cnt);
      }
    }
    __syncthreads();
  }
  const BathCtl &fin = s.ctl[r & 1];
  if (r == max_rounds) {
    if (tid == 0) atomicOr(d.flags, F_BATH_DRAWS);
    return;
  }
  // the history of the next launch: the draws before the first unused one
  const uint32_t pos = fin.base + 2 * fin.m, keep = BATH_HIST + min(fin.raw_end - pos, (uint32_t)(BATH_KEEP - BATH_HIST));
  for (uint32_t n = tid; n < keep; n += BATH_THREADS)
    d.bath_hist[(size_t)h * BATH_KEEP + n] = s.raw[(pos - BATH_HIST + n) % BATH_RAW];
  if (tid == 0) {
    d.bath_kept[h] = keep;
    d.bath_t[h] = t + 1;
  }
}

// LIFCADynamic, non-PerseoDyn branch (DPSNN_neuron_sim.c:664-824): lifca_pre
// below.
struct NeuronRegs {
  double v, c, tr, te;
  int fired;
};
// A sub-population's parameters, and 1/Tau, 1/TauC rounded to nearest: read
// from memory where they are used (LifcaMem), or kept in registers.  The
// thread-per-neuron kernel, whose events' buffers already fill its 64
// registers, takes 0.137 ms per 24x24 step with the first and 0.159 with the
// second; the merged streams' kernel (80 registers) 30 us per busy 16 000
// neurons with the second and 35 with the first.
struct LifcaMem {
  const NetConst *net;
  uint32_t s;
  __device__ double Tau() const { return net->Tau[s]; }
  __device__ double r_tau() const { return net->r_tau[s]; }
  __device__ double TauC() const { return net->TauC[s]; }
  __device__ double r_tauC() const { return net->r_tauC[s]; }
  __device__ double Theta() const { return net->Theta[s]; }
  __device__ double H() const { return net->H[s]; }
  __device__ double Tarp() const { return net->Tarp[s]; }
  __device__ double AlphaC() const { return net->AlphaC[s]; }
  __device__ double gC() const { return net->gC[s]; }
};
struct LifcaRegs {
  double tau, rtau, tauc, rtauc, theta, h, tarp, alphac, gc;
  __device__ LifcaRegs(const NetConst *net, uint32_t s)
      : tau(net->Tau[s]), rtau(net->r_tau[s]), tauc(net->TauC[s]), rtauc(net->r_tauC[s]), theta(net->Theta[s]),
        h(net->H[s]), tarp(net->Tarp[s]), alphac(net->AlphaC[s]), gc(net->gC[s]) {}
  __device__ double Tau() const { return tau; }
  __device__ double r_tau() const { return rtau; }
  __device__ double TauC() const { return tauc; }
  __device__ double r_tauC() const { return rtauc; }
  __device__ double Theta() const { return theta; }
  __device__ double H() const { return h; }
  __device__ double Tarp() const { return tarp; }
  __device__ double AlphaC() const { return alphac; }
  __device__ double gC() const { return gc; }
};
// a / b by b's reciprocal r (Markstein's theorem, IBM J. Res. Dev. 34, 1990:
// with r the reciprocal rounded to nearest and q within an ulp of a/b, q +
// r (a - b q) rounds to the quotient rounded to nearest; the first correction
// brings q = a r within an ulp).  Five operations and no branch, where a
// division's code has both; r = 0: b is out of the range in which nothing
// overflows or underflows on the way, and is divided by.  The same bits as a / b
// for 12 G pairs (a of 2^-60 to 2^30, b of 2^-40 to 2^40, an eighth of them with
// a float's or an almost full mantissa).
__device__ static inline double div_by(double a, double b, double r) {
  if (r == 0.0) return a / b;
  double q = a * r;
  q = fma(fma(-q, b, a), r, q);
  return fma(fma(-q, b, a), r, q);
}

// The coefficients of one update: deltaT = t - Tr.  They depend on event
// times only (Tr is the previous event's time), so the neuron run computes
// them one event ahead, off the dependent chain of v and c.
template <typename Par>
__device__ static inline void lifca_coeff(const Par &p, double deltaT, double &dth, double &rmh, double &poly) {
  dth = deltaT / 2;
  rmh = div_by(dth, p.Tau(), p.r_tau());
  const double rc = div_by(deltaT, p.TauC(), p.r_tauC());
  poly = 1 - rc + rc * rc / 2;
}

// The calcium decay over the refractory period: once per spike.  Out of line
// it is no faster.
__device__ __forceinline__ static double exp_cr_call(double x) { return exp_cr(x); }

// LIFCADynamic with the coefficients of this event computed ahead; the branch
// that leaves the refractory period moves deltaT, and recomputes them.
template <typename Par>
__device__ static inline void lifca_pre(const Par &p, NeuronRegs &n, double t, double I, double dth, double rmh,
                                        double poly) {
  double v = n.v, c = n.c, Te = n.te;
  const double Tr = n.tr, TFLES = t - Te;
  if (TFLES > p.Tarp()) {
    const double TrTe = Tr - Te;
    if (TrTe < p.Tarp()) {
      const double deltaT0 = t - Tr;
      c *= exp_cr_call(-(deltaT0 - TFLES + p.Tarp()) / p.TauC());
      lifca_coeff(p, TFLES - p.Tarp(), dth, rmh, poly);
    }
    v = v - v * rmh - p.gC() * c * dth;
    v = v - v * rmh - p.gC() * c * dth;
    c = c * poly;
    v += I;
    if (v >= p.Theta()) {
      v = p.H();
      c += p.AlphaC();
      Te = t;
      n.fired = 1;
    }
  } else {
    c = c * poly;
  }
  n.v = v;
  n.c = c;
  n.tr = t;
  n.te = Te;
}

__device__ static inline double event_time(const Dev &d, uint32_t key, uint32_t t, uint32_t D, uint32_t N) {
  uint32_t dl = (D - 1) - (key >> 25), q = key & ((1u << 25) - 1);
  double te = d.ring_te[(size_t)((t + RING_SLOTS - dl) % RING_SLOTS) * N + q];
  return (double)t + (te - floor(te));   // thisTimeStepF + modf(originalEmissionTime)
}

// Runs the merged event sequence of one neuron: synaptic events (sorted by
// (time, key)) merged with the bath events (time-ordered), synaptic first on
// equal times (mergeFunction, DPSNN_neuron_sim.c:391-421, called at :644-646).
// One event of a light neuron's insertion sort (thread-local): one 16-byte
// load or store per move.  The warp sorts keep separate arrays, whose 8- and
// 4-byte shared accesses conflict less at the network's short strides.
struct __align__(16) SortEv {
  double tau;
  uint32_t key;
  float val;
};

__device__ static inline bool sortev_gt(const SortEv &a, const SortEv &b) {
  return (a.tau > b.tau) || (a.tau == b.tau && a.key > b.key);
}


// be: its nb bath events ({time, input}; the bath's emitters look the input
// up, where the time, then the LUT index, then the LUT value were three
// dependent loads per event), in global memory or staged in shared memory.
template <typename Events>
__device__ static inline int run_neuron_ev(const Dev &d, uint32_t i, uint32_t t, const Events &evs, uint32_t ns,
                                           const double2 *be, uint32_t nb) {
  const LifcaMem par{d.net, d.sub[i]};
  double2 b0 = nb ? be[0] : make_double2(0.0, 0.0);
  NeuronRegs n;
  n.v = d.v[i];
  n.c = d.c[i];
  n.tr = d.tr[i];
  n.te = d.te[i];
  n.fired = 0;
  const double T0 = (double)t;
  uint32_t a = 0, b = 0;
  // the merge's next event (time, input)
  auto next = [&](double &ct, double &I) -> bool {
    if (a < ns && (b >= nb || evs.time(a) <= b0.x)) {
      ct = evs.time(a);
      I = (double)evs.weight(a);
      a++;
      return true;
    }
    if (b < nb) {
      ct = b0.x;
      I = b0.y;
      b++;
      if (b < nb) b0 = be[b];
      return true;
    }
    return false;
  };
  bool bad = false;
  double ct = 0, I = 0, dth = 0, rmh = 0, poly = 0;
  bool have = next(ct, I);
  if (have) lifca_coeff(par, ct - n.tr, dth, rmh, poly);
  while (have) {
    double ct1 = 0, I1 = 0, dth1 = 0, rmh1 = 0, poly1 = 0;
    const bool have1 = next(ct1, I1);
    if (have1) lifca_coeff(par, ct1 - ct, dth1, rmh1, poly1);   // after this event Tr = ct
    bad |= ((ct - T0) >= 1.0) || ((ct - T0) < 0);
    lifca_pre(par, n, ct, I, dth, rmh, poly);
    ct = ct1;
    I = I1;
    dth = dth1;
    rmh = rmh1;
    poly = poly1;
    have = have1;
  }
  if (bad) atomicOr(d.flags, F_TIME_WINDOW);
  d.v[i] = n.v;
  d.c[i] = n.c;
  d.tr[i] = n.tr;
  d.te[i] = n.te;
  return n.fired;
}

struct EvArrays {   // sorted times and weights in two arrays
  const double *tau;
  const float *val;
  __device__ double time(uint32_t a) const { return tau[a]; }
  __device__ float weight(uint32_t a) const { return val[a]; }
};
struct EvRecords {  // sorted 16-byte records
  const SortEv *se;
  __device__ double time(uint32_t a) const { return se[a].tau; }
  __device__ float weight(uint32_t a) const { return se[a].val; }
};

__device__ static inline int run_neuron(const Dev &d, uint32_t i, uint32_t t, const double *tau,
                                        const float *val, uint32_t ns) {
  const uint2 at = d.bath_at[i];
  return run_neuron_ev(d, i, t, EvArrays{tau, val}, ns, d.bath_ev + at.x, at.y);
}

// A neuron that fired, run apart from its block.
__device__ static inline void mark_fired(const Dev &d, uint32_t i) {
  d.fired[i] = 1;
  atomicAdd(&d.block_fired[i / NEURON_BLOCK], 1u);
}

// Step 4: neuron update (regularDynamicTimeStep, DPSNN_neuron_sim.c:522-662).
// Light neurons (at most LOCAL_EVENTS synaptic events this step): one thread
// each, insertion sort by (arrival time, key) in registers/local memory.
// Heavier neurons are queued for the heavy path below.
__device__ static inline uint32_t warp_path_max(const NetConst *net);

// A warp's neurons' bath events follow one another in memory (one rank's are
// written in neuron order): the warp loads them into shared memory at once,
// coalesced, and each thread reads its own from there.  A warp that spans two
// ranks, or whose neurons have more than NEURON_STAGE events, reads global
// memory.  What bounds it: the latency of a warp's chain, events one after
// another in 16 lanes of 32 on average (720 000 neurons without synaptic
// events: 80 us alone; 180 000: 32 us, DRAM at 6.5 %, an instruction every 5
// cycles per scheduler).  A step of 24x24 takes 228 us with the staged pairs and
// div_by against 239 with three dependent loads per event and two divisions.
#define NEURON_STAGE 192

// The warp's bath events staged in st where they fit; the thread's first one.
__device__ static inline const double2 *stage_bath(const Dev &d, uint2 at, double2 *st, uint32_t lane) {
  const double2 *be = d.bath_ev + at.x;
  const uint32_t lo = __reduce_min_sync(0xffffffffu, at.y ? at.x : 0xFFFFFFFFu);
  const uint32_t hi = __reduce_max_sync(0xffffffffu, at.y ? at.x + at.y : 0u);
  if (hi > lo && hi - lo <= NEURON_STAGE) {
    for (uint32_t k = lane; k < hi - lo; k += 32) st[k] = d.bath_ev[lo + k];
    be = st + (at.y ? at.x - lo : 0u);
  }
  __syncwarp();
  return be;
}

// A light neuron: at most LOCAL_EVENTS synaptic events, sorted by insertion.
__device__ static inline int run_light(const Dev &d, uint32_t i, uint32_t t, uint32_t cnt, const double2 *be,
                                       uint32_t nb) {
  const uint32_t N = d.net->N, D = d.net->D, cap = d.net->ev_cap;
        SortEv se[LOCAL_EVENTS];
        const uint2 *ev = d.ev + (size_t)i * cap;
        // events in groups of NEURON_BATCH: the loads, then the arrival-time
        // gathers, are all in flight together; then insertion by (time, key)
        for (uint32_t e0 = 0; e0 < cnt; e0 += NEURON_BATCH) {
          uint2 x[NEURON_BATCH];
          double tm[NEURON_BATCH];
  #pragma unroll
          for (int u = 0; u < NEURON_BATCH; u++)
            if (e0 + u < cnt) x[u] = ev[e0 + u];
  #pragma unroll
          for (int u = 0; u < NEURON_BATCH; u++)
            if (e0 + u < cnt) tm[u] = event_time(d, x[u].x, t, D, N);
  #pragma unroll
          for (int u = 0; u < NEURON_BATCH; u++) {
            if (e0 + u < cnt) {
              SortEv y;
              y.tau = tm[u];
              y.key = x[u].x;
              y.val = __uint_as_float(x[u].y);
              uint32_t p = e0 + u;
              while (p > 0 && sortev_gt(se[p - 1], y)) {
                se[p] = se[p - 1];
                p--;
              }
              se[p] = y;
            }
          }
        }
  return run_neuron_ev(d, i, t, EvRecords{se}, cnt, be, nb);
}

__global__ void __launch_bounds__(NEURON_BLOCK, 4) neuron_kernel(Dev d) {
  __shared__ double2 s_bath[NEURON_BLOCK / 32][NEURON_STAGE];
  const NetConst *net = d.net;
  const uint32_t t = *d.t, N = net->N;
  const uint32_t i = blockIdx.x * NEURON_BLOCK + threadIdx.x, lane = threadIdx.x & 31;
  const uint2 at = i < N ? d.bath_at[i] : make_uint2(0, 0);
  const double2 *be = stage_bath(d, at, s_bath[threadIdx.x >> 5], lane);
  int fired = 0;
  if (i < N) {
    const uint32_t cnt = d.ev_cnt[i];
    d.ev_cnt[i] = 0;
    if (cnt > net->light_max) {
      const uint32_t path = (cnt <= warp_path_max(net)) ? 0u : 1u;
      const uint32_t k = atomicAdd(&d.heavy_cnt[path], 1u);
      if (k < N) {
        d.heavy_list[2ull * N * path + k] = i;
        d.heavy_list[2ull * N * path + N + k] = cnt;
      }
    } else {
      fired = run_light(d, i, t, cnt, be, at.y);
      if (fired) d.fired[i] = 1;
    }
  }
  const uint32_t bc = __syncthreads_count(fired);
  if (threadIdx.x == 0) d.block_fired[blockIdx.x] = bc;
}

// Heavy neurons, more than LOCAL_EVENTS synaptic events in one step.
// heavy_sort_kernel: one warp per neuron with at most HEAVY_WARP_MAX events
// loads its bucket into registers, computes the arrival times, sorts by
// (time, key) and writes the sorted events back into the bucket;
// heavy_run_kernel then runs those neurons one thread each.  Neurons with
// more events (including any beyond the bucket, in the overflow list) are
// sorted by huge_kernel, one block each; those with at most half a bucket of
// events go back to the bucket and run in heavy_run_kernel, the others run
// in their block.
#define HEAVY_WARP_MAX 256     // events a warp sorts (8 per lane)
#define HEAVY_MAX 8192
#define HEAVY_THREADS 256
#define HUGE_SMEM_EVENTS 2048   // a huge neuron sorted in shared memory (32 KB); more in global scratch

__device__ static inline void bitonic_sort_shared(double *tau, uint32_t *key, float *val, uint32_t n2,
                                                  uint32_t tid, uint32_t nthr, bool warp_only) {
  for (uint32_t k = 2; k <= n2; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      // pair p compares a = p with bit j inserted as 0, and b = a | j
      for (uint32_t p = tid; p < (n2 >> 1); p += nthr) {
        const uint32_t a = ((p & ~(j - 1)) << 1) | (p & (j - 1)), b = a | j;
        const bool up = (a & k) == 0;
        const double ta = tau[a], tb = tau[b];
        const uint32_t ka = key[a], kb = key[b];
        const bool gt = (ta > tb) || (ta == tb && ka > kb);
        if (gt == up) {
          tau[a] = tb;
          tau[b] = ta;
          key[a] = kb;
          key[b] = ka;
          const float va = val[a];
          val[a] = val[b];
          val[b] = va;
        }
      }
      if (warp_only) __syncwarp(); else __syncthreads();
    }
  }
}

// Events per neuron handled by the warp path: at most the bucket size.
// (the sorted times and weights are written back into the first half and
// the second half of the bucket)
__device__ static inline uint32_t warp_path_max(const NetConst *net) {
  return min(net->ev_cap / 2, (uint32_t)HEAVY_WARP_MAX);
}

// A warp's sort of one heavy neuron's events: a bucket sort on the arrival
// time.  Arrival times lie in [t, t+1); bucket (time - t) * 256 is monotone
// in the time, so buckets order the events, and inside a bucket each event's
// place is the number of the bucket's events before it in (time, key) order
// (keys are unique per target).  Buckets are small unless many events share
// one arrival time, as a cascade's do; then the count is quadratic in the
// bucket's size, spread over the lanes.
#define HS_BUCKETS 256

#define HS_BATH_MAX 128         // bath events a warp merges into the sorted stream

struct HeavySortWarp {
  uint32_t start[HS_BUCKETS + 1];   // counts, then the buckets' first positions
  double tau[HEAVY_WARP_MAX + HS_BATH_MAX];   // events staged by bucket for the counts
  uint32_t key[HEAVY_WARP_MAX + HS_BATH_MAX];
};

// A heavy neuron's merged event stream in its bucket: {time, input} per
// event, synaptic and bath events in the order the reference merges them
// (mergeFunction, DPSNN_neuron_sim.c:391-421: a synaptic event first on
// equal times).  The list's count entry carries this flag when the sort
// left the stream merged.
#define HEAVY_MERGED 0x80000000u

// One heavy neuron's n <= 32*E events (element e = lane + 32r in register r):
// loaded with their arrival times and sorted by (time, key).  When the
// merged stream fits half the bucket, the neuron's bath events join the sort
// with keys above every synaptic key (so a synaptic event comes first on
// equal times, and bath events keep their order) and the bucket receives the
// merged stream {time, input}; otherwise it receives the sorted times in its
// first half and the weights in its second half.  Returns whether merged.
#define HS_BATH_KEY 0xFFFFFF80u   // + j for bath event j; synaptic keys are below 80 << 25
static_assert(RING_SLOTS <= 127, "synaptic keys (D-1-d) << 25 | q stay below the bath keys");

template <int E>
__device__ static inline bool heavy_sort_one(const Dev &d, uint32_t i, uint2 *ev, uint32_t n, uint32_t t, uint32_t D,
                                             uint32_t N, uint32_t cap, uint32_t lane, HeavySortWarp &w) {
  const double T0 = (double)t;
  const uint2 at = d.bath_at[i];
  const double2 *be = d.bath_ev + at.x;
  const uint32_t bcnt = at.y;
  const bool merged = n + bcnt <= cap / 2 && bcnt <= HS_BATH_MAX;
  const uint32_t bc = merged ? bcnt : 0u;
  for (uint32_t b = lane; b <= HS_BUCKETS; b += 32) w.start[b] = 0;
  uint2 x[E];
#pragma unroll
  for (int r = 0; r < E; r++) {
    const uint32_t e = lane + 32u * r;
    if (e < n) x[r] = ev[e];
  }
  __syncwarp();
  double tau[E];
  uint32_t bs[E], bb[HS_BATH_MAX / 32];   // bucket << 16 | place among the bucket's elements in arrival order
#pragma unroll
  for (int r = 0; r < E; r++) {
    const uint32_t e = lane + 32u * r;
    if (e < n) {
      tau[r] = event_time(d, x[r].x, t, D, N);
      const uint32_t b = min((uint32_t)((tau[r] - T0) * (double)HS_BUCKETS), (uint32_t)HS_BUCKETS - 1);
      bs[r] = (b << 16) | atomicAdd(&w.start[b], 1u);
    }
  }
#pragma unroll
  for (int r = 0; r < HS_BATH_MAX / 32; r++) {
    const uint32_t j = lane + 32u * r;
    if (j < bc) {
      const double btj = be[j].x;
      const uint32_t b = min((uint32_t)((btj - T0) * (double)HS_BUCKETS), (uint32_t)HS_BUCKETS - 1);
      bb[r] = (b << 16) | atomicAdd(&w.start[b], 1u);
    }
  }
  __syncwarp();
  // exclusive prefix of the counts, 8 consecutive buckets per lane
  {
    uint32_t c[HS_BUCKETS / 32], tot = 0;
#pragma unroll
    for (int q = 0; q < HS_BUCKETS / 32; q++) {
      c[q] = w.start[lane * (HS_BUCKETS / 32) + q];
      const uint32_t v = c[q];
      c[q] = tot;
      tot += v;
    }
    uint32_t incl = tot;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (uint32_t)o) incl += y;
    }
#pragma unroll
    for (int q = 0; q < HS_BUCKETS / 32; q++) w.start[lane * (HS_BUCKETS / 32) + q] = incl - tot + c[q];
    if (lane == 31) w.start[HS_BUCKETS] = incl;
  }
  __syncwarp();
  // staged by bucket; bs/bb become bucket << 16 | staged position
#pragma unroll
  for (int r = 0; r < E; r++) {
    const uint32_t e = lane + 32u * r;
    if (e < n) {
      const uint32_t b = bs[r] >> 16, p = w.start[b] + (bs[r] & 0xFFFFu);
      w.tau[p] = tau[r];
      w.key[p] = x[r].x;
      bs[r] = (b << 16) | p;
    }
  }
#pragma unroll
  for (int r = 0; r < HS_BATH_MAX / 32; r++) {
    const uint32_t j = lane + 32u * r;
    if (j < bc) {
      const uint32_t b = bb[r] >> 16, p = w.start[b] + (bb[r] & 0xFFFFu);
      w.tau[p] = be[j].x;
      w.key[p] = HS_BATH_KEY + j;
      bb[r] = (b << 16) | p;
    }
  }
  __syncwarp();
  // each element's place: its bucket's start plus the bucket's elements
  // before it in (time, key) order
  auto place = [&](uint32_t v) -> uint32_t {
    const uint32_t b = v >> 16, p = v & 0xFFFFu;
    const uint32_t b0 = w.start[b], b1 = w.start[b + 1], k = w.key[p];
    const double tm = w.tau[p];
    uint32_t rank = 0;
    for (uint32_t j = b0; j < b1; j++) {
      const double tj = w.tau[j];
      rank += (tj < tm) || (tj == tm && w.key[j] < k);
    }
    return b0 + rank;
  };
  double2 *ms = reinterpret_cast<double2 *>(ev);
  double *st = reinterpret_cast<double *>(ev);
  float *sv = reinterpret_cast<float *>(ev + cap / 2);
#pragma unroll
  for (int r = 0; r < E; r++) {
    const uint32_t e = lane + 32u * r;
    if (e < n) {
      const uint32_t pos = place(bs[r]);
      const double tm = w.tau[bs[r] & 0xFFFFu];
      if (merged) {
        ms[pos] = make_double2(tm, (double)__uint_as_float(x[r].y));
      } else {
        st[pos] = tm;
        sv[pos] = __uint_as_float(x[r].y);
      }
    }
  }
  if (merged) {
#pragma unroll
    for (int r = 0; r < HS_BATH_MAX / 32; r++) {
      const uint32_t j = lane + 32u * r;
      if (j < bc) ms[place(bb[r])] = be[j];
    }
  }
  __syncwarp();   // the warp's next neuron reuses the staging arrays
  return merged;
}

#define HEAVY_SORT_THREADS 256

// A warp per neuron of the warp path (LOCAL_EVENTS < n <= HEAVY_WARP_MAX),
// each warp with its own bucket-sort arrays in shared memory.  Two kernels
// over the same list: up to 64 events (one or two per lane, the common case
// outside bursts) at four blocks per SM, more events (four or eight per lane,
// more registers) at two.
#define HEAVY_SORT_SMALL 64

template <bool SMALL>
__device__ static inline void heavy_sort_list(const Dev &d) {
  __shared__ HeavySortWarp s_ws[HEAVY_SORT_THREADS / 32];
  const NetConst *net = d.net;
  const uint32_t t = *d.t, N = net->N, D = net->D, cap = net->ev_cap, wmax = warp_path_max(net);
  const uint32_t lane = threadIdx.x & 31;
  HeavySortWarp &ws = s_ws[threadIdx.x >> 5];
  const uint32_t nh = min(d.heavy_cnt[0], N);
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  // a neuron not listed here was sorted already by the other kernel, which
  // flags the count
  auto mine = [&](uint32_t n) { return n <= wmax && (SMALL ? n <= HEAVY_SORT_SMALL : n > HEAVY_SORT_SMALL); };
  // the warp's list entries are read two neurons ahead, and the next
  // neuron's events are prefetched into L2 while this one is sorted
  uint32_t hh = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  uint32_t i = 0, n = 0, i1 = 0, n1 = 0;
  if (hh < nh) {
    i = d.heavy_list[hh];
    n = d.heavy_list[N + hh];
  }
  if (hh + nwarps < nh) {
    i1 = d.heavy_list[hh + nwarps];
    n1 = d.heavy_list[N + hh + nwarps];
  }
  for (; hh < nh; hh += nwarps) {
    const uint32_t h2 = hh + 2u * nwarps;
    uint32_t i2 = 0, n2 = 0;
    if (h2 < nh) {
      i2 = d.heavy_list[h2];
      n2 = d.heavy_list[N + h2];
    }
    // 16 events (128 bytes) per lane's line, inside neuron i1's bucket
    if (hh + nwarps < nh && mine(n1) && lane * 16u < n1)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(d.ev + (size_t)i1 * cap + lane * 16u));
    if (mine(n)) {
      uint2 *ev = d.ev + (size_t)i * cap;
      bool merged;
      if (SMALL) {
        if (n <= 32)
          merged = heavy_sort_one<1>(d, i, ev, n, t, D, N, cap, lane, ws);
        else
          merged = heavy_sort_one<2>(d, i, ev, n, t, D, N, cap, lane, ws);
      } else {
        if (n <= 128)
          merged = heavy_sort_one<4>(d, i, ev, n, t, D, N, cap, lane, ws);
        else
          merged = heavy_sort_one<8>(d, i, ev, n, t, D, N, cap, lane, ws);
      }
      if (merged && lane == 0) d.heavy_list[N + hh] = n | HEAVY_MERGED;
    }
    i = i1;
    n = n1;
    i1 = i2;
    n1 = n2;
  }
}

// For a kernel that runs beside the one before it on the stream (launch_main's
// `early`, and no wait at its start): its last block ends after that kernel's,
// so what comes next follows both.  One block is enough, and the others leave
// their room at once.
__device__ static inline void end_after_previous() {
  if (blockIdx.x == gridDim.x - 1) cudaGridDependencySynchronize();
}

// The two sorts and huge_kernel take different neurons of lists that are
// complete before the first of them starts (an entry's merged flag, which the
// other sort may or may not see, is no count that it sorts): each starts when
// the blocks of the one before it have all started, and fills the room that
// its last blocks leave; heavy_rest_kernel runs beside heavy_run_kernel in the
// same way.  The sort of the few longest neurons goes first.  One after
// another, a 24x24 step took 504 us against 492 (active, 4.1 M events), 339
// against 328 (around the onset), 220 against 213 (no synaptic event: three
// launches' gaps beside the bath).
__global__ void __launch_bounds__(HEAVY_SORT_THREADS, 2) heavy_sort_big_kernel(Dev d) {
  cudaTriggerProgrammaticLaunchCompletion();
  heavy_sort_list<false>(d);
}
__global__ void __launch_bounds__(HEAVY_SORT_THREADS, 4) heavy_sort_kernel(Dev d) {
  cudaTriggerProgrammaticLaunchCompletion();
  heavy_sort_list<true>(d);
  end_after_previous();
}

// Runs a neuron whose events were left sorted in its bucket (arrival times,
// then weights): the warp path's neurons, and the block path's neurons with
// at most half a bucket of events, which huge_kernel sorts and leaves there.
// Same merge and arithmetic as run_neuron.
__device__ static inline bool huge_runs_here(const NetConst *net, uint32_t cnt) {
  return cnt <= net->ev_cap / 2 && cnt <= MAX_INPUTS_PER_STEP;
}

// A neuron's merged stream of ne events ({time, input}, in the order they
// apply): LIFCADynamic over it, four events' loads in flight ahead of the
// four being applied, each update's coefficients computed off the v/c chain.
__device__ static inline int run_neuron_merged(const Dev &d, uint32_t i, uint32_t t, const double2 *ms,
                                               uint32_t ne) {
  const LifcaRegs par(d.net, d.sub[i]);
  NeuronRegs n;
  n.v = d.v[i];
  n.c = d.c[i];
  n.tr = d.tr[i];
  n.te = d.te[i];
  n.fired = 0;
  const double T0 = (double)t;
  double2 cur[4], nxt[4];
#pragma unroll
  for (int u = 0; u < 4; u++) cur[u] = (u < (int)ne) ? ms[u] : make_double2(0.0, 0.0);
  bool bad = false;
  for (uint32_t e0 = 0; e0 < ne; e0 += 4) {
#pragma unroll
    for (int u = 0; u < 4; u++) nxt[u] = (e0 + 4 + u < ne) ? ms[e0 + 4 + u] : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (e0 + u < ne) {
        const double ct = cur[u].x;
        double dth, rmh, poly;
        lifca_coeff(par, ct - n.tr, dth, rmh, poly);
        bad |= ((ct - T0) >= 1.0) || ((ct - T0) < 0);
        lifca_pre(par, n, ct, cur[u].y, dth, rmh, poly);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) cur[u] = nxt[u];
  }
  if (bad) atomicOr(d.flags, F_TIME_WINDOW);
  d.v[i] = n.v;
  d.c[i] = n.c;
  d.tr[i] = n.tr;
  d.te[i] = n.te;
  return n.fired;
}

// The warp path's neurons whose sort left a merged stream, a thread each.
__global__ void __launch_bounds__(128, 6) heavy_run_kernel(Dev d) {
  cudaTriggerProgrammaticLaunchCompletion();
  const NetConst *net = d.net;
  const uint32_t t = *d.t, N = net->N, cap = net->ev_cap;
  const uint32_t nh = min(d.heavy_cnt[0], N);
  for (uint32_t hh = blockIdx.x * blockDim.x + threadIdx.x; hh < nh; hh += gridDim.x * blockDim.x) {
    const uint32_t i = d.heavy_list[hh], ns = d.heavy_list[N + hh];
    if (!(ns & HEAVY_MERGED)) continue;
    const uint32_t ne = (ns & ~HEAVY_MERGED) + d.bath_at[i].y;
    if (run_neuron_merged(d, i, t, reinterpret_cast<const double2 *>(d.ev + (size_t)i * cap), ne)) mark_fired(d, i);
  }
}

// The other neurons left sorted in their bucket (times and weights in its
// halves, merged with the bath events here): the warp path's neurons whose
// merged stream would not fit half the bucket, and the block path's with at
// most half a bucket of events.  A thread each.
__global__ void heavy_rest_kernel(Dev d) {
  const NetConst *net = d.net;
  const uint32_t t = *d.t, N = net->N, cap = net->ev_cap, wmax = warp_path_max(net);
  const uint32_t nh0 = min(d.heavy_cnt[0], N), nh = nh0 + min(d.heavy_cnt[1], N);
  for (uint32_t hh = blockIdx.x * blockDim.x + threadIdx.x; hh < nh; hh += gridDim.x * blockDim.x) {
    uint32_t i, ns;
    if (hh < nh0) {
      i = d.heavy_list[hh];
      ns = d.heavy_list[N + hh];
      if ((ns & HEAVY_MERGED) || ns > wmax) continue;
    } else {
      i = d.heavy_list[2ull * N + (hh - nh0)];
      ns = d.heavy_list[3ull * N + (hh - nh0)];
      if (ns <= wmax || !huge_runs_here(net, ns)) continue;
    }
    const uint2 *ev = d.ev + (size_t)i * cap;
    const double *st = reinterpret_cast<const double *>(ev);
    const float *sv = reinterpret_cast<const float *>(ev + cap / 2);
    if (run_neuron(d, i, t, st, sv, ns)) mark_fired(d, i);
  }
  end_after_previous();
}

// Gather a neuron's events (bucket, then overflow list) into shared arrays.
__device__ static inline uint32_t gather_events(const Dev &d, uint32_t i, uint32_t cnt, uint32_t *key, float *val,
                                                uint32_t capacity, uint32_t tid, uint32_t nthr, uint32_t *counter) {
  const NetConst *net = d.net;
  const uint32_t cap = net->ev_cap, nb = min(cnt, cap);
  for (uint32_t e = tid; e < nb; e += nthr) {
    const uint2 x = d.ev[(size_t)i * cap + e];
    key[e] = x.x;
    val[e] = __uint_as_float(x.y);
  }
  if (tid == 0) *counter = nb;
  __syncthreads();
  if (cnt > cap) {
    const uint32_t novf = min(*d.ovf_cnt, net->ovf_cap);
    for (uint32_t o = tid; o < novf; o += nthr) {
      const uint4 x = d.ovf[o];
      if (x.x == i) {
        uint32_t k = atomicAdd(counter, 1u);
        if (k < capacity) {
          key[k] = x.y;
          val[k] = __uint_as_float(x.z);
        }
      }
    }
    __syncthreads();
  }
  return min(*counter, capacity);
}

// The block path's list, neurons strided over the blocks; fired(i) for a
// neuron run here.
template <typename Fired>
__device__ static inline void huge_sort(const Dev &d, const Fired &fired) {
  // 32 KB of shared memory, so that a block fits on an SM beside the bath's
  // blocks; the rare neuron with more events sorts in its block's global
  // scratch (HEAVY_MAX events)
  __shared__ double sh_tau[HUGE_SMEM_EVENTS];
  __shared__ uint32_t sh_key[HUGE_SMEM_EVENTS];
  __shared__ float sh_val[HUGE_SMEM_EVENTS];
  __shared__ uint32_t s_n;
  const NetConst *net = d.net;
  const uint32_t t = *d.t, N = net->N, D = net->D, tid = threadIdx.x;
  const uint32_t nh = min(d.heavy_cnt[1], N);
  const uint32_t *hl = d.heavy_list + 2ull * N;
  for (uint32_t hh = blockIdx.x; hh < nh; hh += gridDim.x) {
    const uint32_t i = hl[hh], cnt = hl[N + hh];
    if (cnt <= warp_path_max(net)) continue;   // not listed here
    if (cnt > MAX_INPUTS_PER_STEP) {
      if (tid == 0) atomicOr(d.flags, F_TOO_MANY_INPUTS);
      continue;
    }
    const bool in_smem = cnt <= HUGE_SMEM_EVENTS;
    double *s_tau = in_smem ? sh_tau : d.huge_tau + (size_t)blockIdx.x * HEAVY_MAX;
    uint32_t *s_key = in_smem ? sh_key : d.huge_key + (size_t)blockIdx.x * HEAVY_MAX;
    float *s_val = in_smem ? sh_val : d.huge_val + (size_t)blockIdx.x * HEAVY_MAX;
    const uint32_t n = gather_events(d, i, cnt, s_key, s_val, in_smem ? HUGE_SMEM_EVENTS : HEAVY_MAX, tid,
                                     blockDim.x, &s_n);
    uint32_t n2 = 1;
    while (n2 < n) n2 <<= 1;
    for (uint32_t e = tid; e < n2; e += blockDim.x) {
      if (e < n) {
        s_tau[e] = event_time(d, s_key[e], t, D, N);
      } else {
        s_tau[e] = INFINITY;
        s_key[e] = 0xFFFFFFFFu;
      }
    }
    __syncthreads();
    bitonic_sort_shared(s_tau, s_key, s_val, n2, tid, blockDim.x, false);
    if (huge_runs_here(net, cnt)) {
      // sorted back into the bucket's halves; heavy_run_kernel runs the
      // neuron, beside the others, one thread each
      uint2 *ev = d.ev + (size_t)i * net->ev_cap;
      double *st = reinterpret_cast<double *>(ev);
      float *sv = reinterpret_cast<float *>(ev + net->ev_cap / 2);
      for (uint32_t e = tid; e < n; e += blockDim.x) {
        st[e] = s_tau[e];
        sv[e] = s_val[e];
      }
    } else if (tid == 0) {
      if (run_neuron(d, i, t, s_tau, s_val, n)) fired(i);
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(HEAVY_THREADS) huge_kernel(Dev d) {
  huge_sort(d, [&](uint32_t i) { mark_fired(d, i); });
  end_after_previous();
}

// ------------------------------------------------------------------ small networks
// Up to SMALL_N neurons a step is bound by its launches, about 5 us each with
// the gap between two, and most of the large form's blocks find nothing to do.
// Here a step is three kernels (and the bath): deliver_small_kernel with the
// compaction, neuron_small_kernel with the warp path's sorts and runs, and
// tail_small_kernel, each brought up while the one before it ends.  Measured
// per step: 19 us from 45 for 100 neurons, 23 from 54 for 1155 in 5 ranks, 60
// from 113 for 16 000 busy ones (8 events per neuron); what is left is the
// update's chain of events, and the bath where a rank is long.

// A block of WARPS warps per 32 neurons: warp 0 runs the light ones while the
// others (and then it too) sort the heavier ones, which then run a lane each.
// Light: up to SMALL_LIGHT events.  A thread's insertion sort and merge of 16
// take its warp 40 000 cycles, a warp's sort of as many 4000 and their run by
// lanes half of the former (16 000 busy neurons: 60 us per step against 67 with
// the line at 16; 3 and 9 are within 2 us of 6).
#define SMALL_LIGHT 6
template <int WARPS>
__global__ void __launch_bounds__(32 * WARPS, 16 / WARPS) neuron_small_kernel(Dev d) {
  __shared__ HeavySortWarp s_ws[WARPS];
  __shared__ double2 s_bath[NEURON_STAGE];
  __shared__ uint32_t s_i[32], s_n[32], s_nh, s_next;
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  const NetConst *net = d.net;
  const uint32_t t = *d.t, N = net->N, D = net->D, cap = net->ev_cap;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t i = blockIdx.x * 32 + lane;
  uint32_t cnt = 0;
  bool light = false;
  if (warp == 0) {
    if (i < N) {
      cnt = d.ev_cnt[i];
      if (cnt) d.ev_cnt[i] = 0;
    }
    light = i < N && cnt <= min(net->light_max, (uint32_t)SMALL_LIGHT);
    const bool heavy = !light && cnt && cnt <= warp_path_max(net);
    const uint32_t bal = __ballot_sync(0xffffffffu, heavy);
    if (heavy) {
      const uint32_t k = __popc(bal & ((1u << lane) - 1));
      s_i[k] = i;
      s_n[k] = cnt;
    } else if (i < N && !light) {
      const uint32_t k = atomicAdd(&d.heavy_cnt[1], 1u);
      d.heavy_list[2ull * N + k] = i;
      d.heavy_list[3ull * N + k] = cnt;
    }
    if (lane == 0) {
      s_nh = __popc(bal);
      s_next = 0;
    }
  }
  __syncthreads();
  const uint32_t nh = s_nh;
  uint32_t bits = 0;
  if (warp == 0) {
    const uint2 at = i < N ? d.bath_at[i] : make_uint2(0, 0);
    const double2 *be = stage_bath(d, at, s_bath, lane);
    int fired = 0;
    if (light) fired = run_light(d, i, t, cnt, be, at.y);
    bits = __ballot_sync(0xffffffffu, fired);
  }
  if (nh) {
    for (;;) {
      uint32_t k = 0;
      if (lane == 0) k = atomicAdd(&s_next, 1u);
      k = __shfl_sync(0xffffffffu, k, 0);
      if (k >= nh) break;
      const uint32_t j = s_i[k], n = s_n[k];
      uint2 *ev = d.ev + (size_t)j * cap;
      const bool merged = n <= 32    ? heavy_sort_one<1>(d, j, ev, n, t, D, N, cap, lane, s_ws[warp])
                          : n <= 64  ? heavy_sort_one<2>(d, j, ev, n, t, D, N, cap, lane, s_ws[warp])
                          : n <= 128 ? heavy_sort_one<4>(d, j, ev, n, t, D, N, cap, lane, s_ws[warp])
                                     : heavy_sort_one<8>(d, j, ev, n, t, D, N, cap, lane, s_ws[warp]);
      if (merged && lane == 0) s_n[k] = n | HEAVY_MERGED;
    }
    __syncthreads();
  }
  if (warp == 0) {
    uint32_t mine = 0;
    if (lane < nh) {
      const uint32_t j = s_i[lane], n = s_n[lane] & ~HEAVY_MERGED;
      const uint2 *ev = d.ev + (size_t)j * cap;
      const int fired =
          (s_n[lane] & HEAVY_MERGED)
              ? run_neuron_merged(d, j, t, reinterpret_cast<const double2 *>(ev), n + d.bath_at[j].y)
              : run_neuron(d, j, t, reinterpret_cast<const double *>(ev), reinterpret_cast<const float *>(ev + cap / 2), n);
      if (fired) mine = 1u << (j & 31);
    }
    bits |= __reduce_or_sync(0xffffffffu, mine);
    if (lane == 0) d.fired_bits[blockIdx.x] = bits;
  }
}

// Neurons beyond the warp path, sorted by blocks and then run a thread each,
// and the end of the step (the last block to finish).
__global__ void __launch_bounds__(HEAVY_THREADS) tail_small_kernel(Dev d) {
  __shared__ uint32_t s_last;
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  const NetConst *net = d.net;
  const uint32_t N = net->N, nh = min(d.heavy_cnt[1], N);
  if (nh) {
    const uint32_t t = *d.t, cap = net->ev_cap;
    auto fired = [&](uint32_t i) { atomicOr(&d.fired_bits[i >> 5], 1u << (i & 31)); };
    huge_sort(d, fired);
    __syncthreads();
    for (uint32_t hh = blockIdx.x + gridDim.x * threadIdx.x; hh < nh; hh += gridDim.x * blockDim.x) {
      const uint32_t i = d.heavy_list[2ull * N + hh], ns = d.heavy_list[3ull * N + hh];
      if (!huge_runs_here(net, ns)) continue;
      const uint2 *ev = d.ev + (size_t)i * cap;
      if (run_neuron(d, i, t, reinterpret_cast<const double *>(ev), reinterpret_cast<const float *>(ev + cap / 2), ns))
        fired(i);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(d.ticket, 1u) == gridDim.x - 1;
    if (s_last) {
      *d.ticket = 0;
      *d.ovf_cnt = 0;
      d.heavy_cnt[0] = 0;
      d.heavy_cnt[1] = 0;
      *d.t = *d.t + 1;
    }
  }
}

// Long term plasticity at x999 ms (longTermPlasticity, DPSNN_localNet_sim.c:312-414),
// one warp per presynaptic neuron.
__global__ void ltp_kernel(Dev d) {
  const NetConst *net = d.net;
  const uint32_t t = *d.t;
  if (!((t % 1000) == 999 && t >= net->start_pl && t <= net->stop_pl)) return;
  const uint32_t N = net->N, lane = threadIdx.x & 31;
  for (uint32_t P = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; P < N;
       P += (gridDim.x * blockDim.x) >> 5) {
    uint32_t sp = d.sub[P];
    for (uint64_t k = d.row_ptr[P] + lane; k < d.row_ptr[P + 1]; k += 32) {
      uint32_t tp = d.sub[d.post[k]];
      float maxv = (float)(2.0 * net->J[sp * DPSNN_MAX_SUBPOP + tp]);
      float rmaxv = (float)(2.0 * net->J[tp * DPSNN_MAX_SUBPOP + sp]);
      float clamp = 0.0f;
      float td = d.tderiv[k];
      const int16_t w0 = d.w16[k];
      if (d.probe_w) {
        d.probe_w[k] = w0;
        d.probe_td[k] = td;
      }
      if (maxv > 0.0 && rmaxv > 0.0) {
        float wF = (float)(w0 * net->w2f);
        float dF = td;
        dF += net->stdp_drift;
        wF = wF + dF;
        if (wF > maxv) { clamp = (wF - maxv); dF = dF - clamp; wF = maxv; }
        if (wF < 0.0) { clamp = wF; dF = dF - clamp; wF = 0.0f; }
        d.w16[k] = (int16_t)(wF * net->f2w);
        td = dF;
      }
      if (d.probe_w) d.probe_td_mid[k] = td;
      if (net->stdp_tauDecay == 1.0f)
        td = 0.0f;
      else
        td = (td - net->stdp_drift + clamp) * (1 - 1 / net->stdp_tauDecay);
      d.tderiv[k] = td;
    }
  }
}

__global__ void end_step_kernel(Dev d) {
  *d.ovf_cnt = 0;
  d.heavy_cnt[0] = 0;
  d.heavy_cnt[1] = 0;
  *d.t = *d.t + 1;
}

// Per-(neuron, delay) counts of the chosen hypothesis -> per-row totals and
// the in-row per-delay offsets.
__global__ void counts_to_csr_kernel(const NetConst *net, const uint16_t *cnt_out,
                                     const int32_t *hyp, uint16_t *sub_off, uint32_t *row_len) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= net->N) return;
  uint32_t D = net->D;
  int h = hyp[i / net->npcm];
  const uint16_t *c = cnt_out + ((size_t)h * net->N + i) * D;
  uint32_t acc = 0;
  for (uint32_t dl = 0; dl < D; dl++) {
    sub_off[(size_t)i * (D + 1) + dl] = (uint16_t)acc;
    acc += c[dl];
  }
  sub_off[(size_t)i * (D + 1) + D] = (uint16_t)acc;
  row_len[i] = acc;
}

__global__ void init_neurons_kernel(Dev d) {
  const NetConst *net = d.net;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= net->N) return;
  // initNeuralKind (DPSNN_neuron_init.c:99-115); Tr is zero (static storage)
  d.v[i] = net->H[d.sub[i]];
  d.c[i] = 0.0;
  d.te[i] = -1000;
  d.nb[i] = 0.0;
  d.tr[i] = 0.0;
  d.fired[i] = 0;
  d.last_spike_ms[i] = -100000;  // DPSNN_localNet_init.c:217
  d.ev_cnt[i] = 0;
}

// incoming-synapse lists (causal STDP), per post neuron
__global__ void in_count_kernel(const NetConst *net, const uint32_t *post, uint64_t S, uint64_t *in_ptr) {
  for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < S; k += (uint64_t)gridDim.x * blockDim.x)
    atomicAdd((unsigned long long *)&in_ptr[post[k] + 1], 1ull);
}
__global__ void in_fill_kernel(const NetConst *net, const uint32_t *post, uint64_t S, const uint64_t *in_ptr,
                               unsigned long long *fill, uint32_t *in_idx) {
  for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < S; k += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t j = post[k];
    unsigned long long p = atomicAdd(&fill[j], 1ull);
    in_idx[in_ptr[j] + p] = (uint32_t)k;
  }
}

// per (rank, delay): max and min presynaptic index among synapses aimed at
// that rank -- used to detect the reference's run-over-group-end search case.
// Most of a network's synapses cannot move an extremum that the first sources
// looked at have set: the minima are taken over ascending sources, the maxima
// over descending ones, and a synapse does an atomic only where it would
// change what it reads (a stale value only costs an atomic).  An atomic or two
// per synapse took 55 ms at the 24x24 network's 0.81 G.
__global__ void group_extrema_kernel(const NetConst *net, const uint64_t *row_ptr, const uint16_t *sub_off,
                                     const uint32_t *post, uint32_t *gmax, uint32_t *gmin) {
  const uint32_t N = net->N, D = net->D, lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5, w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  for (int up = 0; up < 2; up++)
    for (uint32_t w = w0; w < N; w += nw) {
      const uint32_t P = up ? w : N - 1 - w;
      const uint64_t row = row_ptr[P];
      const uint16_t *so = sub_off + (size_t)P * (D + 1);
      const uint32_t len = so[D];
      uint32_t dl = 0;
      for (uint32_t k = lane; k < len; k += 32) {
        while (so[dl + 1] <= k) dl++;
        const uint32_t g = post[row + k] / net->locN * D + dl;
        if (up) {
          if (gmin[g] > P) atomicMin(&gmin[g], P);
        } else {
          if (gmax[g] < P) atomicMax(&gmax[g], P);
        }
      }
    }
}

// Spike lists of a run of steps for the host, written straight into its
// pinned memory: the error flags, the counts, and the lists one after another
// when they fit.  One kernel and one wait; a copy per step and array cost
// about 9 us each (80 steps of a small network: 240 copies, 2 ms).
struct SpikeRead {
  uint32_t flags, total;
  uint32_t counts[RING_SLOTS];
};
static __host__ __device__ inline double *spike_read_te(SpikeRead *r) { return reinterpret_cast<double *>(r + 1); }
static_assert(sizeof(SpikeRead) % 8 == 0, "the emission times follow, then the ids");
#define READ_PACK_THREADS 256
__global__ void __launch_bounds__(READ_PACK_THREADS) read_pack_kernel(Dev d, uint32_t t0, uint32_t n, uint32_t cap,
                                                                      SpikeRead *out) {
  __shared__ uint32_t s_pre[RING_SLOTS + 1];
  const uint32_t N = d.net->N;
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) s_pre[k + 1] = d.ring_cnt[(t0 + k) % RING_SLOTS];
  __syncthreads();
  if (blockIdx.x == 0)
    for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) out->counts[k] = s_pre[k + 1];
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t acc = 0;   // at most RING_SLOTS * 2^25 < 2^32
    s_pre[0] = 0;
    for (uint32_t k = 1; k <= n; k++) s_pre[k] = acc += s_pre[k];
    if (blockIdx.x == 0) {
      out->flags = *d.flags;
      out->total = acc;
    }
  }
  __syncthreads();
  const uint32_t total = s_pre[n];
  if (total > cap) return;
  double *te = spike_read_te(out);
  uint32_t *ids = reinterpret_cast<uint32_t *>(te + cap);
  for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = n - 1;   // the last step that starts at or before g
    while (lo < hi) {
      const uint32_t mid = (lo + hi + 1) >> 1;
      if (s_pre[mid] <= g) lo = mid; else hi = mid - 1;
    }
    const size_t at = (size_t)((t0 + lo) % RING_SLOTS) * N + (g - s_pre[lo]);
    te[g] = d.ring_te[at];
    ids[g] = d.ring_ids[at];
  }
}

// ------------------------------------------------------------------ host engine
struct dpsnn_engine {
  NetConst hnet;
  Dev d;
  cudaStream_t stream = nullptr;
  // The bath of step t+1 runs on bath_stream while step t runs on stream:
  // its outputs and nextBath are double-buffered by step parity.
  cudaStream_t bath_stream = nullptr;
  cudaEvent_t ev_bath[2] = {nullptr, nullptr}, ev_neuron[2] = {nullptr, nullptr}, ev_start = nullptr;
  bool bath_primed = false;
  double *nb2[2] = {nullptr, nullptr};
  double2 *bath_ev2[2] = {nullptr, nullptr};
  uint2 *bath_at2[2] = {nullptr, nullptr};
  int device = 0;
  uint64_t S = 0;
  bool low_caps = false;   // some neuron's maxExternCurrentCount is below 16 (bath_kernel)
  uint32_t t_host = 0;   // steps enqueued
  uint32_t probe_t = UINT32_MAX;   // step of the last LTP probe taken
  uint32_t stdp_log_t = UINT32_MAX;   // step the STDP event log holds
  std::vector<uint64_t> h_row;     // host copies of the CSR row and delay offsets
  std::vector<uint16_t> h_so;      // (for the STDP event log's order)
  std::vector<void *> allocs;
  std::vector<void *> temps;       // build scratch, released when the build ends
  std::vector<void *> spare;       // scratch that the build is done with, released then too, or when memory runs out
  uint64_t bytes = 0;              // device memory held (allocs)
  uint32_t grid_neuron = 0, grid_deliver = 0, grid_heavy = 0, grid_heavy_run = 0, grid_huge = 0, grid_tail = 0;
  int sms = 148;                   // the device's SMs (default grids)
  int timing = 0;
  bool capturing = false;          // steps are being recorded into a graph
  struct TimedLaunch { int family; cudaEvent_t a, b; cudaStream_t st; };
  std::vector<TimedLaunch> pending;   // recorded, not yet read
  std::vector<cudaEvent_t> event_pool;
  double ktime[DPSNN_TIMING_SLOTS] = {};
  uint64_t klaunch[DPSNN_TIMING_SLOTS] = {};
  uint64_t launches = 0;               // kernels enqueued by dpsnn_step
  uint32_t *h_pin = nullptr;          // pinned {flags, spike count} of dpsnn_rank_spikes_noalloc
  SpikeRead *h_read = nullptr;        // pinned, mapped: what read_pack_kernel writes, h_read_cap spikes
  uint32_t h_read_cap = 0;
  std::mutex read_mu;                 // held from that kernel's launch until its lists are copied out
  // spike lists are read on their own stream as soon as the compaction of
  // their step is done, while the rest of that step (and later ones) run
  cudaStream_t read_stream = nullptr;
  cudaEvent_t ev_slot[RING_SLOTS] = {};
};

static void collect_timings(dpsnn_engine *e);

// The rule between a step's two forms, in us per step at rest / busy (8 events
// per neuron and ms), small form against large.  Up to 16 384 neurons the small
// one is as fast or faster: 16 000 in 1 rank 426 / 432 against 430 / 433, in 8
// ranks 67 / 74 against 68 / 97, in 64 ranks 32 / 61 against 47 / 104; 100 in one
// 19 against 45.  Beyond, it is with short ranks (32 400 in 120: 37 / 101 against
// 54 / 115, in 40: 46 / 102 against 50 / 122); with long ones both wait for the
// baths, which the small one's update slows (in 4 ranks 229 / 239 against 227 /
// 232, in 10 ranks 106 / 120 against 101 / 114).  Near the line one is ahead at
// rest and the other busy (15 ranks of 2160: 80 / 98 against 73 / 110; 20 of 1620:
// 66 / 101 against 59 / 111).
static bool small_form(uint64_t neurons, uint64_t rank_neurons) {
  return neurons <= SMALL_N && (neurons <= SMALL_N / 2 || rank_neurons <= 2048);
}

// The grids that dpsnn_set_launch_shape sets (0: the default).  The
// delivery's default is a warp per four neurons, up to eight blocks per SM:
// a spike's 20 or so segments are items of its warps, and a small network's
// further blocks would only look for items.
static void default_grids(dpsnn_engine *e, uint32_t deliver, uint32_t heavy_sort, uint32_t heavy_run) {
  const uint32_t sms = (uint32_t)e->sms;
  e->grid_deliver = deliver ? deliver : std::max(4u, std::min(sms * 8, (e->hnet.N + 31) / 32));
  e->grid_heavy = heavy_sort ? heavy_sort : sms * 8;
  e->grid_heavy_run = heavy_run ? heavy_run : sms * 16;
}

// Device allocations are stream-ordered on the engine stream (the
// device's memory pool): unlike cudaMalloc/cudaFree they do not synchronise
// the device, so engines built from several host threads, or while other
// engines step, do not wait for each other.  `temp` allocations (the
// connectome build's scratch) are released at the end of the build: earlier,
// the pool would unmap and map the same memory again (24x24: 30 of 200 ms).
// Where memory runs out before, the finished generation's, hundreds of bytes
// per neuron, goes first.
static void free_list(dpsnn_engine *e, std::vector<void *> &v) {
  for (void *q : v) cudaFreeAsync(q, e->stream);
  v.clear();
}
static void free_temps(dpsnn_engine *e) {
  free_list(e, e->spare);
  free_list(e, e->temps);
}
template <typename T>
static int dalloc(dpsnn_engine *e, T **p, size_t n, bool temp = false) {
  void *q = nullptr;
  size_t bytes = std::max<size_t>(n * sizeof(T), 16);
  cudaError_t err = cudaMallocAsync(&q, bytes, e->stream);
  if (err == cudaErrorMemoryAllocation && !e->spare.empty()) {
    cudaGetLastError();
    free_list(e, e->spare);
    CK(cudaStreamSynchronize(e->stream));
    err = cudaMallocAsync(&q, bytes, e->stream);
  }
  if (err != cudaSuccess)
    return dpsnn_fail(DPSNN_E_NOMEM, "cudaMallocAsync(%zu bytes): %s", bytes, cudaGetErrorString(err));
  (temp ? e->temps : e->allocs).push_back(q);
  if (!temp) e->bytes += bytes;
  err = cudaMemsetAsync(q, 0, bytes, e->stream);
  if (err != cudaSuccess) return dpsnn_fail(DPSNN_E_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(err));
  *p = (T *)q;
  return 0;
}
#define DALLOC(ptr, n)                          \
  do {                                          \
    int rc_ = dalloc(e, &(ptr), (size_t)(n));   \
    if (rc_) return rc_;                        \
  } while (0)
#define TALLOC(ptr, n)                                \
  do {                                                \
    int rc_ = dalloc(e, &(ptr), (size_t)(n), true);   \
    if (rc_) return rc_;                              \
  } while (0)

// The fix-up table on the device: a bit per float that has one, and per result
// binade the fix-up inputs' least distance from the float their logarithm
// rounds to (half an ulp at a midpoint), with a margin of 1e-3 ulp for the
// last bits of the log that bath_lapse takes.  A bitmap built on the host is
// 32 MB to fill and upload, and its 184 699 logarithms as much again: 9 ms of
// a small network's build.
__global__ void fix_clear_kernel(double *near) { near[threadIdx.x] = INFINITY; }
__global__ void fix_table_kernel(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals, uint32_t n,
                                 uint32_t *bitmap, double *near, uint32_t *other) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t key = keys[i];
  if (key < 0x30000000u || key > 0x3F800000u) return;
  atomicOr(&bitmap[(key - 0x30000000u) >> 5], 1u << ((key - 0x30000000u) & 31));
  const float x = __uint_as_float(key);
  const double y = log((double)x);
  const float f = logf_cr_from(x, y);
  const uint32_t fb = __float_as_uint(f), E = (fb >> 23) & 0xFFu;
  // a fix-up that is not the float on the other side of the midpoint
  if (vals[i] != fb + (y < (double)f ? 1u : 0xFFFFFFFFu)) *other = 1;
  if ((fb & 0x7FFFFFu) == 0) return;   // always looked up
  const double dist = fmax(fabs(y - (double)f) - ldexp(1e-3, (int)E - 150), 0.0);
  atomicMin((unsigned long long *)&near[E], (unsigned long long)__double_as_longlong(dist));   // no negative doubles
}

static int load_logf_fixup(dpsnn_engine *e) {
  std::string path = std::string(dpsnn_library_dir()) + "/logf_fixup.bin";
  const char *envp = getenv("DPSNN_LOGF_FIXUP");
  if (envp) path = envp;
  FILE *f = fopen(path.c_str(), "rb");
  if (!f) return dpsnn_fail(DPSNN_E_PARAM, "cannot open %s (built with the engine)", path.c_str());
  uint32_t n = 0;
  bool ok = fread(&n, 4, 1, f) == 1;
  std::vector<uint32_t> keys(n), vals(n);
  ok = ok && fread(keys.data(), 4, n, f) == n;
  ok = ok && fread(vals.data(), 4, n, f) == n;
  fclose(f);
  if (!ok) return dpsnn_fail(DPSNN_E_PARAM, "truncated %s", path.c_str());
  {
    const size_t words = ((size_t)(0x3F800000u - 0x30000000u) + 1 + 31) / 32;
    uint32_t *dbm, *dkeys, *dvals, *dother, other = 0;
    double *dnear;
    DALLOC(dbm, words);
    DALLOC(dnear, 256);
    TALLOC(dkeys, n);
    TALLOC(dvals, n);
    TALLOC(dother, 1);
    CK(cudaMemcpyAsync(dkeys, keys.data(), 4ull * n, cudaMemcpyHostToDevice, e->stream));
    CK(cudaMemcpyAsync(dvals, vals.data(), 4ull * n, cudaMemcpyHostToDevice, e->stream));
    fix_clear_kernel<<<1, 256, 0, e->stream>>>(dnear);
    fix_table_kernel<<<(n + 255) / 256 + 1, 256, 0, e->stream>>>(dkeys, dvals, n, dbm, dnear, dother);
    CK(cudaGetLastError());
    CK(cudaMemcpyAsync(&other, dother, 4, cudaMemcpyDeviceToHost, e->stream));
    std::vector<double2> tab(LOG_TAB_N);
    for (int k = 0; k < LOG_TAB_N; k++) {   // the logarithm that goes with the rounded 64/i
      const double c = 64.0 / (LOG_TAB_0 + k);
      tab[k] = make_double2(c, c == 1.0 ? 0.0 : -log_cr(c));
    }
    double2 *dtab;
    DALLOC(dtab, LOG_TAB_N);
    CK(cudaMemcpyAsync(dtab, tab.data(), sizeof(double2) * LOG_TAB_N, cudaMemcpyHostToDevice, e->stream));
    CK(cudaStreamSynchronize(e->stream));
    if (other) {   // the table's values are searched: it stays on the device
      uint32_t *k, *v;
      DALLOC(k, n);
      DALLOC(v, n);
      CK(cudaMemcpyAsync(k, dkeys, 4ull * n, cudaMemcpyDeviceToDevice, e->stream));
      CK(cudaMemcpyAsync(v, dvals, 4ull * n, cudaMemcpyDeviceToDevice, e->stream));
      e->hnet.fix_keys = k;
      e->hnet.fix_vals = v;
      e->hnet.fix_n = n;
      CK(cudaMemcpyAsync(e->d.net, &e->hnet, sizeof e->hnet, cudaMemcpyHostToDevice, e->stream));
      CK(cudaStreamSynchronize(e->stream));
    }
    e->d.fix_bitmap = dbm;
    e->d.fix_near = dnear;
    e->d.log_tab = dtab;
  }
  return 0;
}

// ---- erflib Gaussian LUT on the host (erflib.c:41-169), C library exp
static double h_erfcc(double x) {
  double t, z, ans;
  z = fabs(x);
  t = 1.0 / (1.0 + 0.5 * z);
  ans = t * exp(-z * z - 1.26551223 +
                t * (1.00002368 +
                     t * (0.37409196 +
                          t * (0.09678418 +
                               t * (-0.18628806 +
                                    t * (0.27886807 +
                                         t * (-1.13520398 +
                                              t * (1.48851587 + t * (-0.82215223 + t * 0.17087277)))))))));
  return x >= 0.0 ? ans : 2.0 - ans;
}
static double h_normcum(double x, double mu, double sigma) {
  return 1 - 0.5 * h_erfcc((x - mu) / (sqrt(2.0) * sigma));
}
static double h_cutnormcum(double x, double mu, double sigma, double a, double b) {
  double n0 = h_normcum(a, mu, sigma);
  return (h_normcum(x, mu, sigma) - n0) / (h_normcum(b, mu, sigma) - n0);
}
static double h_findprob(double p, double mu, double sigma, double a, double b) {
  double err = 1e-6, x, xmin = a, xmax = b;
  int maxit = 256, i = 0;
  if (p <= 0.0) return a;
  if (p >= 1.0) return b;
  while ((xmax - xmin) > err && i < maxit) {
    x = (xmax + xmin) * 0.5;
    if (h_cutnormcum(x, mu, sigma, a, b) < p)
      xmin = x;
    else
      xmax = x;
    i++;
  }
  return (xmax + xmin) * 0.5;
}
static void h_gaussian_lut(double mu, double sigma, double xmin, double xmax, double *table) {
  if (sigma > 0.0) {
    double dp = 1.0 / 256.0, x0, x1 = xmin, p;
    int i;
    for (p = dp, i = 0; p <= 1.0; p += dp, i++) {
      x0 = x1;
      x1 = h_findprob(p, mu, sigma, xmin, xmax);
      table[i] = (x1 + x0) * 0.5;
    }
  } else {
    for (int i = 0; i < 256; i++) table[i] = mu;
  }
}

static void (*const BATH_KERNELS[4])(Dev) = {bath_kernel<false, false>, bath_kernel<false, true>,
                                             bath_kernel<true, false>, bath_kernel<true, true>};

// The kernels' shared-memory attributes, set once per device and process,
// before the device's first build: setting an attribute waits for the
// kernel's running instances, which would serialise the builds of engines
// built concurrently, and builds with other engines' steps.
static int set_kernel_attributes(int device) {
  static std::mutex mu;
  static std::vector<int> done;
  std::lock_guard<std::mutex> lock(mu);
  if ((int)done.size() <= device) done.resize(device + 1, 0);
  if (done[device]) return 0;
  CK(cudaFuncSetAttribute(gen_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GEN_SMEM));
  CK(cudaFuncSetAttribute(gen_fill_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          (int)(GEN_FILL_WARPS * sizeof(GenFillWarp))));
  // the bath's blocks stay resident for most of a step: with the largest
  // shared-memory carveout, the SMs that hold two of them still have room for
  // a block of the main stream's kernels that use shared memory
  for (auto bath : BATH_KERNELS) {
    CK(cudaFuncSetAttribute(bath, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BathSmem)));
    CK(cudaFuncSetAttribute(bath, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
  }
  done[device] = 1;
  return 0;
}

// ---- synapse generation, host side
static int gen_error(uint32_t err, uint32_t arg) {
  const char *what[] = {"", "too many synapses generated for neuron", "synaptic weight out of minSynWeight_f range",
                        "connection probability in (0,1e-5] is not supported", "delay >= env_D",
                        "zero mean synaptic efficacy",
                        "ERROR: delay level generated beyond the 80 max allowed delay levels, source neuron",
                        "ERROR: delay generated beyond the pair's DMax, source neuron"};
  return dpsnn_fail(DPSNN_E_MODEL, "synapse generation: %s (%u)", what[err], arg);
}

struct GenPlan {
  std::vector<GenRow> rows;
  std::vector<uint32_t> row_off;   // [nsub + 1] by source sub-population
  std::vector<GenTab> tabs;
  size_t c_len = 0;
};
#define GEN_TABS_MAX 4096   // distinct probabilities (a 10 x 10 stencil has at most 100 per pair)

// The warp form's plan; false where the thread form has to do: a weight may
// be rejected (NormDev's values are below sqrt(-2 ln 4e-18) = 8.96, so with
// sigma under 1/8.97 of the mean none is; near the denormal floats their
// rounding moves sigma and the weights too far), a probability that the
// reference does not take, or more distinct probabilities than tables.
static bool gen_plan(const NetConst &n, const std::vector<float> &prob, GenPlan &g) {
  const uint32_t st = n.stencil, M = n.max_mod;
  g.row_off.push_back(0);
  for (uint32_t s = 0; s < n.nsub; s++) {
    for (uint32_t t = 0; t < n.nsub; t++)
      for (uint32_t x = 0; x < st; x++)
        for (uint32_t y = 0; y < st; y++) {
          const float pf = prob[(((size_t)s * DPSNN_MAX_SUBPOP + t) * st + x) * st + y];
          if (!(pf > 0)) continue;
          const double mean = n.J[s * DPSNN_MAX_SUBPOP + t];
          if (!(pf > 0.00001f) || !(8.97 * fabs(n.DJ[s * DPSNN_MAX_SUBPOP + t]) <= 0.999) ||
              (mean != 0 && !(fabs(mean) > 1e-30)))
            return false;
          uint32_t k = 0;
          while (k < g.tabs.size() && g.tabs[k].pf != pf) k++;
          if (k == g.tabs.size()) {
            if (k == GEN_TABS_MAX) return false;
            g.tabs.push_back(GenTab{pf, (float)(1.0 / log2(1.0 - (double)pf)), 0, 0});
          }
          g.tabs[k].len = std::max(g.tabs[k].len, n.count[t] + 1);
          g.rows.push_back(GenRow{(int32_t)x - (int32_t)M, (int32_t)y - (int32_t)M, t, k});
        }
    g.row_off.push_back((uint32_t)g.rows.size());
  }
  for (GenTab &tb : g.tabs) {
    tb.off = (uint32_t)g.c_len;
    g.c_len += tb.len;
  }
  return g.c_len < (1u << 28);
}

// The CSR rows from the neurons' synapse counts, and the connectome's arrays.
static int alloc_rows(dpsnn_engine *e, const std::vector<uint32_t> &len) {
  const uint32_t N = e->hnet.N;
  std::vector<uint64_t> hrow(N + 1);
  hrow[0] = 0;
  for (uint32_t i = 0; i < N; i++) hrow[i + 1] = hrow[i] + len[i];
  e->S = hrow[N];
  DALLOC(e->d.row_ptr, N + 1);
  CK(cudaMemcpyAsync(e->d.row_ptr, hrow.data(), 8ull * (N + 1), cudaMemcpyHostToDevice, e->stream));
  DALLOC(e->d.post, e->S);
  DALLOC(e->d.w16, e->S);
  CK(cudaStreamSynchronize(e->stream));
  return 0;
}

static int generate_by_warps(dpsnn_engine *e, const GenPlan &g, const uint32_t *bath_tmpl, uint32_t *hist0) {
  const NetConst &n = e->hnet;
  Dev &d = e->d;
  const uint32_t N = n.N, nmod = n.nmod, hyps = n.mods_per_rank > 1 ? 2 : 1;
  GenRow *rows;
  GenTab *tabs;
  GenChain *chain;
  GenStart *start;
  double *gen_c;
  uint32_t *row_off, *tot;
  TALLOC(rows, g.rows.size());
  TALLOC(tabs, g.tabs.size());
  TALLOC(gen_c, g.c_len);
  TALLOC(row_off, n.nsub + 1);
  TALLOC(chain, 2 * nmod);
  TALLOC(start, (size_t)hyps * N);
  TALLOC(tot, (size_t)hyps * N);
  CK(cudaMemcpyAsync(rows, g.rows.data(), sizeof(GenRow) * g.rows.size(), cudaMemcpyHostToDevice, e->stream));
  CK(cudaMemcpyAsync(tabs, g.tabs.data(), sizeof(GenTab) * g.tabs.size(), cudaMemcpyHostToDevice, e->stream));
  CK(cudaMemcpyAsync(row_off, g.row_off.data(), 4 * g.row_off.size(), cudaMemcpyHostToDevice, e->stream));
  if (!g.tabs.empty())
    gen_tab_kernel<<<((uint32_t)g.tabs.size() + 31) / 32, 32, 0, e->stream>>>(tabs, (uint32_t)g.tabs.size(), gen_c);
  gen_chain_kernel<<<2 * nmod, 32, 0, e->stream>>>(d.net, rows, row_off, tabs, gen_c, chain, start, tot);
  CK(cudaGetLastError());
  std::vector<GenChain> rec(2 * nmod);
  std::vector<uint32_t> htot((size_t)hyps * N);
  CK(cudaMemcpyAsync(rec.data(), chain, sizeof(GenChain) * 2 * nmod, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaMemcpyAsync(htot.data(), tot, 4 * htot.size(), cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  // NormDev's cache from module to module of a rank
  std::vector<int32_t> hyp(nmod, 0);
  std::vector<uint2> cache(nmod, make_uint2(0, 0));
  for (uint32_t h = 0; h < n.P; h++) {
    bool full = false;
    uint2 c = make_uint2(0, 0);
    for (uint32_t m = h * n.mods_per_rank; m < (h + 1) * n.mods_per_rank; m++) {
      hyp[m] = full ? 1 : 0;
      cache[m] = c;
      const GenChain &r = rec[2 * m + hyp[m]];
      if (r.err) return gen_error(r.err, r.err_arg);
      if (r.set_out == 2) continue;   // no synapse: as the module found it
      full = r.set_out != 0;
      c = make_uint2(r.c_out[0], r.c_out[1]);
    }
  }
  std::vector<uint32_t> len(N);
  for (uint32_t m = 0; m < nmod; m++)
    memcpy(&len[(size_t)m * n.npcm], &htot[(size_t)hyp[m] * N + (size_t)m * n.npcm], 4ull * n.npcm);
  DALLOC(d.sub_off, (size_t)N * (n.D + 1));
  int rc = alloc_rows(e, len);
  if (rc) return rc;
  int32_t *dhyp;
  uint2 *dcache;
  unsigned long long *derr, herr = ~0ull;
  GenFillScratch *scratch = nullptr;
  TALLOC(dhyp, nmod);
  TALLOC(dcache, nmod);
  TALLOC(derr, 1);
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
  const uint32_t blocks = std::min<uint32_t>((N + GEN_FILL_WARPS - 1) / GEN_FILL_WARPS, (uint32_t)sms * 4);
  if (N && *std::max_element(len.begin(), len.end()) > GEN_FILL_LIST) TALLOC(scratch, (size_t)blocks * GEN_FILL_WARPS);
  CK(cudaMemcpyAsync(dhyp, hyp.data(), 4ull * nmod, cudaMemcpyHostToDevice, e->stream));
  CK(cudaMemcpyAsync(dcache, cache.data(), sizeof(uint2) * nmod, cudaMemcpyHostToDevice, e->stream));
  CK(cudaMemcpyAsync(derr, &herr, 8, cudaMemcpyHostToDevice, e->stream));
  gen_fill_kernel<<<blocks, 32 * GEN_FILL_WARPS, GEN_FILL_WARPS * sizeof(GenFillWarp), e->stream>>>(
      d.net, rows, row_off, tabs, gen_c, start, dhyp, dcache, d.row_ptr, d.sub_off, d.post, d.w16, scratch, derr,
      bath_tmpl, d.inv_nu, d.max_ext, d.sub);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(&herr, derr, 8, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  if (herr != ~0ull) {
    const uint32_t err = (uint32_t)(herr >> 22) & 15u;
    return gen_error(err, err == GEN_ERR_DELAY ? (uint32_t)herr & 0x3FFFFFu : (uint32_t)(herr >> 39));
  }
  memcpy(hist0, rec[2 * (n.mods_per_rank - 1) + hyp[n.mods_per_rank - 1]].hist, sizeof(uint32_t) * GEN_HIST);
  return 0;
}

static int generate_by_threads(dpsnn_engine *e, const std::vector<float> &prob, const uint32_t *bath_tmpl,
                               uint32_t *hist0) {
  const NetConst &n = e->hnet;
  Dev &d = e->d;
  const uint32_t N = n.N, D = n.D, P = n.P, nmod = n.nmod;
  float *dprob;
  TALLOC(dprob, prob.size());
  CK(cudaMemcpyAsync(dprob, prob.data(), prob.size() * sizeof(float), cudaMemcpyHostToDevice, e->stream));
  // pass A (both NormDev-cache hypotheses)
  GenRecord *drec;
  uint16_t *cnt_out;
  uint32_t *scratch;
  TALLOC(drec, 2 * nmod);
  TALLOC(cnt_out, 2ull * N * D);
  TALLOC(scratch, (size_t)2 * nmod * MAX_SYN_PER_NEURON);
  int32_t *dhyp;
  double *dcache;
  TALLOC(dhyp, nmod);
  TALLOC(dcache, nmod);
  gen_kernel<<<(2 * nmod + GEN_THREADS - 1) / GEN_THREADS, GEN_THREADS, GEN_SMEM, e->stream>>>(
      d.net, dprob, 0, drec, dhyp, dcache, cnt_out,
                                                          nullptr, nullptr, nullptr, nullptr, scratch,
                                                          bath_tmpl, nullptr, nullptr, nullptr);
  CK(cudaGetLastError());
  std::vector<GenRecord> rec(2 * nmod);
  CK(cudaMemcpyAsync(rec.data(), drec, sizeof(GenRecord) * 2 * nmod, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  for (uint32_t k = 0; k < 2 * nmod; k++)
    if (rec[k].err && !((k & 1) && (k / 2) % n.mods_per_rank == 0)) return gen_error(rec[k].err, rec[k].err_arg);
  // resolve the NormDev cache hand-off rank by rank, module by module
  std::vector<int32_t> hyp(nmod);
  std::vector<double> cache(nmod, 0.0);
  for (uint32_t h = 0; h < P; h++) {
    int32_t set = 0;
    double cval = 0.0;
    for (uint32_t mm = 0; mm < n.mods_per_rank; mm++) {
      uint32_t m = h * n.mods_per_rank + mm;
      int choose = 0;
      if (mm > 0 && set == 1) {
        const GenRecord &r1 = rec[2 * m + 1];
        if (!r1.used_normdev) {
          choose = 1;
        } else {
          float mean = r1.first_mean, sigma = r1.first_sigma;
          float wf = (float)(mean + cval * sigma);
          bool acc = (mean > 0.0) ? !((wf < 0.0) || (wf >= 2.0 * mean)) : !((wf <= 2.0 * mean) || (wf > 0));
          choose = acc ? 1 : 0;
        }
      }
      hyp[m] = choose;
      cache[m] = cval;
      const GenRecord &r = rec[2 * m + choose];
      if (r.used_normdev) {
        set = r.set_out;
        cval = r.cache_out;
      }
    }
  }
  CK(cudaMemcpyAsync(dhyp, hyp.data(), 4ull * nmod, cudaMemcpyHostToDevice, e->stream));
  CK(cudaMemcpyAsync(dcache, cache.data(), 8ull * nmod, cudaMemcpyHostToDevice, e->stream));
  // ---- CSR offsets from the chosen counts
  uint32_t *row_len;
  DALLOC(d.sub_off, (size_t)N * (D + 1));
  TALLOC(row_len, N);
  counts_to_csr_kernel<<<(N + 255) / 256, 256, 0, e->stream>>>(d.net, cnt_out, dhyp, d.sub_off, row_len);
  CK(cudaGetLastError());
  std::vector<uint32_t> hlen(N);
  CK(cudaMemcpyAsync(hlen.data(), row_len, 4ull * N, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  int rc = alloc_rows(e, hlen);
  if (rc) return rc;
  // ---- pass B: regenerate the chosen hypothesis straight into the CSR
  gen_kernel<<<(nmod + GEN_THREADS - 1) / GEN_THREADS, GEN_THREADS, GEN_SMEM, e->stream>>>(
      d.net, dprob, 1, drec, dhyp, dcache, cnt_out, d.row_ptr,
                                                      d.sub_off, d.post, d.w16, scratch, bath_tmpl, d.inv_nu,
                                                      d.max_ext, d.sub);
  CK(cudaGetLastError());
  std::vector<GenRecord> recB(nmod);
  CK(cudaMemcpyAsync(recB.data(), drec, sizeof(GenRecord) * nmod, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  for (uint32_t m = 0; m < nmod; m++)
    if (recB[m].err) return dpsnn_fail(DPSNN_E_MODEL, "synapse generation pass B error %d", recB[m].err);
  memcpy(hist0, recB[n.mods_per_rank - 1].hist, sizeof(uint32_t) * GEN_HIST);
  return 0;
}

// A rank's bath event slots.  A neuron has 1/invNuExt events per step on
// average, Poisson distributed, one more at step 0 (nextBath = 0), and at most
// its cap, 20 times the mean.  The rank's mean and 32 deviations (passed with a
// probability below 1e-100; checked once a round), no more than its caps, and a
// quarter of them at least: an event takes 16 bytes, in two buffers, and all the
// caps of the 24x24 network 1.1 GB, a quarter 0.3.  The ranks' rows closer
// together are slower by where they lie (a quiet 24x24 step 217 us, 213 with a
// quarter, 215 with all).
static uint64_t bath_slots(const uint32_t *max_ext, const double *inv_nu, uint32_t neurons) {
  uint64_t caps = 0;
  double mean = 0;
  for (uint32_t i = 0; i < neurons; i++) {
    if (!(inv_nu[i] > 0)) continue;
    caps += max_ext[i];
    mean += std::min((double)max_ext[i], 1.0 + 1.0 / inv_nu[i]);
  }
  return std::min(caps, std::max(caps / 4, (uint64_t)(mean + 32.0 * sqrt(mean)) + 64));
}

static int engine_build(dpsnn_engine *e, const dpsnn_params *p, const dpsnn_options *o) {
  NetConst &n = e->hnet;
  memset(&n, 0, sizeof n);
  if (p->nsub == 0 || p->nsub > DPSNN_MAX_SUBPOP)
    return dpsnn_fail(DPSNN_E_PARAM, "number of sub-populations %u out of range", p->nsub);
  if (p->stencil_dim == 0 || !p->spec || !p->bath) return dpsnn_fail(DPSNN_E_PARAM, "missing stencil description");
  if (p->D == 0 || p->D > RING_SLOTS) return dpsnn_fail(DPSNN_E_PARAM, "env_D=%u out of range [1,%d]", p->D, RING_SLOTS);
  if (p->glob_h == 0) return dpsnn_fail(DPSNN_E_PARAM, "env_globH must be >= 1");
  n.nsub = p->nsub;
  n.npcm = 0;
  for (uint32_t s = 0; s < n.nsub; s++) {
    n.offset[s] = n.npcm;
    n.count[s] = p->count[s];
    n.npcm += p->count[s];
  }
  if (n.npcm == 0) return dpsnn_fail(DPSNN_E_PARAM, "neuronsPerCM <= 0");
  n.cfx = p->cfx;
  n.cfy = p->cfy;
  n.nmod = p->cfx * p->cfy;
  if (n.nmod == 0) return dpsnn_fail(DPSNN_E_PARAM, "empty grid");
  if ((n.nmod % p->glob_h) != 0 || p->glob_h > n.nmod)
    return dpsnn_fail(DPSNN_E_PARAM, "#processes and #cort. columns must be multiple OR equal");
  n.P = p->glob_h;
  n.mods_per_rank = n.nmod / n.P;
  n.locN = n.npcm * n.mods_per_rank;
  n.N = n.locN * n.P;
  if ((uint64_t)n.npcm * n.nmod >= (1ull << 25))
    return dpsnn_fail(DPSNN_E_PARAM, "network of %llu neurons exceeds the engine limit of 2^25",
                      (unsigned long long)n.npcm * n.nmod);
  n.D = p->D;
  n.stencil_dim = p->stencil_dim;
  n.max_mod = p->stencil_dim - 1;
  n.stencil = 2 * p->stencil_dim - 1;
  for (uint32_t s = 0; s < n.nsub; s++) {
    n.Tau[s] = p->Tau[s];
    n.Theta[s] = p->Theta[s];
    n.H[s] = p->H[s];
    n.Tarp[s] = p->Tarp[s];
    n.AlphaC[s] = p->AlphaC[s];
    n.TauC[s] = p->TauC[s];
    auto reciprocal = [](double x) { return x > 1e-100 && x < 1e100 ? 1.0 / x : 0.0; };
    n.r_tau[s] = reciprocal(n.Tau[s]);
    n.r_tauC[s] = reciprocal(n.TauC[s]);
    n.gC[s] = p->gC[s];
    n.NuExt[s] = p->NuExt[s];
    for (uint32_t t = 0; t < n.nsub; t++) {
      n.J[s * DPSNN_MAX_SUBPOP + t] = p->J[s * p->nsub + t];
      n.DJ[s * DPSNN_MAX_SUBPOP + t] = p->DJ[s * p->nsub + t];
      n.DMin[s * DPSNN_MAX_SUBPOP + t] = p->DMin[s * p->nsub + t];
      n.DMax[s * DPSNN_MAX_SUBPOP + t] = p->DMax[s * p->nsub + t];
    }
  }
  {
    double dmin = 1e36, dmax = 0;
    for (uint32_t s = 0; s < n.nsub; s++)
      for (uint32_t t = 0; t < n.nsub; t++) {
        if (n.DMax[s * DPSNN_MAX_SUBPOP + t] > dmax) dmax = n.DMax[s * DPSNN_MAX_SUBPOP + t];
        if (n.DMin[s * DPSNN_MAX_SUBPOP + t] < dmin) dmin = n.DMin[s * DPSNN_MAX_SUBPOP + t];
      }
    n.delay_min = (uint32_t)dmin;
    n.delay_max = (uint32_t)dmax;
    n.delay_exp = p->delay_exponential ? 1u : 0u;
    n.inv_log_tn = (float)(1.0 / log_cr(0.05));
  }
  if (!(p->min_syn_weight_f < 0) || p->min_syn_weight_f < -6.0f)
    return dpsnn_fail(DPSNN_E_PARAM, "env_minSynWeigth out of range -6.000000 - 0.0");
  n.f2w = -32767 / p->min_syn_weight_f;
  n.w2f = p->min_syn_weight_f / -32767;
  n.min_w = p->min_syn_weight_f;
  n.global_seed = p->global_seed;
  n.start_pl = p->start_plasticity_ms;
  n.stop_pl = p->stop_plasticity_ms;
  n.stdp_on = (p->start_plasticity_ms <= p->stop_plasticity_ms &&
               p->start_plasticity_ms < (p->total_sim_time_ms ? p->total_sim_time_ms : 0xFFFFFFFFu)) ? 1 : 0;
  n.causal_tab[0] = p->stdp_causalMax * p->stdp_multiplier;
  n.causal_tab[1] = n.causal_tab[0];
  n.anti_tab[0] = p->stdp_antiCausalCoeff * p->stdp_antiCausalMax * p->stdp_multiplier;
  for (int i = 1; i < 128; i++) n.causal_tab[i] = (1 - 1 / p->stdp_tau_ms) * n.causal_tab[i - 1];
  for (int i = 1; i < 128; i++) n.anti_tab[i] = (1 - 1 / p->stdp_tau_ms) * n.anti_tab[i - 1];
  n.stdp_drift = p->stdp_drift;
  n.stdp_tauDecay = p->stdp_tauDecay_s;
  n.ev_cap = (o && o->events_per_neuron) ? o->events_per_neuron : DEFAULT_EVENT_CAP;
  {  // tuning knob: the largest event count of the thread-per-neuron path
    const char *lm = getenv("DPSNN_LIGHT_EVENTS");
    n.light_max = lm ? (uint32_t)atoi(lm) : LOCAL_EVENTS;
    if (n.light_max < 1 || n.light_max > LOCAL_EVENTS) n.light_max = LOCAL_EVENTS;
  }
  // at least what the thread-per-neuron path reads of a bucket, and even: the
  // sorted streams of two doubles per event start at a multiple of 16 bytes
  n.ev_cap = std::min(4096u, std::max<uint32_t>(LOCAL_EVENTS, n.ev_cap));
  n.ev_cap += n.ev_cap & 1;
  if (!(o && o->events_per_neuron)) {   // default: at most 16 GiB of event slots
    while (n.ev_cap > 64 && 8ull * n.ev_cap * n.N > (16ull << 30)) n.ev_cap >>= 1;
  }
  n.ovf_cap = (o && o->overflow_events) ? o->overflow_events : (1u << 22);

  Dev &d = e->d;
  const uint32_t N = n.N, D = n.D, P = n.P;
  DALLOC(d.net, 1);
  CK(cudaMemcpyAsync(d.net, &n, sizeof n, cudaMemcpyHostToDevice, e->stream));
  // bath LUTs (initLUT, DPSNN_LIFCAcorticalModuleGen.cpp:347-356)
  {
    std::vector<double> lut((size_t)n.nsub * 256);
    for (uint32_t s = 0; s < n.nsub; s++) {
      float J = p->JExt[s], DJ = p->DJExt[s];
      h_gaussian_lut(J, J * DJ, 0.0, 2.0 * J, &lut[(size_t)s * 256]);
    }
    DALLOC(d.lut, lut.size());
    CK(cudaMemcpyAsync(d.lut, lut.data(), lut.size() * sizeof(double), cudaMemcpyHostToDevice, e->stream));
    CK(cudaStreamSynchronize(e->stream));
  }
  // mirrored stencil probabilities (initProbConnectMatrix, LIFCAconnectome.cpp:136-198)
  const uint32_t st = n.stencil;
  std::vector<float> prob((size_t)DPSNN_MAX_SUBPOP * DPSNN_MAX_SUBPOP * st * st, 0.0f);
  {
    const uint32_t M = n.max_mod, S = p->stencil_dim;
    for (uint32_t s = 0; s < n.nsub; s++)
      for (uint32_t t = 0; t < n.nsub; t++)
        for (uint32_t x = 0; x <= M; x++)
          for (uint32_t y = 0; y <= M; y++) {
            float v = p->spec[((size_t)(s * n.nsub + t) * S + x) * S + y];
            auto at = [&](uint32_t X, uint32_t Y) -> float & {
              return prob[(((size_t)s * DPSNN_MAX_SUBPOP + t) * st + X) * st + Y];
            };
            at(M + x, M + y) = v;
            at(M - x, M + y) = v;
            at(M - x, M - y) = v;
            at(M + x, M - y) = v;
          }
  }
  // neuron arrays
  DALLOC(d.v, N); DALLOC(d.c, N); DALLOC(d.tr, N); DALLOC(d.te, N);
  DALLOC(e->nb2[0], N); DALLOC(e->nb2[1], N);
  d.nb = e->nb2[0];
  d.nb_prev = e->nb2[1];
  DALLOC(d.inv_nu, N); DALLOC(d.max_ext, N); DALLOC(d.sub, N); DALLOC(d.fired, N);
  DALLOC(d.last_spike_ms, N);
  e->grid_neuron = (N + NEURON_BLOCK - 1) / NEURON_BLOCK;
  DALLOC(d.block_fired, e->grid_neuron);
  DALLOC(d.fired_bits, (N + 31) / 32);
  DALLOC(d.ticket, 1);

  // ---- synapse generation
  const uint32_t SD = p->stencil_dim;
  uint32_t *bath_tmpl;
  {
    TALLOC(bath_tmpl, SD * SD);
    std::vector<uint32_t> bath(p->bath, p->bath + SD * SD);
    CK(cudaMemcpyAsync(bath_tmpl, bath.data(), 4ull * SD * SD, cudaMemcpyHostToDevice, e->stream));
    int rc = set_kernel_attributes(e->device);
    if (rc) return rc;
  }
  uint32_t hist0[GEN_HIST];   // rank 0's stream after the build: its dynamics go on from there
  GenPlan plan;
  {
    const bool warp_form = gen_plan(n, prob, plan);
    int rc = warp_form ? generate_by_warps(e, plan, bath_tmpl, hist0) : generate_by_threads(e, prob, bath_tmpl, hist0);
    if (rc) return rc;
    e->spare.swap(e->temps);
  }
  // ---- run-over-group-end check (see DPSNN_synapse.c:211-265): the reference's
  // search continues past a (delay, source rank) group while the next entry has
  // the same presynaptic index; this happens only when the last source of a
  // delay group is also the first source of the next non-empty group.
  {
    uint32_t *gmax, *gmin;
    TALLOC(gmax, (size_t)P * D);
    TALLOC(gmin, (size_t)P * D);
    CK(cudaMemsetAsync(gmin, 0xFF, 4ull * P * D, e->stream));
    group_extrema_kernel<<<std::min<uint32_t>(4096, (N + 7) / 8), 256, 0, e->stream>>>(d.net, d.row_ptr,
                                                                                     d.sub_off, d.post, gmax, gmin);
    CK(cudaGetLastError());
    std::vector<uint32_t> hmax((size_t)P * D), hmin((size_t)P * D);
    CK(cudaMemcpyAsync(hmax.data(), gmax, 4ull * P * D, cudaMemcpyDeviceToHost, e->stream));
    CK(cudaMemcpyAsync(hmin.data(), gmin, 4ull * P * D, cudaMemcpyDeviceToHost, e->stream));
    CK(cudaStreamSynchronize(e->stream));
    for (uint32_t h = 0; h < P; h++)
      for (uint32_t dl = 0; dl < D; dl++) {
        if (hmin[h * D + dl] == 0xFFFFFFFFu) continue;
        uint32_t dn = dl + 1;
        while (dn < D && hmin[h * D + dn] == 0xFFFFFFFFu) dn++;
        if (dn < D && hmax[h * D + dl] == hmin[h * D + dn])
          return dpsnn_fail(DPSNN_E_MODEL,
                            "rank %u: neuron %u ends delay group %u and starts group %u; the reference's "
                            "search would run across the group boundary (not reproduced)",
                            h, hmax[h * D + dl], dl, dn);
      }
  }
  // ---- STDP arrays
  if (n.stdp_on && e->S > 0xFFFFFFFFull)   // in_idx holds 32-bit synapse indices
    return dpsnn_fail(DPSNN_E_CAPACITY, "plasticity supports at most 2^32-1 synapses (%llu generated)",
                      (unsigned long long)e->S);
  if (n.stdp_on) {
    DALLOC(d.tderiv, e->S);
    DALLOC(d.last_act, e->S);
    DALLOC(d.in_ptr, N + 1);
    DALLOC(d.in_idx, e->S);
    unsigned long long *fill;
    TALLOC(fill, N);
    in_count_kernel<<<2048, 256, 0, e->stream>>>(d.net, d.post, e->S, d.in_ptr);
    CK(cudaGetLastError());
    std::vector<uint64_t> ip(N + 1);
    CK(cudaMemcpyAsync(ip.data(), d.in_ptr, 8ull * (N + 1), cudaMemcpyDeviceToHost, e->stream));
    CK(cudaStreamSynchronize(e->stream));
    for (uint32_t i = 0; i < N; i++) {
      if (ip[i + 1] >= 2 * MAX_SYN_PER_NEURON)
        return dpsnn_fail(DPSNN_E_MODEL, "ERROR too many syn incoming on neuron glob_n=%u", i);
      ip[i + 1] += ip[i];
    }
    CK(cudaMemcpyAsync(d.in_ptr, ip.data(), 8ull * (N + 1), cudaMemcpyHostToDevice, e->stream));
    in_fill_kernel<<<2048, 256, 0, e->stream>>>(d.net, d.post, e->S, d.in_ptr, fill, d.in_idx);
    CK(cudaGetLastError());
  }
  // ---- ring, events, bath
  DALLOC(d.ring_ids, (size_t)RING_SLOTS * N);
  DALLOC(d.ring_te, (size_t)RING_SLOTS * N);
  DALLOC(d.ring_cnt, RING_SLOTS);
  DALLOC(d.ev_cnt, N);
  DALLOC(d.ev, (size_t)N * n.ev_cap);
  DALLOC(d.ovf_cnt, 1);
  DALLOC(d.ovf, n.ovf_cap);
  DALLOC(d.heavy_list, 4ull * N);
  {   // huge_kernel's global scratch: one neuron of up to HEAVY_MAX events per block
    int nsm = 148;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, e->device);
    DALLOC(d.huge_tau, (size_t)nsm * HEAVY_MAX);
    DALLOC(d.huge_key, (size_t)nsm * HEAVY_MAX);
    DALLOC(d.huge_val, (size_t)nsm * HEAVY_MAX);
  }
  DALLOC(d.heavy_cnt, 2);
  DALLOC(d.t, 1);
  DALLOC(d.bath_t, P);
  DALLOC(d.flags, 4);
  DALLOC(d.events, 1);
  init_neurons_kernel<<<(N + 255) / 256, 256, 0, e->stream>>>(d);
  CK(cudaGetLastError());
  {
    std::vector<uint32_t> mx(N);
    std::vector<double> inv(N);
    CK(cudaMemcpyAsync(mx.data(), d.max_ext, 4ull * N, cudaMemcpyDeviceToHost, e->stream));
    CK(cudaMemcpyAsync(inv.data(), d.inv_nu, 8ull * N, cudaMemcpyDeviceToHost, e->stream));
    CK(cudaStreamSynchronize(e->stream));
    std::vector<uint64_t> base(P + 1, 0);
    for (uint32_t h = 0; h < P; h++)
      base[h + 1] = base[h] + bath_slots(&mx[(size_t)h * n.locN], &inv[(size_t)h * n.locN], n.locN);
    uint32_t mx_max = 0;
    for (uint32_t i = 0; i < N; i++) {
      mx_max = std::max(mx_max, mx[i]);
      e->low_caps |= inv[i] > 0 && mx[i] < 16;
    }
    if (mx_max > BATH_MAX_EXT)
      return dpsnn_fail(DPSNN_E_CAPACITY, "maxExternCurrentCount %u exceeds what the bath ring holds (%d)", mx_max,
                        BATH_MAX_EXT);
    DALLOC(d.bath_rank_base, P + 1);
    CK(cudaMemcpyAsync(d.bath_rank_base, base.data(), 8ull * (P + 1), cudaMemcpyHostToDevice, e->stream));
    for (int b = 0; b < 2; b++) {
      DALLOC(e->bath_ev2[b], base[P]);   // below 2^25 * BATH_MAX_EXT < 2^32
      DALLOC(e->bath_at2[b], N);
    }
    d.bath_ev = e->bath_ev2[0];
    d.bath_at = e->bath_at2[0];
    // dynamics streams: SetRandomSeed(loc_h) (DPSNN_localNet_init.c:283).
    // Rank 0 continues its generation stream; others re-initialise.
    std::vector<uint32_t> hist((size_t)P * BATH_KEEP), kept(P, BATH_HIST);
    for (uint32_t h = 0; h < P; h++) {
      uint32_t h55[55];
      if (h == 0) {
        memcpy(h55, hist0, sizeof h55);
      } else {
        Ran3 g;
        memset(&g, 0, sizeof g);
        g.idum = -(int32_t)h;
        // table initialisation only; the draw SetRandomSeed makes is x[0]
        int32_t mj = MSEED - (int32_t)h, mk;
        mj = (mj < 0 ? -mj : mj) % MBIG;
        g.ma[55] = mj;
        mk = 1;
        for (int i = 1; i <= 54; i++) {
          int ii = (21 * i) % 55;
          g.ma[ii] = mk;
          mk = mj - mk;
          if (mk < 0) mk += MBIG;
          mj = g.ma[ii];
        }
        for (int k = 1; k <= 4; k++)
          for (int i = 1; i <= 55; i++) {
            g.ma[i] -= g.ma[1 + (i + 30) % 55];
            if (g.ma[i] < 0) g.ma[i] += MBIG;
          }
        g.inext = 0;
        r3_history(g, h55);
      }
      // h55 is x[-55..-1].  The neurons' draws start at x[1]: the history is
      // x[1-BATH_HIST..0], x[0] = x[-55] - x[-24] and the older ones by the
      // recurrence backwards, x[k] = x[k+55] + x[k+31] (mod MBIG)
      uint32_t *x = &hist[(size_t)h * BATH_KEEP] + BATH_HIST - 1;   // x[0]
      for (int k = 0; k < 55; k++) x[k - 55] = h55[k];
      x[0] = x[-55] >= x[-24] ? x[-55] - x[-24] : x[-55] + MBIG - x[-24];
      for (int k = -56; k > -BATH_HIST; k--) x[k] = (uint32_t)(((uint64_t)x[k + 55] + x[k + 31]) % MBIG);
    }
    DALLOC(d.bath_hist, (size_t)P * BATH_KEEP);
    DALLOC(d.bath_kept, P);
    CK(cudaMemcpyAsync(d.bath_hist, hist.data(), 4ull * P * BATH_KEEP, cudaMemcpyHostToDevice, e->stream));
    CK(cudaMemcpyAsync(d.bath_kept, kept.data(), 4ull * P, cudaMemcpyHostToDevice, e->stream));
    CK(cudaStreamSynchronize(e->stream));
  }
  int rc = load_logf_fixup(e);
  if (rc) return rc;
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device);
  e->sms = sms;
  default_grids(e, 0, 0, 0);
  // The tail's blocks.  A block per 32 neurons where few neurons can have more
  // than 256 events in a step (one per incoming synapse at most): with one per
  // 256, 80 steps of 32 networks of 1250 to 20 000 neurons took 258 ms against
  // 146 around their onset, and 65 against 45 later; a graph of 16 networks of
  // 120 to 1920 neurons with 150 synapses each takes 3.6 ms, 3.9 with one per 8.
  // One per 8 where a burst brings most neurons more: a step of 2000 neurons with
  // 1900 synapses each in their burst 1.84 ms from 3.92, of 1250 with 1125 0.27
  // from 0.44.  Smaller buckets than the default's send neurons of fewer events
  // there, and each searches the overflow list: a block per SM (the burst of 1250
  // neurons with 64 and 512 slots: 1.38 and 0.39 ms per step, 4.5 and 1.09 with a
  // block per 32 neurons).
  const uint32_t per_block = e->S > 2ull * HEAVY_WARP_MAX * N ? 8 : 32;
  e->grid_tail = n.ev_cap < DEFAULT_EVENT_CAP ? (uint32_t)sms
                                              : std::min<uint32_t>((uint32_t)sms, (N + per_block - 1) / per_block);
  e->grid_huge = (uint32_t)sms;
  free_temps(e);   // after their last use on this stream
  CK(cudaStreamSynchronize(e->stream));
  return 0;
}

extern "C" int dpsnn_create(const dpsnn_params *p, const dpsnn_options *opts, dpsnn_engine **out) {
  if (!p || !out) return dpsnn_fail(DPSNN_E_PARAM, "null argument");
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return dpsnn_fail(DPSNN_E_CUDA, "no CUDA device available");
  dpsnn_engine *e = new dpsnn_engine();
  if (opts && opts->device >= 0 && opts->device < ndev) {
    e->device = opts->device;
  } else {
    cudaGetDevice(&e->device);
  }
  // The bath of the next step runs beside this step's kernels.  A network that
  // fills the GPU waits for its main stream, whose blocks go first when both
  // wait for room; a small one for its bath, whose few blocks would otherwise
  // wait for the update's to drain (16 000 neurons in 64 busy ranks: 76 us per
  // step against 67).
  uint64_t npcm = 0;
  for (uint32_t s = 0; s < std::min<uint32_t>(p->nsub, DPSNN_MAX_SUBPOP); s++) npcm += p->count[s];
  const uint64_t neurons = npcm * p->cfx * p->cfy;
  const bool small = small_form(neurons, p->glob_h ? neurons / p->glob_h : 0);
  int prio_least = 0, prio_greatest = 0;
  bool ok = cudaSetDevice(e->device) == cudaSuccess &&
            cudaDeviceGetStreamPriorityRange(&prio_least, &prio_greatest) == cudaSuccess &&
            cudaStreamCreateWithPriority(&e->stream, cudaStreamNonBlocking, small ? prio_least : prio_greatest) == cudaSuccess &&
            cudaStreamCreateWithPriority(&e->bath_stream, cudaStreamNonBlocking, small ? prio_greatest : prio_least) == cudaSuccess;
  for (int b = 0; b < 2 && ok; b++)
    ok = cudaEventCreateWithFlags(&e->ev_bath[b], cudaEventDisableTiming) == cudaSuccess &&
         cudaEventCreateWithFlags(&e->ev_neuron[b], cudaEventDisableTiming) == cudaSuccess;
  ok = ok && cudaEventCreateWithFlags(&e->ev_start, cudaEventDisableTiming) == cudaSuccess;
  ok = ok && cudaStreamCreateWithFlags(&e->read_stream, cudaStreamNonBlocking) == cudaSuccess;
  for (int k = 0; k < RING_SLOTS && ok; k++)
    ok = cudaEventCreateWithFlags(&e->ev_slot[k], cudaEventDisableTiming) == cudaSuccess;
  // the read buffer: what 80 steps of a network at rest make several times
  // over (a burst's lists are copied one by one)
  e->h_read_cap = (uint32_t)std::min<uint64_t>(32768, std::max<uint64_t>(1024, 4 * neurons));
  const size_t read_bytes = sizeof(SpikeRead) + 12ull * e->h_read_cap;
  ok = ok && cudaHostAlloc((void **)&e->h_read, read_bytes + 8, cudaHostAllocMapped) == cudaSuccess;
  if (ok) e->h_pin = reinterpret_cast<uint32_t *>(reinterpret_cast<char *>(e->h_read) + read_bytes);
  if (!ok) {
    const int dev = e->device;
    dpsnn_destroy(e);
    return dpsnn_fail(DPSNN_E_CUDA, "cannot set up device %d", dev);
  }
  int rc = engine_build(e, p, opts);
  if (rc) {
    dpsnn_destroy(e);
    return rc;
  }
  *out = e;
  return 0;
}

extern "C" void dpsnn_destroy(dpsnn_engine *e) {
  if (!e) return;
  cudaSetDevice(e->device);
  if (e->bath_stream) cudaStreamSynchronize(e->bath_stream);
  if (e->read_stream) cudaStreamSynchronize(e->read_stream);
  if (e->stream) {
    free_temps(e);   // a build that stopped early
    for (void *q : e->allocs) cudaFreeAsync(q, e->stream);
    cudaStreamSynchronize(e->stream);
  }
  collect_timings(e);
  for (cudaEvent_t ev : e->event_pool) cudaEventDestroy(ev);
  for (int b = 0; b < 2; b++) {
    if (e->ev_bath[b]) cudaEventDestroy(e->ev_bath[b]);
    if (e->ev_neuron[b]) cudaEventDestroy(e->ev_neuron[b]);
  }
  if (e->ev_start) cudaEventDestroy(e->ev_start);
  for (int k = 0; k < RING_SLOTS; k++)
    if (e->ev_slot[k]) cudaEventDestroy(e->ev_slot[k]);
  if (e->read_stream) {
    cudaStreamSynchronize(e->read_stream);
    cudaStreamDestroy(e->read_stream);
  }
  if (e->h_read) cudaFreeHost(e->h_read);
  if (e->bath_stream) cudaStreamDestroy(e->bath_stream);
  if (e->stream) cudaStreamDestroy(e->stream);
  delete e;
}

static int flags_error(uint32_t f);
static int check_flags(dpsnn_engine *e) {
  uint32_t f = 0;
  CK(cudaMemcpyAsync(&f, e->d.flags, 4, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  return flags_error(f);
}
static int flags_error(uint32_t f) {
  if (!f) return 0;
  if (f & F_TIME_WINDOW) return dpsnn_fail(DPSNN_E_MODEL, "ERROR in neu dynamic: input currentTime in wrong ms");
  if (f & F_NO_TARGET) return dpsnn_fail(DPSNN_E_MODEL, "ERROR neuSpikToAxSp: no forw host targ for a spiking neuron");
  if (f & F_TOO_MANY_INPUTS)
    return dpsnn_fail(DPSNN_E_CAPACITY, "more than %d synaptic inputs on one neuron in one step", MAX_INPUTS_PER_STEP);
  if (f & F_OVERFLOW) return dpsnn_fail(DPSNN_E_CAPACITY, "event overflow list full");
  if (f & F_BATH_DRAWS) return dpsnn_fail(DPSNN_E_CAPACITY, "bath draw buffer exhausted");
  return dpsnn_fail(DPSNN_E_MODEL, "device error flags 0x%x", f);
}

// Kernel timing records an event pair per kernel family and step on the
// engine stream without synchronising; dpsnn_kernel_times reads them.
static cudaEvent_t pool_event(dpsnn_engine *e) {
  if (e->event_pool.empty()) {
    cudaEvent_t ev;
    cudaEventCreate(&ev);
    return ev;
  }
  cudaEvent_t ev = e->event_pool.back();
  e->event_pool.pop_back();
  return ev;
}
static void timed_launch_begin(dpsnn_engine *e, int k, cudaStream_t st = nullptr) {
  if (!e->timing) return;
  dpsnn_engine::TimedLaunch tl;
  tl.family = k;
  tl.a = pool_event(e);
  tl.b = pool_event(e);
  tl.st = st ? st : e->stream;
  cudaEventRecord(tl.a, tl.st);
  e->pending.push_back(tl);
}
static void timed_launch_end(dpsnn_engine *e, int k) {
  if (!e->timing) return;
  (void)k;
  cudaEventRecord(e->pending.back().b, e->pending.back().st);
}
static void collect_timings(dpsnn_engine *e) {
  for (auto &tl : e->pending) {
    cudaEventSynchronize(tl.b);
    float ms = 0;
    cudaEventElapsedTime(&ms, tl.a, tl.b);
    e->ktime[tl.family] += ms * 1e-3;
    e->klaunch[tl.family]++;
    e->event_pool.push_back(tl.a);
    e->event_pool.push_back(tl.b);
  }
  e->pending.clear();
}

// The bath of step t (bath_kernel) depends only on the ranks' RNG streams
// and nextBath, not on synaptic input, so it runs one step ahead on its own
// stream, overlapping the delivery and neuron update of the previous step.
// Its outputs (per-neuron bath events) and nextBath live in two buffers by
// step parity: bath(t) writes set t&1 once neuron(t-2), the last reader of
// that set, is done; neuron(t) reads set t&1 once bath(t) is done.
static void enqueue_bath(dpsnn_engine *e, uint32_t t) {
  Dev db = e->d;
  const int b = t & 1;
  db.nb_prev = e->nb2[b ^ 1];
  db.nb = e->nb2[b];
  db.bath_ev = e->bath_ev2[b];
  db.bath_at = e->bath_at2[b];
  cudaStreamWaitEvent(e->bath_stream, e->ev_neuron[b], 0);
  timed_launch_begin(e, 2, e->bath_stream);
  // each rank's block keeps its step in d.bath_t (baths are launched in step order)
  const auto kernel = BATH_KERNELS[2 * (e->hnet.fix_n != 0) + e->low_caps];
  kernel<<<e->hnet.P, BATH_THREADS, sizeof(BathSmem), e->bath_stream>>>(db);
  e->launches++;
  timed_launch_end(e, 2);
  cudaEventRecord(e->ev_bath[b], e->bath_stream);
}

// A kernel of the main stream.  With `early` it may be brought up while the
// kernel before it on the stream still runs (it starts by waiting for that
// kernel's end): the gap between two dependent kernels is then about 1 us.
// A kernel that takes nothing from the one before it need not wait so, but
// ends after it (end_after_previous).
template <typename K>
static void launch_main(dpsnn_engine *e, K kernel, uint32_t grid, uint32_t block, const Dev &d, bool early) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.stream = e->stream;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = a;
  c.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&c, kernel, d);
  e->launches++;
}

// Slot t of the ring is final: spike lists may be read (inside a graph: an
// event the graph records on every run).
static void record_slot(dpsnn_engine *e, uint32_t t) {
  if (e->capturing)
    cudaEventRecordWithFlags(e->ev_slot[t % RING_SLOTS], e->stream, cudaEventRecordExternal);
  else
    cudaEventRecord(e->ev_slot[t % RING_SLOTS], e->stream);
}

// The plasticity kernels around the delivery and after the update.
static void enqueue_causal(dpsnn_engine *e, const Dev &d) {
  timed_launch_begin(e, 4);
  causal_stdp_kernel<<<e->grid_deliver, 256, 0, e->stream>>>(d);
  timed_launch_end(e, 4);
  e->launches++;
}
static void enqueue_anti_log(dpsnn_engine *e, const Dev &d) {
  if (!d.stdp_log) return;
  stdp_anti_log_kernel<<<e->grid_deliver, 256, 0, e->stream>>>(d);
  e->launches++;
}
static void enqueue_ltp(dpsnn_engine *e, const Dev &d, uint32_t t) {
  if (d.probe_w && t % 1000 == 999 && t >= e->hnet.start_pl && t <= e->hnet.stop_pl) e->probe_t = t;
  timed_launch_begin(e, 4);
  ltp_kernel<<<e->grid_deliver, 256, 0, e->stream>>>(d);
  timed_launch_end(e, 4);
  e->launches++;
}

// A small network's step: three kernels.  Bath t+1 writes the buffers that
// step t-1 read, and follows step t's delivery.
static void enqueue_small(dpsnn_engine *e, const Dev &d, uint32_t t) {
  const int b = t & 1;
  if (e->hnet.stdp_on) {
    timed_launch_begin(e, 0);
    launch_main(e, compact_small_kernel, std::min<uint32_t>(e->grid_deliver, 32), DELIVER_THREADS, d, true);
    timed_launch_end(e, 0);
    record_slot(e, t);
    enqueue_causal(e, d);
    timed_launch_begin(e, 1);
    launch_main(e, deliver_kernel, e->grid_deliver, DELIVER_THREADS, d, false);
    timed_launch_end(e, 1);
    enqueue_anti_log(e, d);
  } else {
    timed_launch_begin(e, 1);
    launch_main(e, deliver_small_kernel, e->grid_deliver, DELIVER_THREADS, d, true);
    timed_launch_end(e, 1);
    record_slot(e, t);
  }
  cudaEventRecord(e->ev_neuron[b ^ 1], e->stream);
  enqueue_bath(e, t + 1);
  cudaStreamWaitEvent(e->stream, e->ev_bath[b], 0);
  timed_launch_begin(e, 3);
  // four warps per 32 neurons while all the blocks are resident at once (four
  // per SM), then two
  const uint32_t blocks = (e->hnet.N + 31) / 32;
  if (blocks <= 4 * (uint32_t)e->sms)
    launch_main(e, neuron_small_kernel<4>, blocks, 128, d, false);
  else
    launch_main(e, neuron_small_kernel<2>, blocks, 64, d, false);
  timed_launch_end(e, 3);
  if (e->hnet.stdp_on) enqueue_ltp(e, d, t);
  timed_launch_begin(e, 7);
  launch_main(e, tail_small_kernel, e->grid_tail, HEAVY_THREADS, d, !e->hnet.stdp_on);
  timed_launch_end(e, 7);
}

static void enqueue_large(dpsnn_engine *e, const Dev &d, uint32_t t) {
  const int b = t & 1;
  enqueue_bath(e, t + 1);
  timed_launch_begin(e, 0);
  compact_kernel<<<e->grid_neuron, NEURON_BLOCK, 0, e->stream>>>(d);
  timed_launch_end(e, 0);
  record_slot(e, t);
  if (e->hnet.stdp_on) enqueue_causal(e, d);
  timed_launch_begin(e, 1);
  deliver_kernel<<<e->grid_deliver, DELIVER_THREADS, 0, e->stream>>>(d);
  timed_launch_end(e, 1);
  enqueue_anti_log(e, d);
  cudaStreamWaitEvent(e->stream, e->ev_bath[b], 0);
  timed_launch_begin(e, 3);
  neuron_kernel<<<e->grid_neuron, NEURON_BLOCK, 0, e->stream>>>(d);
  timed_launch_end(e, 3);
  timed_launch_begin(e, 5);
  launch_main(e, heavy_sort_big_kernel, e->grid_heavy, HEAVY_SORT_THREADS, d, false);
  launch_main(e, heavy_sort_kernel, e->grid_heavy, HEAVY_SORT_THREADS, d, true);
  timed_launch_end(e, 5);
  timed_launch_begin(e, 7);
  launch_main(e, huge_kernel, e->grid_huge, HEAVY_THREADS, d, true);
  timed_launch_end(e, 7);
  timed_launch_begin(e, 6);
  launch_main(e, heavy_run_kernel, e->grid_heavy_run, 128, d, false);
  timed_launch_end(e, 6);
  timed_launch_begin(e, 7);
  launch_main(e, heavy_rest_kernel, e->grid_huge, 128, d, true);
  timed_launch_end(e, 7);
  cudaEventRecord(e->ev_neuron[b], e->stream);
  if (e->hnet.stdp_on) enqueue_ltp(e, d, t);
  end_step_kernel<<<1, 1, 0, e->stream>>>(d);
  e->launches += 4;
}

static int enqueue_step(dpsnn_engine *e) {
  const uint32_t t = e->t_host;
  const int b = t & 1;
  if (!e->bath_primed) {   // the first bath waits for the network build
    cudaEventRecord(e->ev_start, e->stream);
    cudaStreamWaitEvent(e->bath_stream, e->ev_start, 0);
    enqueue_bath(e, t);
    e->bath_primed = true;
  }
  if (e->d.stdp_log) {
    cudaMemsetAsync(e->d.stdp_log_cnt, 0, 4, e->stream);
    e->stdp_log_t = t;
  }
  Dev d = e->d;
  d.bath_ev = e->bath_ev2[b];
  d.bath_at = e->bath_at2[b];
  if (small_form(e->hnet.N, e->hnet.locN))
    enqueue_small(e, d, t);
  else
    enqueue_large(e, d, t);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return dpsnn_fail(DPSNN_E_CUDA, "kernel launch: %s", cudaGetErrorString(err));
  e->t_host++;
  return 0;
}

extern "C" int dpsnn_step(dpsnn_engine *e, uint32_t nsteps) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  cudaSetDevice(e->device);
  for (uint32_t k = 0; k < nsteps; k++) {
    int rc = enqueue_step(e);
    if (rc) return rc;
  }
  return 0;
}

extern "C" int dpsnn_step_many(dpsnn_engine *const *engines, uint32_t n, uint32_t nsteps) {
  if (!engines && n) return dpsnn_fail(DPSNN_E_PARAM, "null engine array");
  for (uint32_t i = 0; i < n; i++)
    if (!engines[i]) return dpsnn_fail(DPSNN_E_PARAM, "null engine %u", i);
  // one step of every engine in turn: each engine's kernels queue on its own
  // streams, so the networks' steps overlap on the device
  for (uint32_t k = 0; k < nsteps; k++)
    for (uint32_t i = 0; i < n; i++) {
      dpsnn_engine *e = engines[i];
      cudaSetDevice(e->device);
      int rc = enqueue_step(e);
      if (rc) return rc;
    }
  return 0;
}

// ------------------------------------------------------------------ graphs of batched steps
// nsteps steps of n engines queued as dpsnn_step_many does, recorded once into
// a CUDA graph and run as one launch: the host cost of a step of many small
// networks (a dozen launches and event operations per network) is paid once.
// A graph encodes the engines' ring slots and step parities, so it runs only
// when every engine is at the step (mod 80) it was recorded at; nsteps is a
// multiple of 80, so consecutive runs chain.
// The events that order an engine's two streams between steps, recorded at
// the streams' current ends: after a graph run (whose own copies of them are
// internal to the graph) later steps wait on everything before.
static void rearm_step_events(dpsnn_engine *e) {
  for (int b = 0; b < 2; b++) {
    cudaEventRecord(e->ev_neuron[b], e->stream);
    cudaEventRecord(e->ev_bath[b], e->bath_stream);
  }
}

struct dpsnn_graph {
  std::vector<dpsnn_engine *> engines;
  std::vector<uint32_t> t0;        // each engine's step (mod RING_SLOTS) at recording
  std::vector<cudaEvent_t> pre;    // per engine: its two streams' last work before a run
  uint32_t nsteps = 0;
  uint64_t launches_per_run = 0;
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaEvent_t fork = nullptr, done = nullptr;
};

extern "C" void dpsnn_graph_destroy(dpsnn_graph *g) {
  if (!g) return;
  cudaSetDevice(g->device);
  if (g->stream) cudaStreamSynchronize(g->stream);
  if (g->exec) cudaGraphExecDestroy(g->exec);
  if (g->graph) cudaGraphDestroy(g->graph);
  for (cudaEvent_t ev : g->pre) cudaEventDestroy(ev);
  if (g->fork) cudaEventDestroy(g->fork);
  if (g->done) cudaEventDestroy(g->done);
  if (g->stream) cudaStreamDestroy(g->stream);
  delete g;
}

extern "C" int dpsnn_graph_create(dpsnn_engine *const *engines, uint32_t n, uint32_t nsteps, dpsnn_graph **out) {
  if (!out || (!engines && n)) return dpsnn_fail(DPSNN_E_PARAM, "null argument");
  *out = nullptr;
  if (n == 0 || nsteps == 0 || nsteps % RING_SLOTS)
    return dpsnn_fail(DPSNN_E_PARAM, "a graph holds a positive multiple of %d steps of at least one engine",
                      RING_SLOTS);
  for (uint32_t i = 0; i < n; i++) {
    const dpsnn_engine *e = engines[i];
    if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine %u", i);
    if (e->device != engines[0]->device) return dpsnn_fail(DPSNN_E_PARAM, "engines on different devices");
    if (!e->bath_primed) return dpsnn_fail(DPSNN_E_STATE, "engine %u has not run its first step", i);
    if (e->timing || e->d.stdp_log || e->d.probe_w)
      return dpsnn_fail(DPSNN_E_STATE, "engine %u has kernel timing, the STDP event log or the LTP probe on", i);
    for (uint32_t k = 0; k < i; k++)
      if (engines[k] == e) return dpsnn_fail(DPSNN_E_PARAM, "engine %u is listed twice", i);
  }
  dpsnn_graph *g = new dpsnn_graph();
  g->device = engines[0]->device;
  g->nsteps = nsteps;
  g->engines.assign(engines, engines + n);
  cudaSetDevice(g->device);
  auto fail = [&](int rc) {
    dpsnn_graph_destroy(g);
    return rc;
  };
  if (cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&g->fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&g->done, cudaEventDisableTiming) != cudaSuccess)
    return fail(dpsnn_fail(DPSNN_E_CUDA, "cannot create the graph's stream and events"));
  g->pre.resize(2 * n, nullptr);
  for (auto &ev : g->pre)
    if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess)
      return fail(dpsnn_fail(DPSNN_E_CUDA, "cannot create the graph's events"));
  std::vector<uint32_t> t_saved(n);
  std::vector<uint64_t> l_saved(n);
  cudaError_t err = cudaStreamBeginCapture(g->stream, cudaStreamCaptureModeThreadLocal);
  if (err != cudaSuccess) return fail(dpsnn_fail(DPSNN_E_CUDA, "cudaStreamBeginCapture: %s", cudaGetErrorString(err)));
  cudaEventRecord(g->fork, g->stream);
  int rc = 0;
  for (uint32_t i = 0; i < n; i++) {
    dpsnn_engine *e = engines[i];
    t_saved[i] = e->t_host;
    l_saved[i] = e->launches;
    g->t0.push_back(e->t_host % RING_SLOTS);
    // both streams join the recording; the events they wait on between
    // each other are recorded inside it from here on
    cudaStreamWaitEvent(e->stream, g->fork, 0);
    cudaStreamWaitEvent(e->bath_stream, g->fork, 0);
    for (int b = 0; b < 2; b++) {
      cudaEventRecord(e->ev_neuron[b], e->stream);
      cudaEventRecord(e->ev_bath[b], e->bath_stream);
    }
    e->capturing = true;
  }
  for (uint32_t k = 0; k < nsteps && !rc; k++)
    for (uint32_t i = 0; i < n && !rc; i++) rc = enqueue_step(engines[i]);
  for (uint32_t i = 0; i < n; i++) {
    dpsnn_engine *e = engines[i];
    e->capturing = false;
    cudaEventRecord(g->pre[2 * i], e->stream);
    cudaEventRecord(g->pre[2 * i + 1], e->bath_stream);
    cudaStreamWaitEvent(g->stream, g->pre[2 * i], 0);
    cudaStreamWaitEvent(g->stream, g->pre[2 * i + 1], 0);
    g->launches_per_run += e->launches - l_saved[i];
    e->t_host = t_saved[i];   // nothing ran
    e->launches = l_saved[i];
  }
  err = cudaStreamEndCapture(g->stream, &g->graph);
  // the streams' order events were last recorded inside the capture: record
  // them again outside it, so that plain steps can wait on them (no step ran)
  for (uint32_t i = 0; i < n; i++) rearm_step_events(engines[i]);
  if (rc) return fail(rc);
  if (err != cudaSuccess) return fail(dpsnn_fail(DPSNN_E_CUDA, "cudaStreamEndCapture: %s", cudaGetErrorString(err)));
  err = cudaGraphInstantiate(&g->exec, g->graph, 0);
  if (err != cudaSuccess) return fail(dpsnn_fail(DPSNN_E_CUDA, "cudaGraphInstantiate: %s", cudaGetErrorString(err)));
  *out = g;
  return 0;
}

extern "C" int dpsnn_graph_run(dpsnn_graph *g) {
  if (!g) return dpsnn_fail(DPSNN_E_PARAM, "null graph");
  cudaSetDevice(g->device);
  const uint32_t n = (uint32_t)g->engines.size();
  for (uint32_t i = 0; i < n; i++)
    if (g->engines[i]->t_host % RING_SLOTS != g->t0[i])
      return dpsnn_fail(DPSNN_E_STATE, "engine %u is at step %u; the graph was recorded at a step = %u (mod %d)", i,
                        g->engines[i]->t_host, g->t0[i], RING_SLOTS);
  for (uint32_t i = 0; i < n; i++) {   // after the engines' queued work
    dpsnn_engine *e = g->engines[i];
    CK(cudaEventRecord(g->pre[2 * i], e->stream));
    CK(cudaEventRecord(g->pre[2 * i + 1], e->bath_stream));
    CK(cudaStreamWaitEvent(g->stream, g->pre[2 * i], 0));
    CK(cudaStreamWaitEvent(g->stream, g->pre[2 * i + 1], 0));
  }
  CK(cudaGraphLaunch(g->exec, g->stream));
  CK(cudaEventRecord(g->done, g->stream));
  for (uint32_t i = 0; i < n; i++) {   // later work on the engines' streams follows the graph
    dpsnn_engine *e = g->engines[i];
    CK(cudaStreamWaitEvent(e->stream, g->done, 0));
    CK(cudaStreamWaitEvent(e->bath_stream, g->done, 0));
    rearm_step_events(e);
    e->t_host += g->nsteps;
  }
  g->engines[0]->launches += g->launches_per_run;   // counted on the first engine
  return 0;
}

extern "C" int dpsnn_set_launch_shape(dpsnn_engine *e, uint32_t deliver_blocks, uint32_t heavy_sort_blocks,
                                      uint32_t heavy_run_blocks) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  const uint32_t lim = 1u << 20;
  if (deliver_blocks > lim || heavy_sort_blocks > lim || heavy_run_blocks > lim)
    return dpsnn_fail(DPSNN_E_PARAM, "a grid of more than %u blocks", lim);
  default_grids(e, deliver_blocks, heavy_sort_blocks, heavy_run_blocks);
  return 0;
}

extern "C" int dpsnn_sync(dpsnn_engine *e) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  cudaSetDevice(e->device);
  CK(cudaStreamSynchronize(e->stream));
  return check_flags(e);
}

extern "C" uint32_t dpsnn_glob_n(const dpsnn_engine *e) { return e ? e->hnet.N : 0; }
extern "C" uint32_t dpsnn_time_ms(const dpsnn_engine *e) { return e ? e->t_host : 0; }
extern "C" uint64_t dpsnn_synapse_count(const dpsnn_engine *e) { return e ? e->S : 0; }
extern "C" uint64_t dpsnn_events_delivered(const dpsnn_engine *e) {
  if (!e) return 0;
  unsigned long long v = 0;
  cudaSetDevice(e->device);
  cudaMemcpyAsync(&v, e->d.events, 8, cudaMemcpyDeviceToHost, e->stream);
  cudaStreamSynchronize(e->stream);
  return v;
}

// The lists of steps t0 .. t0+n-1 (1 <= n <= RING_SLOTS) after the compaction
// of the last of them (steps complete in order on the engine stream; the rest
// of that step and later ones may still run): the error flags, the counts, and
// whether the lists fitted, in the read buffer, which the caller holds (read_mu).
static int read_lists(dpsnn_engine *e, uint32_t t0, uint32_t n, bool &packed) {
  CK(cudaStreamWaitEvent(e->read_stream, e->ev_slot[(t0 + n - 1) % RING_SLOTS], 0));
  read_pack_kernel<<<n == 1 ? 2 : 16, READ_PACK_THREADS, 0, e->read_stream>>>(e->d, t0, n, e->h_read_cap, e->h_read);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(e->read_stream));
  packed = e->h_read->total <= e->h_read_cap;
  return 0;
}
static const uint32_t *read_ids(const dpsnn_engine *e) {
  return reinterpret_cast<const uint32_t *>(spike_read_te(e->h_read) + e->h_read_cap);
}

extern "C" int dpsnn_spikes(dpsnn_engine *e, uint32_t t_ms, uint32_t *ids, double *te, uint32_t cap,
                            uint32_t *count) {
  if (!e || !count) return dpsnn_fail(DPSNN_E_PARAM, "null argument");
  if (t_ms >= e->t_host || t_ms + RING_SLOTS < e->t_host)
    return dpsnn_fail(DPSNN_E_STATE, "step %u is not among the last %d completed steps", t_ms, RING_SLOTS);
  cudaSetDevice(e->device);
  std::lock_guard<std::mutex> lock(e->read_mu);
  bool packed;
  int rc = read_lists(e, t_ms, 1, packed);
  if (!rc) rc = flags_error(e->h_read->flags);
  if (rc) return rc;
  const uint32_t cnt = e->h_read->total, k = std::min(cnt, cap);
  *count = cnt;
  if (packed) {
    if (ids) memcpy(ids, read_ids(e), 4ull * k);
    if (te) memcpy(te, spike_read_te(e->h_read), 8ull * k);
    return 0;
  }
  const size_t at = (size_t)(t_ms % RING_SLOTS) * e->hnet.N;
  if (k && ids) CK(cudaMemcpyAsync(ids, e->d.ring_ids + at, 4ull * k, cudaMemcpyDeviceToHost, e->read_stream));
  if (k && te) CK(cudaMemcpyAsync(te, e->d.ring_te + at, 8ull * k, cudaMemcpyDeviceToHost, e->read_stream));
  if (k && (ids || te)) CK(cudaStreamSynchronize(e->read_stream));
  return 0;
}

extern "C" int dpsnn_spikes_range(dpsnn_engine *e, uint32_t t0, uint32_t n, uint32_t *ids, double *te,
                                  uint64_t cap, uint32_t *counts) {
  if (!e || !counts || (n && (!ids || !te))) return dpsnn_fail(DPSNN_E_PARAM, "null argument");
  if (n == 0) return 0;
  if (n > RING_SLOTS || t0 + n > e->t_host || t0 + RING_SLOTS < e->t_host)
    return dpsnn_fail(DPSNN_E_STATE, "steps %u..%u are not among the last %d completed steps", t0, t0 + n - 1,
                      RING_SLOTS);
  cudaSetDevice(e->device);
  std::lock_guard<std::mutex> lock(e->read_mu);
  bool packed;
  int rc = read_lists(e, t0, n, packed);
  if (rc) return rc;
  memcpy(counts, e->h_read->counts, 4ull * n);
  rc = flags_error(e->h_read->flags);
  if (rc) return rc;
  uint64_t off = e->h_read->total;
  if (off > cap) return dpsnn_fail(DPSNN_E_CAPACITY, "%llu spikes in steps %u..%u exceed the buffers (%llu)",
                                   (unsigned long long)off, t0, t0 + n - 1, (unsigned long long)cap);
  if (packed) {
    memcpy(ids, read_ids(e), 4ull * off);
    memcpy(te, spike_read_te(e->h_read), 8ull * off);
    return 0;
  }
  off = 0;
  for (uint32_t k = 0; k < n; k++) {
    const size_t slot = (t0 + k) % RING_SLOTS;
    if (counts[k]) {
      CK(cudaMemcpyAsync(ids + off, e->d.ring_ids + slot * e->hnet.N, 4ull * counts[k], cudaMemcpyDeviceToHost,
                         e->read_stream));
      CK(cudaMemcpyAsync(te + off, e->d.ring_te + slot * e->hnet.N, 8ull * counts[k], cudaMemcpyDeviceToHost,
                         e->read_stream));
    }
    off += counts[k];
  }
  CK(cudaStreamSynchronize(e->read_stream));
  return 0;
}

extern "C" uint64_t dpsnn_device_bytes(const dpsnn_engine *e) { return e ? e->bytes : 0; }

extern "C" int dpsnn_state(dpsnn_engine *e, double *v, double *c, double *tr, double *te, double *nb) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  int rc = dpsnn_sync(e);
  if (rc) return rc;
  size_t B = 8ull * e->hnet.N;
  if (v) CK(cudaMemcpy(v, e->d.v, B, cudaMemcpyDeviceToHost));
  if (c) CK(cudaMemcpy(c, e->d.c, B, cudaMemcpyDeviceToHost));
  if (tr) CK(cudaMemcpy(tr, e->d.tr, B, cudaMemcpyDeviceToHost));
  if (te) CK(cudaMemcpy(te, e->d.te, B, cudaMemcpyDeviceToHost));
  // nextBath after the last completed step (the bath of the next step may
  // already have run into the other buffer)
  if (nb) CK(cudaMemcpy(nb, e->nb2[e->t_host ? (e->t_host - 1) & 1 : 1], B, cudaMemcpyDeviceToHost));
  return 0;
}

extern "C" int dpsnn_bath_params(dpsnn_engine *e, double *inv_nu_ext, uint32_t *max_ext) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  int rc = dpsnn_sync(e);
  if (rc) return rc;
  if (inv_nu_ext) CK(cudaMemcpy(inv_nu_ext, e->d.inv_nu, 8ull * e->hnet.N, cudaMemcpyDeviceToHost));
  if (max_ext) CK(cudaMemcpy(max_ext, e->d.max_ext, 4ull * e->hnet.N, cudaMemcpyDeviceToHost));
  return 0;
}

// Host-side view of the connectome.
struct HostCsr {
  std::vector<uint64_t> row;
  std::vector<uint16_t> so;
  std::vector<uint32_t> post;
  std::vector<int16_t> w;
};
static int fetch_csr(dpsnn_engine *e, HostCsr &h) {
  int rc = dpsnn_sync(e);
  if (rc) return rc;
  const uint32_t N = e->hnet.N, D = e->hnet.D;
  h.row.resize(N + 1);
  h.so.resize((size_t)N * (D + 1));
  h.post.resize(e->S);
  h.w.resize(e->S);
  CK(cudaMemcpy(h.row.data(), e->d.row_ptr, 8ull * (N + 1), cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(h.so.data(), e->d.sub_off, 2ull * N * (D + 1), cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(h.post.data(), e->d.post, 4ull * e->S, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(h.w.data(), e->d.w16, 2ull * e->S, cudaMemcpyDeviceToHost));
  return 0;
}

// ------------------------------------------------------------------ a rank's synapse list
// The reference's order (inflateIntermToBackwardSynList): delay, then
// presynaptic neuron, then generation order, of the synapses aimed at one
// rank.  On the device: the list's segments, one per (delay, presynaptic
// neuron), are counted, summed and written in place, and only the rank's list
// crosses to the host.  (The host walked a copy of the whole connectome, twice
// with the count: 6 ms of a small network's dump, seconds of a large one's.)
#define LIST_SCAN_THREADS 256
#define LIST_SCAN_ITEMS 8
#define LIST_SCAN_TILE (LIST_SCAN_THREADS * LIST_SCAN_ITEMS)
// seg[dl * N + P]: synapses of the segment (P, dl) in the rank's neurons
// [lo, hi), a warp per presynaptic neuron.
__global__ void list_count_kernel(Dev d, uint32_t lo, uint32_t hi, uint32_t *__restrict__ seg) {
  const uint32_t N = d.net->N, D = d.net->D, lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t P = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; P < N; P += nw) {
    const uint64_t row = d.row_ptr[P];
    const uint16_t *so = d.sub_off + (size_t)P * (D + 1);
    for (uint32_t dl = 0; dl < D; dl++) {
      const uint32_t b = so[dl], e = so[dl + 1];
      uint32_t c = 0;
      for (uint32_t k = b + lane; k < e; k += 32) {
        const uint32_t j = d.post[row + k];
        c += j >= lo && j < hi;
      }
      c = __reduce_add_sync(0xffffffffu, c);
      if (lane == 0) seg[(size_t)dl * N + P] = c;
    }
  }
}
// Sums of tiles of LIST_SCAN_TILE segments, then each tile's base.
__global__ void __launch_bounds__(LIST_SCAN_THREADS) list_sum_kernel(const uint32_t *__restrict__ seg, uint64_t n,
                                                                     uint64_t *__restrict__ tile) {
  __shared__ uint64_t s[LIST_SCAN_THREADS / 32];
  uint64_t c = 0;
  for (uint32_t k = threadIdx.x; k < LIST_SCAN_TILE; k += LIST_SCAN_THREADS) {
    const uint64_t i = (uint64_t)blockIdx.x * LIST_SCAN_TILE + k;
    if (i < n) c += seg[i];
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < LIST_SCAN_THREADS / 32; w++) c += s[w];
    tile[blockIdx.x] = c;
  }
}
__global__ void list_base_kernel(uint64_t *tile, uint32_t n) {   // one warp: exclusive sums; the total at tile[n]
  uint64_t acc = 0;
  for (uint32_t i0 = 0; i0 < n; i0 += 32) {
    const uint32_t i = i0 + threadIdx.x;
    const uint64_t c = i < n ? tile[i] : 0;
    uint64_t incl = c;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (threadIdx.x >= (uint32_t)o) incl += y;
    }
    if (i < n) tile[i] = acc + incl - c;
    acc += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (threadIdx.x == 0) tile[n] = acc;
}
// at[i]: first place of segment i.
__global__ void __launch_bounds__(LIST_SCAN_THREADS) list_place_kernel(const uint32_t *__restrict__ seg, uint64_t n,
                                                                       const uint64_t *__restrict__ tile,
                                                                       uint64_t *__restrict__ at) {
  __shared__ uint32_t s[LIST_SCAN_THREADS / 32];
  const uint64_t i0 = (uint64_t)blockIdx.x * LIST_SCAN_TILE + threadIdx.x * LIST_SCAN_ITEMS;
  uint32_t c[LIST_SCAN_ITEMS], sum = 0;
  for (int k = 0; k < LIST_SCAN_ITEMS; k++) {
    c[k] = i0 + k < n ? seg[i0 + k] : 0u;
    sum += c[k];   // a tile holds below 2^32 synapses (2048 segments of at most 7500)
  }
  uint32_t incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if ((threadIdx.x & 31) >= (uint32_t)o) incl += y;
  }
  if ((threadIdx.x & 31) == 31) s[threadIdx.x >> 5] = incl;
  __syncthreads();
  uint64_t acc = tile[blockIdx.x] + incl - sum;
  for (uint32_t w = 0; w < (threadIdx.x >> 5); w++) acc += s[w];
  for (int k = 0; k < LIST_SCAN_ITEMS; k++)
    if (i0 + k < n) {
      at[i0 + k] = acc;
      acc += c[k];
    }
}
struct SynapseList {   // device arrays of one rank's list; null: not wanted
  uint32_t *pre, *post;
  uint8_t *delay, *kind;
  int16_t *weight;
  float *tderiv;
};
__global__ void list_fill_kernel(Dev d, uint32_t lo, uint32_t hi, const uint64_t *__restrict__ at, SynapseList l) {
  const uint32_t N = d.net->N, D = d.net->D, lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t P = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; P < N; P += nw) {
    const uint64_t row = d.row_ptr[P];
    const uint16_t *so = d.sub_off + (size_t)P * (D + 1);
    const uint8_t kind = d.sub[P];
    for (uint32_t dl = 0; dl < D; dl++) {
      const uint32_t b = so[dl], e = so[dl + 1];
      uint64_t o0 = at[(size_t)dl * N + P];
      for (uint32_t k0 = b; k0 < e; k0 += 32) {
        const uint32_t k = k0 + lane, j = k < e ? d.post[row + k] : 0xFFFFFFFFu;
        const bool in = k < e && j >= lo && j < hi;
        const uint32_t bal = __ballot_sync(0xffffffffu, in);
        if (in) {
          const uint64_t o = o0 + __popc(bal & ((1u << lane) - 1));
          if (l.pre) l.pre[o] = P;
          if (l.post) l.post[o] = j;
          if (l.delay) l.delay[o] = (uint8_t)dl;
          if (l.kind) l.kind[o] = kind;
          if (l.weight) l.weight[o] = d.w16[row + k];
          if (l.tderiv) l.tderiv[o] = d.tderiv ? d.tderiv[row + k] : 0.0f;
        }
        o0 += __popc(bal);
      }
    }
  }
}

// Stream-ordered scratch of one call.
struct CallScratch {
  dpsnn_engine *e;
  std::vector<void *> held;
  explicit CallScratch(dpsnn_engine *eng) : e(eng) {}
  ~CallScratch() {
    for (void *q : held) cudaFreeAsync(q, e->stream);
  }
  template <typename T>
  int get(T **p, size_t n) {
    void *q = nullptr;
    const cudaError_t err = cudaMallocAsync(&q, std::max<size_t>(n * sizeof(T), 16), e->stream);
    if (err != cudaSuccess) return dpsnn_fail(DPSNN_E_NOMEM, "cudaMallocAsync: %s", cudaGetErrorString(err));
    held.push_back(q);
    *p = (T *)q;
    return 0;
  }
};

// Rank h's list: its length, and with `out` its arrays (host; null: not
// wanted).  DPSNN_E_NOMEM where the device has no room for the scratch (12
// bytes per neuron and delay, and the list).
static int rank_list_device(dpsnn_engine *e, uint32_t h, uint64_t *count, const SynapseList *out) {
  int rc = 0;
  const uint32_t N = e->hnet.N, D = e->hnet.D, lo = h * e->hnet.locN, hi = lo + e->hnet.locN;
  const uint64_t nseg = (uint64_t)N * D;
  const uint32_t tiles = (uint32_t)((nseg + LIST_SCAN_TILE - 1) / LIST_SCAN_TILE);
  const uint32_t grid = std::min<uint32_t>((uint32_t)e->sms * 8, (N + 7) / 8);
  CallScratch m(e);
  uint32_t *seg;
  uint64_t *tile, *at, n = 0;
  if ((rc = m.get(&seg, nseg)) || (rc = m.get(&tile, tiles + 1))) return rc;
  list_count_kernel<<<grid, 256, 0, e->stream>>>(e->d, lo, hi, seg);
  list_sum_kernel<<<tiles, LIST_SCAN_THREADS, 0, e->stream>>>(seg, nseg, tile);
  list_base_kernel<<<1, 32, 0, e->stream>>>(tile, tiles);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(&n, tile + tiles, 8, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  if (count) *count = n;
  if (!out || !n) return 0;
  SynapseList l = {};
  if ((rc = m.get(&at, nseg))) return rc;
  if (out->pre && (rc = m.get(&l.pre, n))) return rc;
  if (out->post && (rc = m.get(&l.post, n))) return rc;
  if (out->delay && (rc = m.get(&l.delay, n))) return rc;
  if (out->kind && (rc = m.get(&l.kind, n))) return rc;
  if (out->weight && (rc = m.get(&l.weight, n))) return rc;
  if (out->tderiv && (rc = m.get(&l.tderiv, n))) return rc;
  list_place_kernel<<<tiles, LIST_SCAN_THREADS, 0, e->stream>>>(seg, nseg, tile, at);
  list_fill_kernel<<<grid, 256, 0, e->stream>>>(e->d, lo, hi, at, l);
  CK(cudaGetLastError());
  if (out->pre) CK(cudaMemcpyAsync(out->pre, l.pre, 4 * n, cudaMemcpyDeviceToHost, e->stream));
  if (out->post) CK(cudaMemcpyAsync(out->post, l.post, 4 * n, cudaMemcpyDeviceToHost, e->stream));
  if (out->delay) CK(cudaMemcpyAsync(out->delay, l.delay, n, cudaMemcpyDeviceToHost, e->stream));
  if (out->kind) CK(cudaMemcpyAsync(out->kind, l.kind, n, cudaMemcpyDeviceToHost, e->stream));
  if (out->weight) CK(cudaMemcpyAsync(out->weight, l.weight, 2 * n, cudaMemcpyDeviceToHost, e->stream));
  if (out->tderiv) CK(cudaMemcpyAsync(out->tderiv, l.tderiv, 4 * n, cudaMemcpyDeviceToHost, e->stream));
  CK(cudaStreamSynchronize(e->stream));
  return 0;
}

// The same on the host, from a copy of the connectome.
static int rank_list_host(dpsnn_engine *e, uint32_t h, uint64_t *count, const SynapseList *out) {
  HostCsr c;
  int rc = fetch_csr(e, c);
  if (rc) return rc;
  const uint32_t N = e->hnet.N, D = e->hnet.D, locN = e->hnet.locN;
  std::vector<float> td;
  std::vector<uint8_t> sub(N);
  CK(cudaMemcpy(sub.data(), e->d.sub, N, cudaMemcpyDeviceToHost));
  if (out && out->tderiv && e->d.tderiv) {
    td.resize(e->S);
    CK(cudaMemcpy(td.data(), e->d.tderiv, 4ull * e->S, cudaMemcpyDeviceToHost));
  }
  uint64_t o = 0;
  for (uint32_t dl = 0; dl < D; dl++)
    for (uint32_t P = 0; P < N; P++) {
      const uint64_t b = c.row[P] + c.so[(size_t)P * (D + 1) + dl], en = c.row[P] + c.so[(size_t)P * (D + 1) + dl + 1];
      for (uint64_t k = b; k < en; k++) {
        if (c.post[k] / locN != h) continue;
        if (out && out->pre) out->pre[o] = P;
        if (out && out->post) out->post[o] = c.post[k];
        if (out && out->delay) out->delay[o] = (uint8_t)dl;
        if (out && out->kind) out->kind[o] = sub[P];
        if (out && out->weight) out->weight[o] = c.w[k];
        if (out && out->tderiv) out->tderiv[o] = td.empty() ? 0.0f : td[k];
        o++;
      }
    }
  if (count) *count = o;
  return 0;
}
static int rank_list(dpsnn_engine *e, uint32_t h, uint64_t *count, const SynapseList *out) {
  int rc = dpsnn_sync(e);
  if (!rc) rc = rank_list_device(e, h, count, out);
  if (rc != DPSNN_E_NOMEM) return rc;
  cudaGetLastError();
  return rank_list_host(e, h, count, out);
}

extern "C" uint64_t dpsnn_rank_synapse_count(dpsnn_engine *e, uint32_t h) {
  if (!e || h >= e->hnet.P) return 0;
  if (e->hnet.P == 1) return dpsnn_sync(e) ? 0 : e->S;
  uint64_t n = 0;
  return rank_list(e, h, &n, nullptr) ? 0 : n;
}

extern "C" int dpsnn_backward_synapses(dpsnn_engine *e, uint32_t h, uint32_t *pre, uint32_t *post, uint8_t *delay,
                                       uint8_t *kind, int16_t *weight, float *tderiv) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  if (h >= e->hnet.P) return dpsnn_fail(DPSNN_E_PARAM, "rank %u out of range", h);
  const SynapseList out = {pre, post, delay, kind, weight, tderiv};
  return rank_list(e, h, nullptr, &out);
}

extern "C" int dpsnn_enable_ltp_probe(dpsnn_engine *e) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  if (!e->hnet.stdp_on) return dpsnn_fail(DPSNN_E_PARAM, "the LTP probe needs plasticity switched on");
  if (e->d.probe_w) return 0;
  if (e->t_host) return dpsnn_fail(DPSNN_E_PARAM, "the LTP probe is enabled before the first step");
  cudaSetDevice(e->device);
  DALLOC(e->d.probe_w, e->S);
  DALLOC(e->d.probe_td, e->S);
  DALLOC(e->d.probe_td_mid, e->S);
  return 0;
}

extern "C" int dpsnn_ltp_probe(dpsnn_engine *e, uint32_t h, uint32_t *t_ms, int16_t *w_before, float *td_before,
                               int16_t *w_after, float *td_after) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  if (h >= e->hnet.P) return dpsnn_fail(DPSNN_E_PARAM, "rank %u out of range", h);
  if (!e->d.probe_w) return dpsnn_fail(DPSNN_E_PARAM, "the LTP probe is not enabled");
  if (e->probe_t == UINT32_MAX) return dpsnn_fail(DPSNN_E_PARAM, "no plasticity update has run yet");
  HostCsr c;
  int rc = fetch_csr(e, c);   // synchronises: the probe and the weights are final
  if (rc) return rc;
  std::vector<int16_t> pw(e->S);
  std::vector<float> pt(e->S), pm(e->S);
  CK(cudaMemcpy(pw.data(), e->d.probe_w, 2ull * e->S, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(pt.data(), e->d.probe_td, 4ull * e->S, cudaMemcpyDeviceToHost));
  CK(cudaMemcpy(pm.data(), e->d.probe_td_mid, 4ull * e->S, cudaMemcpyDeviceToHost));
  if (t_ms) *t_ms = e->probe_t;
  // the order of dpsnn_backward_synapses; the weights change only at an LTP
  // update, so the live weights are those the last update wrote
  const uint32_t N = e->hnet.N, D = e->hnet.D, locN = e->hnet.locN;
  uint64_t o = 0;
  for (uint32_t dl = 0; dl < D; dl++)
    for (uint32_t P = 0; P < N; P++) {
      uint64_t b = c.row[P] + c.so[(size_t)P * (D + 1) + dl], en = c.row[P] + c.so[(size_t)P * (D + 1) + dl + 1];
      for (uint64_t k = b; k < en; k++) {
        if (c.post[k] / locN != h) continue;
        if (w_before) w_before[o] = pw[k];
        if (td_before) td_before[o] = pt[k];
        if (w_after) w_after[o] = c.w[k];
        if (td_after) td_after[o] = pm[k];
        o++;
      }
    }
  return 0;
}

extern "C" int dpsnn_enable_stdp_events(dpsnn_engine *e) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  if (!e->hnet.stdp_on) return dpsnn_fail(DPSNN_E_PARAM, "the STDP event log needs plasticity switched on");
  if (e->d.stdp_log) return 0;
  if (e->t_host) return dpsnn_fail(DPSNN_E_PARAM, "the STDP event log is enabled before the first step");
  cudaSetDevice(e->device);
  HostCsr c;
  int rc = fetch_csr(e, c);
  if (rc) return rc;
  e->h_row = std::move(c.row);
  e->h_so = std::move(c.so);
  DALLOC(e->d.stdp_log, STDP_LOG_CAP);
  DALLOC(e->d.stdp_log_cnt, 1);
  return 0;
}

extern "C" int dpsnn_stdp_events(dpsnn_engine *e, uint32_t *t_ms, uint32_t *pre, uint32_t *post, float *contribution,
                                 uint32_t cap, uint32_t *count) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  if (!e->d.stdp_log) return dpsnn_fail(DPSNN_E_PARAM, "the STDP event log is not enabled");
  if (e->stdp_log_t == UINT32_MAX) return dpsnn_fail(DPSNN_E_PARAM, "no step has run yet");
  int rc = dpsnn_sync(e);   // also reports a full log (DPSNN_E_CAPACITY)
  if (rc) return rc;
  uint32_t n = 0;
  CK(cudaMemcpy(&n, e->d.stdp_log_cnt, 4, cudaMemcpyDeviceToHost));
  if (n > STDP_LOG_CAP) return dpsnn_fail(DPSNN_E_CAPACITY, "more than %u STDP events in one step", STDP_LOG_CAP);
  std::vector<uint4> rec(n);
  if (n) CK(cudaMemcpy(rec.data(), e->d.stdp_log, 16ull * n, cudaMemcpyDeviceToHost));
  // presynaptic neuron and delay of each record's synapse from the CSR, then
  // the reference's order: causal events (detection, ascending post, each
  // post's synapses in backward-list order: delay, then presynaptic neuron,
  // then generation order), then anti-causal events (delivery: delay
  // descending, then presynaptic neuron, then generation order)
  const uint32_t D = e->hnet.D;
  struct Ev {
    uint64_t key0, key1;
    uint32_t pre, post;
    float c;
  };
  std::vector<Ev> ev(n);
  for (uint32_t i = 0; i < n; i++) {
    const uint64_t k = (uint64_t)rec[i].x | ((uint64_t)rec[i].y << 32);
    const uint32_t P = (uint32_t)(std::upper_bound(e->h_row.begin(), e->h_row.end(), k) - e->h_row.begin()) - 1;
    uint32_t dl = 0;
    while (dl + 1 < D && e->h_row[P] + e->h_so[(size_t)P * (D + 1) + dl + 1] <= k) dl++;
    const uint32_t j = rec[i].z & 0x7fffffffu, anti = rec[i].z >> 31;
    Ev &v = ev[i];
    v.pre = P;
    v.post = j;
    memcpy(&v.c, &rec[i].w, 4);
    if (anti) {
      v.key0 = (1ull << 63) | (uint64_t)(D - 1 - dl);
    } else {
      v.key0 = ((uint64_t)j << 8) | dl;
    }
    v.key1 = k;
  }
  std::sort(ev.begin(), ev.end(), [](const Ev &a, const Ev &b) {
    return a.key0 != b.key0 ? a.key0 < b.key0 : a.key1 < b.key1;
  });
  if (t_ms) *t_ms = e->stdp_log_t;
  if (count) *count = n;
  const uint32_t m = std::min(n, cap);
  for (uint32_t i = 0; i < m; i++) {
    if (pre) pre[i] = ev[i].pre;
    if (post) post[i] = ev[i].post;
    if (contribution) contribution[i] = ev[i].c;
  }
  return 0;
}

extern "C" int dpsnn_set_timing(dpsnn_engine *e, int enable) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  e->timing = enable;
  return 0;
}

extern "C" uint64_t dpsnn_kernel_launches(const dpsnn_engine *e) { return e ? e->launches : 0; }
extern "C" void *dpsnn_cuda_stream(const dpsnn_engine *e) { return e ? (void *)e->stream : nullptr; }

extern "C" int dpsnn_kernel_times(dpsnn_engine *e, double *seconds, uint64_t *launches) {
  if (!e) return dpsnn_fail(DPSNN_E_PARAM, "null engine");
  cudaSetDevice(e->device);
  collect_timings(e);
  for (int k = 0; k < DPSNN_TIMING_SLOTS; k++) {
    if (seconds) seconds[k] = e->ktime[k];
    if (launches) launches[k] = e->klaunch[k];
  }
  return 0;
}

// ------------------------------------------------------------------ no-allocation rank spike read
// dpsnn_rank_spikes_noalloc: the spike list of one emulated rank at one step,
// gathered on the device into a fixed scratch area that is part of the
// library image (no cudaMalloc/cudaFree on this path), then copied to the
// caller's host buffers.  The scratch holds DPSNN_NOALLOC_MAX_SPIKES spikes,
// the reference's largest rank (miniLocN = 32000 neurons) rounded up; ranks
// with more neurons are rejected.  One scratch per device and process: calls
// that overlap in time on the same device race on it.
struct NoAllocScratch {
  uint32_t count;                            // written by the kernel each call
  uint32_t pad[63];
  uint32_t ids[DPSNN_NOALLOC_MAX_SPIKES];
  double te[DPSNN_NOALLOC_MAX_SPIKES];
};
static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

// One block: binary search of the rank's neuron range [lo, hi) in the
// ascending spike list of the slot, then an ordered copy of that range.
// Nothing in the scratch has to start at zero: count and the copied entries
// are all written here before the host reads them.
__global__ void rank_select_kernel(const uint32_t *__restrict__ ids, const double *__restrict__ te,
                                   const uint32_t *__restrict__ cnt_ptr, uint32_t lo, uint32_t hi,
                                   NoAllocScratch *__restrict__ out) {
  __shared__ uint32_t s_a, s_b;
  const uint32_t cnt = *cnt_ptr;
  if (threadIdx.x == 0) {
    uint32_t a = 0, b = cnt;
    while (a < b) {
      const uint32_t m = (a + b) >> 1;
      if (ids[m] < lo) a = m + 1; else b = m;
    }
    uint32_t c = a, d = cnt;
    while (c < d) {
      const uint32_t m = (c + d) >> 1;
      if (ids[m] < hi) c = m + 1; else d = m;
    }
    s_a = a;
    s_b = c;
    out->count = c - a;
  }
  __syncthreads();
  const uint32_t a = s_a, n = min(s_b - s_a, (uint32_t)DPSNN_NOALLOC_MAX_SPIKES);
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
    out->ids[k] = ids[a + k];
    out->te[k] = te[a + k];
  }
}

#define DPSNN_NOALLOC_MAX_DEVICES 64
static std::mutex g_noalloc_mu;
static NoAllocScratch *g_noalloc_addr[DPSNN_NOALLOC_MAX_DEVICES];

// Device address of the scratch, looked up once per device.
static int noalloc_scratch(int device, NoAllocScratch **out) {
  if (device < 0 || device >= DPSNN_NOALLOC_MAX_DEVICES)
    return dpsnn_fail(DPSNN_E_PARAM, "device %d out of range", device);
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  if (!g_noalloc_addr[device]) {
    void *p = nullptr;
    cudaError_t err = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (err != cudaSuccess)
      return dpsnn_fail(DPSNN_E_CUDA, "cudaGetSymbolAddress(scratch): %s", cudaGetErrorString(err));
    g_noalloc_addr[device] = (NoAllocScratch *)p;
  }
  *out = g_noalloc_addr[device];
  return 0;
}

extern "C" int dpsnn_rank_spikes_noalloc(dpsnn_engine *e, uint32_t t_ms, uint32_t h, uint32_t *ids, double *te,
                                         uint32_t cap, uint32_t *count) {
  if (!e || !count) return dpsnn_fail(DPSNN_E_PARAM, "null argument");
  if (h >= e->hnet.P) return dpsnn_fail(DPSNN_E_PARAM, "rank %u out of range (env_globH = %u)", h, e->hnet.P);
  if (e->hnet.locN > DPSNN_NOALLOC_MAX_SPIKES)
    return dpsnn_fail(DPSNN_E_CAPACITY, "rank of %u neurons exceeds the %d-spike scratch of dpsnn_rank_spikes_noalloc",
                      e->hnet.locN, DPSNN_NOALLOC_MAX_SPIKES);
  if (t_ms >= e->t_host || t_ms + RING_SLOTS < e->t_host)
    return dpsnn_fail(DPSNN_E_STATE, "step %u is not among the last %d completed steps", t_ms, RING_SLOTS);
  cudaSetDevice(e->device);
  NoAllocScratch *s = nullptr;
  int rc = noalloc_scratch(e->device, &s);
  if (rc) return rc;
  const uint32_t slot = t_ms % RING_SLOTS;
  const size_t off = (size_t)slot * e->hnet.N;
  // on the read stream, after the compaction of step t_ms only (as
  // dpsnn_spikes): later steps keep running on the engine stream
  CK(cudaStreamWaitEvent(e->read_stream, e->ev_slot[slot], 0));
  rank_select_kernel<<<1, 256, 0, e->read_stream>>>(e->d.ring_ids + off, e->d.ring_te + off, e->d.ring_cnt + slot,
                                                    h * e->hnet.locN, (h + 1) * e->hnet.locN, s);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(e->h_pin, e->d.flags, 4, cudaMemcpyDeviceToHost, e->read_stream));
  CK(cudaMemcpyAsync(e->h_pin + 1, &s->count, 4, cudaMemcpyDeviceToHost, e->read_stream));
  CK(cudaStreamSynchronize(e->read_stream));
  rc = flags_error(e->h_pin[0]);
  if (rc) return rc;
  const uint32_t n = e->h_pin[1];
  *count = n;
  const uint32_t k = std::min(n, cap);
  if (k && ids) CK(cudaMemcpyAsync(ids, s->ids, 4ull * k, cudaMemcpyDeviceToHost, e->read_stream));
  if (k && te) CK(cudaMemcpyAsync(te, s->te, 8ull * k, cudaMemcpyDeviceToHost, e->read_stream));
  if (k && (ids || te)) CK(cudaStreamSynchronize(e->read_stream));
  return 0;
}
