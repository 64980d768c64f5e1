// pps_resident.cu -- which synchronous runs keep their swarm in shared memory
// for the whole run (pps_resident.cuh), and how they are launched.
//
// Measured on a GB300, us an iteration, one launch per iteration -> resident:
// Rosenbrock 1000 x 3 7.2 -> 1.5, Rastrigin 10000 x 10 9.4 -> 2.0, Ackley
// 20011 x 30 16.2 -> 3.9, Rosenbrock 65536 x 10 9.4 -> 3.6, sphere 100003 x 20
// 18.2 -> 5.5, Rastrigin 10000 x 100 36.1 -> 4.9, 250000 x 10 19.6 -> 9.0,
// 20011 x 128 45.5 -> 14.9 (the pair arithmetic of pps_pair.cuh took large ones
// from 5.9, 9.6 and 16.4; the small ones wait for the exchange, 2100 cycles of
// 3700 at 1000 x 3, 3300 of 9100 at 20011 x 30).  The
// line is the shared memory of all SMs (about 2.8 M coordinates of 12 bytes,
// 2.1 M with the moved terms): beyond it the state has to stream from L2 or
// memory each iteration, which k_sync_step does.
#include <cstdlib>

#include "pps_internal.h"
#include "pps_resident.cuh"

namespace pps {

template <int OBJ, bool SPLIT, bool CONS, int T = kResidentThreads>
__global__ void __launch_bounds__(T, 1)
    k_resident(SwarmDev s, ObjParams op, PhiloxKeys keys, ResidentArgs a) {
  resident_run<OBJ, SPLIT, CONS>(s, op, keys, a, (int)blockIdx.x);
}

constexpr size_t kResidentSmem = 227u << 10;  // a block's shared memory, static part included
constexpr size_t kResidentStatic = 2048;
constexpr int kResidentMaxDim = 1024;  // g and bounds of more dims crowd the state out
constexpr int64_t kResidentOneBlock = 1536;  // coordinates one block takes alone
constexpr int64_t kResidentCoords = 256;     // coordinates a block of several has at least
constexpr int kResidentMinBlocks = 16;

static bool terms_moved(int objective) { return objective == kRastrigin || objective == kAckley; }

unsigned int wait_polls(unsigned int usual) {
  const char* e = getenv("PPS_WAIT_POLLS");
  if (!e || *e < '0' || *e > '9') return usual;
  const unsigned long n = strtoul(e, nullptr, 10);
  return n < usual ? (unsigned int)n : usual;
}

// bytes of the exchange words the swarm's run needs (0: none)
size_t resident_exchange_bytes(int objective, int dim, int64_t n, int ncons, int sm_count) {
  ResidentPlan p;
  if (!resident_plan(objective, dim, n, ncons, sm_count, &p) || p.blocks == 1) return 0;
  return sizeof(unsigned long long) * 2 * resident_words(p.blocks, dim);
}

bool resident_fit(int objective, int dim, int64_t n, bool cons, int blocks, int most, size_t smem, ResidentPlan* p) {
  const int64_t chunk = (n + blocks - 1) / blocks;
  const int np = (dim + 1) / 2;
  if (chunk > (1 << 20)) return false;
  int groups = (int)(most / chunk);
  if (groups > np) groups = np;
  if (groups > 1) groups = (np + (np + groups - 1) / groups - 1) / ((np + groups - 1) / groups);  // even shares
  bool split = cons || groups > 1;
  if (!cons && split && resident_smem(dim, (int)chunk, terms_moved(objective)) > smem) {
    split = false;  // no room for the terms: one thread walks all dims
  }
  split = split || is_user(objective);
  if (groups < 1 || !split) groups = 1;
  p->split = split;
  p->groups = groups;
  p->chunk = (int)chunk;
  p->blocks = (int)((n + chunk - 1) / chunk);
  const int64_t want = groups > 1 ? chunk * groups : chunk;
  const int64_t rounds = (want + most - 1) / most;
  p->threads = (int)(((want + rounds - 1) / rounds + 31) / 32 * 32);
  p->smem = resident_smem(dim, (int)chunk, split && terms_moved(objective));
  if (p->smem > smem) return false;
  return true;
}

bool resident_plan(int objective, int dim, int64_t n, int ncons, int sm_count, ResidentPlan* p) {
  switch (objective) {
    case kSphere: case kRosenbrock: case kRastrigin: case kAckley: case kShiftedSphere: case kBeale: case kBooth:
    case kHimmelblau: case kQuadratic: case kBoundaryQuadratic: break;
    default:
      if (!is_user(objective)) return false;
  }
  if (dim > kResidentMaxDim || n < 1 || sm_count < 1) return false;
  // Blocks: one while the iteration is shorter than an exchange between
  // blocks (about 1 us; Rosenbrock, us an iteration, 1 block / 19: 100 x 3
  // 0.97 / 1.91, 300 x 3 1.39 / 1.63, 1000 x 3 2.39 / 1.71), then as many as
  // keep kResidentCoords coordinates each (1000 x 3 on 19 / 38 / 76 / 152
  // blocks 1.71 / 1.78 / 1.91 / 1.98; Rastrigin 2000 x 10 2.36 / 1.89 / 1.95 /
  // 2.20; 10000 x 10 3.86 / 3.26 / 2.61 / 2.30), at most one per SM.
  const int64_t coords = n * (int64_t)((dim + 1) / 2 * 2);
  int64_t blocks = coords <= kResidentOneBlock ? 1 : coords / kResidentCoords;
  if (coords > kResidentOneBlock && blocks < kResidentMinBlocks) blocks = kResidentMinBlocks;
  // a user objective's own cost is unknown: spread from a warp of particles a block
  if (is_user(objective)) blocks = (n + 31) / 32;
  if (blocks > sm_count) blocks = sm_count;
  if (blocks > n) blocks = n;
  for (const int64_t b : {blocks, (int64_t)sm_count}) {
    // the constrained and the user form have the narrow kernel only
    const bool wide = !is_user(objective) && ncons == 0 && (n + b - 1) / b > kResidentThreads;
    if (resident_fit(objective, dim, n, ncons > 0, (int)b, wide ? kResidentMaxThreads : kResidentThreads,
                     kResidentSmem - kResidentStatic, p))
      return true;
  }
  return false;
}

static int launch_one(const void* kernel, pps_swarm* s, const ResidentPlan& p, PhiloxKeys keys, ResidentArgs a,
                      bool* taken) {
  if (p.smem + kResidentStatic > (48u << 10))
    PPS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kResidentSmem - kResidentStatic)));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)p.blocks);
  cfg.blockDim = dim3((unsigned)p.threads);
  cfg.dynamicSmemBytes = p.smem;
  cfg.stream = s->stream;
  cudaLaunchAttribute at[1];
  cfg.attrs = at;
  cfg.numAttrs = 0;
  if (p.blocks > 1) {
    at[0].id = cudaLaunchAttributeCooperative;  // all blocks resident, or the launch fails
    at[0].val.cooperative = 1;
    cfg.numAttrs = 1;
  }
  void* args[] = {&s->dv, &s->op, &keys, &a};
  const cudaError_t e = cudaLaunchKernelExC(&cfg, kernel, args);
  if (e == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs than the device reports: step by step instead
    cudaGetLastError();
    return PPS_OK;
  }
  if (e != cudaSuccess) return cuda_error(e, "cudaLaunchKernelExC(k_resident)");
  *taken = true;
  return PPS_OK;
}

template <int OBJ>
static int launch_obj(pps_swarm* s, const ResidentPlan& p, const PhiloxKeys& keys, const ResidentArgs& a, bool* taken) {
  if (s->dv.ncons > 0) return launch_one(reinterpret_cast<const void*>(k_resident<OBJ, true, true>), s, p, keys, a, taken);
  if constexpr (OBJ < kBeale) {
    if (p.split) return launch_one(reinterpret_cast<const void*>(k_resident<OBJ, true, false>), s, p, keys, a, taken);
  }
  if (p.threads > kResidentThreads)
    return launch_one(reinterpret_cast<const void*>(k_resident<OBJ, false, false, kResidentMaxThreads>), s, p, keys, a,
                      taken);
  return launch_one(reinterpret_cast<const void*>(k_resident<OBJ, false, false>), s, p, keys, a, taken);
}

int launch_resident(pps_swarm* s, const ResidentPlan& p, int32_t iters, float w, float wdamp, float c1, float c2,
                    int from_position, bool* taken) {
  *taken = false;
  ResidentArgs a{};
  a.chunk = p.chunk;
  a.blocks = p.blocks;
  a.groups = p.groups;
  a.iters = iters;
  a.t0 = s->t;
  a.w0 = w;
  a.wdamp = wdamp;
  a.c1s = c1 * 0x1p-24f;
  a.c2s = c2 * 0x1p-24f;
  a.from_position = from_position;
  a.seq0 = s->xch_seq;
  a.start_limit = kResidentStartLimit;
  a.poll_limit = wait_polls(kResidentPollLimit);
  a.one = 1.0f;
  a.xch = s->xch_dev;
  a.status = &s->dv.st->status;
  const PhiloxKeys keys = philox_round_keys(s->seed);
  int rc;
  if (is_user(s->objective)) {
    const void* kernel = nullptr;
    if ((rc = user_resident_kernel(s->objective, &kernel))) return rc;
    cudaFuncAttributes fa;
    PPS_CUDA(cudaFuncGetAttributes(&fa, kernel));
    if (fa.sharedSizeBytes > kResidentStatic) return PPS_OK;  // the source's own shared memory leaves no room
    a.poll_limit = wait_polls(kResidentStartLimit);
    rc = launch_one(kernel, s, p, keys, a, taken);
    if (*taken) s->xch_seq += (uint32_t)iters;
    return rc;
  }
  switch (s->objective) {
    case kSphere: rc = launch_obj<kSphere>(s, p, keys, a, taken); break;
    case kRosenbrock: rc = launch_obj<kRosenbrock>(s, p, keys, a, taken); break;
    case kRastrigin: rc = launch_obj<kRastrigin>(s, p, keys, a, taken); break;
    case kAckley: rc = launch_obj<kAckley>(s, p, keys, a, taken); break;
    case kShiftedSphere: rc = launch_obj<kShiftedSphere>(s, p, keys, a, taken); break;
    case kBeale: rc = launch_obj<kBeale>(s, p, keys, a, taken); break;
    case kBooth: rc = launch_obj<kBooth>(s, p, keys, a, taken); break;
    case kHimmelblau: rc = launch_obj<kHimmelblau>(s, p, keys, a, taken); break;
    case kQuadratic: rc = launch_obj<kQuadratic>(s, p, keys, a, taken); break;
    default: rc = launch_obj<kBoundaryQuadratic>(s, p, keys, a, taken); break;
  }
  if (*taken) s->xch_seq += (uint32_t)iters;
  return rc;
}

}  // namespace pps
