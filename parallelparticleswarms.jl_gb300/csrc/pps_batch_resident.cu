// pps_batch_resident.cu -- a batch of closed-form swarms with their state in
// shared memory, in waves that fill the GPU.
//
// k_batch (pps_batch.cu) gives each swarm a CTA or a small cluster for its
// whole life and streams the state through L2 every iteration: 256 swarms of 2-64
// dims and 256-2048 particles spend 47 us an iteration of all, waiting for L2
// behind few warps, and the largest swarm on its four CTAs sets the end.  Here
// the batch is cut into waves whose states fit the shared memory of all SMs
// together; in a wave every SM holds one block, the blocks are dealt to the
// swarms by their size, and each swarm runs all its iterations as a resident run
// of its blocks (pps_resident.cuh): the same operations, the same draws, bit for
// bit the swarm's solve alone.  A wave is a cooperative launch, so blocks that
// wait for each other are all resident.
//
// Measured on a GB300, ms a batch of 300 iterations, streaming -> resident: 16
// swarms of the mix above 8.3 -> 1.5, 32 8.1 -> 1.6, 64 8.4 -> 2.9, 128 13.0 ->
// 7.0, 256 13.8 -> 11.7, 512 26.4 -> 27 (streaming fills the GPU by then); 256
// with 100 to 2000 iterations 77 -> 49; 500 swarms of 100-600 x 2-20 3.9 -> 3.2;
// 1000 of 50-300 x 2-5 1.6 -> 2.2 (an SM runs several such swarms at once when
// streaming); 64 of 100-500 x 100-400 15.8 -> 16.8 (few particles a block, a long
// sum each).  Blocks of 512 threads with two pairs unrolled; of 1024: 12.5 for
// the 256 swarms, 55 for the uneven ones.
#include <algorithm>
#include <new>
#include <queue>
#include <utility>

#include "pps_batch.h"
#include "pps_resident.cuh"

namespace pps {

// The lines of the figures above: the mean coordinates of a swarm, the largest
// dim and the waves up to which a batch takes this form.
constexpr int64_t kBatchResidentMean = 1500;
constexpr int kBatchResidentMaxDim = 128;
constexpr int64_t kBatchResidentWaves = 5;
// coordinates below which a block gains nothing from sharing its swarm further
constexpr int64_t kBatchResidentCoords = 1024;

struct ResidentJob {
  SwarmDev s;
  ObjParams op;
  PhiloxKeys keys;
  ResidentArgs a;
  float* result;
  int objective;
  int split;
};

// Sampling and the first global best (src/utils.jl:57-84, src/init.jl:102-106) by
// `share` blocks of one swarm, this one `rank` of them.
constexpr int kBatchInitThreads = 512;
template <int OBJ>
__device__ __forceinline__ unsigned long long init_swarm(const BatchSwarm& sw, int rank, int share) {
  const uint32_t k0 = (uint32_t)sw.seed, k1 = (uint32_t)(sw.seed >> 32);
  unsigned long long best = ~0ull;
  for (int64_t i = (int64_t)rank * blockDim.x + threadIdx.x; i < sw.n; i += (int64_t)share * blockDim.x) {
    Acc<OBJ> acc;
    for (int j = 0; j < sw.dim; j += 4) {
      const Rand4 r = philox4x32_10((uint32_t)i, (uint32_t)(j >> 2), 0u, kTagInit, k0, k1);
      const uint32_t rr[4] = {r.a, r.b, r.c, r.d};
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int d = j + h;
        if (d >= sw.dim) break;
        const float u = u01(rr[h]);
        float x;
        if (sw.sampler == PPS_SAMPLER_UNBOUNDED) {
          const float z = sw.u0[d];
          const float a = fabsf(z);
          x = (a > 0.0f) ? __fadd_rn(z, __fmul_rn(u, a)) : u;
        } else {
          x = __fadd_rn(__fmul_rn(u, __fsub_rn(sw.ub[d], sw.lb[d])), sw.lb[d]);
        }
        const int64_t o = (int64_t)d * sw.ld + i;
        sw.X[o] = x;
        sw.V[o] = 0.0f;
        sw.P[o] = x;
        acc.add(sw.op, d, x);
      }
    }
    const float c = finalize<OBJ>(sw.op, acc.s1, acc.s2);
    sw.cost[i] = c;
    sw.pcost[i] = c;
    const unsigned long long k = argmin_key(c, (uint32_t)i);
    best = k < best ? k : best;
  }
  return best;
}

// one swarm's sampling across blocks, zero at launch
struct InitCtl {
  unsigned long long inv_key;  // ~ the lowest argmin key so far
  unsigned int done;           // blocks finished
  unsigned int pad;
};

// Block (r, k) samples its share of swarm k; the last of the swarm's blocks takes
// the global best.  As many blocks a swarm as fill the GPU (a sampling alone, us
// with one / with these / by the streaming form's clusters: one swarm of 20,000 x 128-D
// 714 / 60 / 232, four 980 / 102 / 361).
__global__ void __launch_bounds__(kBatchInitThreads)
    k_batch_init(const BatchSwarm* __restrict__ descs, InitCtl* __restrict__ ctls) {
  __shared__ unsigned long long red[kBatchInitThreads / 32];
  __shared__ unsigned long long win_s;
  __shared__ int last_s;
  const BatchSwarm sw = descs[blockIdx.y];
  const int most = (int)((sw.n + kBatchInitThreads - 1) / kBatchInitThreads);
  const int share = most < (int)gridDim.x ? most : (int)gridDim.x, rank = (int)blockIdx.x;
  if (rank >= share) return;
  unsigned long long best = ~0ull;
  switch (sw.objective) {
    case kSphere: best = init_swarm<kSphere>(sw, rank, share); break;
    case kRosenbrock: best = init_swarm<kRosenbrock>(sw, rank, share); break;
    case kRastrigin: best = init_swarm<kRastrigin>(sw, rank, share); break;
    default: best = init_swarm<kAckley>(sw, rank, share); break;
  }
  best = warp_min_key(best);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = best;
  __threadfence();
  __syncthreads();
  if (threadIdx.x < 32) {
    best = warp_min_key(threadIdx.x < kBatchInitThreads / 32 ? red[threadIdx.x] : ~0ull);
    if (threadIdx.x == 0) {
      InitCtl* c = ctls + blockIdx.y;
      atomicMax(&c->inv_key, ~best);  // inverted, so zeroed memory is "none yet"
      __threadfence();
      last_s = atomicAdd(&c->done, 1u) == (unsigned int)(share - 1);
      __threadfence();
      if (last_s) win_s = ~atomicMax(&c->inv_key, 0ull);
    }
  }
  __syncthreads();
  if (!last_s) return;
  const int64_t gi = (int64_t)(uint32_t)win_s;
  for (int d = threadIdx.x; d < sw.dim; d += blockDim.x) sw.g[d] = __ldcg(sw.P + (int64_t)d * sw.ld + gi);
  if (threadIdx.x == 0) {
    sw.result[0] = __ldcg(sw.pcost + gi);
    sw.result[1] = __uint_as_float((uint32_t)gi);
    sw.result[2] = 0.0f;
  }
}

template <int OBJ>
__device__ __forceinline__ void run_job(const ResidentJob& j, int rank) {
  if (j.split)
    resident_run<OBJ, true, false, 2>(j.s, j.op, j.keys, j.a, rank, j.result);
  else
    resident_run<OBJ, false, false, 2>(j.s, j.op, j.keys, j.a, rank, j.result);
}

// blocks[b]: the job and the rank in it of block b
__global__ void __launch_bounds__(kResidentThreads, 1)
    k_batch_resident(const ResidentJob* __restrict__ jobs, const int2* __restrict__ blocks) {
  __shared__ __align__(16) ResidentJob job;
  const int2 at = blocks[blockIdx.x];
  const int* src = reinterpret_cast<const int*>(jobs + at.x);
  for (int k = threadIdx.x; k < (int)(sizeof(ResidentJob) / 4); k += blockDim.x) reinterpret_cast<int*>(&job)[k] = src[k];
  __syncthreads();
  switch (job.objective) {
    case kSphere: run_job<kSphere>(job, at.y); break;
    case kRosenbrock: run_job<kRosenbrock>(job, at.y); break;
    case kRastrigin: run_job<kRastrigin>(job, at.y); break;
    default: run_job<kAckley>(job, at.y); break;
  }
}

// ---------------------------------------------------------------- host side
struct BatchResident {
  void* mem = nullptr;
  size_t cap = 0;
};
BatchResident* batch_resident_create() { return new (std::nothrow) BatchResident(); }
void batch_resident_destroy(BatchResident* t) {
  if (!t) return;
  if (t->mem) cudaFree(t->mem);
  delete t;
}

size_t batch_resident_bytes(const BatchResident* t) { return t ? t->cap : 0; }

// the blocks' limits with `per` of them on an SM
constexpr size_t kJobStatic = 6u << 10;  // static shared memory of k_batch_resident, and the driver's 1 kB a block
static int most_threads(int per) { return kResidentThreads / per; }
static size_t most_smem(int per) { return ((size_t)(227u << 10) / per - kJobStatic) / 16 * 16; }
static bool job_fit(const BatchSwarm& d, int blocks, int per, ResidentPlan* p) {
  return resident_fit(d.objective, d.dim, d.n, false, blocks, most_threads(per), most_smem(per), p);
}
static int64_t coords_of(const BatchSwarm& d) { return d.n * (int64_t)((d.dim + 1) / 2 * 2); }

int batch_resident_launch(BatchResident* t, cudaStream_t stream, const std::vector<BatchSwarm>& descs,
                          const std::vector<std::vector<float>>& host, const BatchSwarm* ddescs, int sm_count,
                          bool* taken, unsigned int** error_word, int* threads) {
  *taken = false;
  const int ns = (int)descs.size();
  // blocks per SM: one of 512 threads, or more and smaller ones while the
  // swarms are small (a block of few coordinates waits for its own latencies)
  int64_t coords = 0;
  for (const auto& d : descs) {
    if (d.dim > kBatchResidentMaxDim) return PPS_OK;
    coords += coords_of(d);
  }
  const int64_t mean = coords / ns;
  if (mean < kBatchResidentMean) return PPS_OK;
  const int per = mean < 8000 ? 2 : 1;
  const int slots = sm_count * per;
  // the fewest blocks that hold each swarm
  std::vector<int> least(ns);
  int64_t total = 0;
  for (int k = 0; k < ns; ++k) {
    const BatchSwarm& d = descs[k];
    if (is_ode(d.objective) || !pair_form(d.objective, d.op, d.dim, host[k].data(), host[k].data() + d.dim, d.c1, d.c2))
      return PPS_OK;
    ResidentPlan p;
    int b = 1;
    while (b <= slots && !job_fit(d, b, per, &p)) ++b;
    if (b > slots) return PPS_OK;
    least[k] = b;
    total += b;
  }
  // waves: swarms of like iteration counts together, as many waves as the
  // fewest blocks need, filled evenly
  std::vector<int> by(ns);
  for (int k = 0; k < ns; ++k) by[k] = k;
  std::stable_sort(by.begin(), by.end(), [&](int a, int b) {
    if (descs[a].maxiters != descs[b].maxiters) return descs[a].maxiters > descs[b].maxiters;
    return coords_of(descs[a]) > coords_of(descs[b]);
  });
  const int64_t nwaves = (total + slots - 1) / slots;
  if (nwaves > kBatchResidentWaves) return PPS_OK;
  const int64_t share = (total + nwaves - 1) / nwaves;
  std::vector<std::vector<int>> waves;
  int64_t load = share;
  for (int k : by) {
    if (load >= share || load + least[k] > slots) {
      waves.emplace_back();
      load = 0;
    }
    waves.back().push_back(k);
    load += least[k];
  }
  // blocks of a wave: every SM's, dealt to the swarm whose blocks hold most
  std::vector<ResidentJob> jobs;
  std::vector<int2> table;
  std::vector<int> wave_at{0};
  std::vector<size_t> wave_smem, job_xch;
  std::vector<int> wave_threads;
  size_t xch_words = 0;
  for (const auto& w : waves) {
    std::vector<int> blocks;
    int used = 0;
    for (int k : w) {
      blocks.push_back(least[k]);
      used += least[k];
    }
    using Load = std::pair<int64_t, int>;
    std::priority_queue<Load> most;
    for (size_t e = 0; e < w.size(); ++e) most.push({coords_of(descs[w[e]]) / blocks[e], (int)e});
    while (used < slots && !most.empty()) {
      const Load l = most.top();
      most.pop();
      const int e = l.second;
      if (l.first < kBatchResidentCoords || blocks[e] >= descs[w[e]].n) continue;  // small enough
      ++blocks[e];
      ++used;
      most.push({coords_of(descs[w[e]]) / blocks[e], e});
    }
    size_t smem = 0;
    int block = 32;
    for (size_t e = 0; e < w.size(); ++e) {
      const BatchSwarm& d = descs[w[e]];
      ResidentPlan p;
      if (!job_fit(d, blocks[e], per, &p) && !job_fit(d, least[w[e]], per, &p)) return PPS_OK;
      ResidentJob j{};
      j.s.X = d.X;
      j.s.V = d.V;
      j.s.P = d.P;
      j.s.pcost = d.pcost;
      j.s.cost = d.cost;
      j.s.g = d.g;
      j.s.lb = const_cast<float*>(d.lb);
      j.s.ub = const_cast<float*>(d.ub);
      j.s.n = j.s.nglobal = d.n;
      j.s.npad = d.ld;
      j.s.dim = d.dim;
      j.op = d.op;
      j.keys = philox_round_keys(d.seed);
      j.a.chunk = p.chunk;
      j.a.blocks = p.blocks;
      j.a.groups = p.groups;
      j.a.iters = d.maxiters;
      j.a.w0 = d.w;
      j.a.wdamp = d.wdamp;
      j.a.c1s = d.c1 * 0x1p-24f;
      j.a.c2s = d.c2 * 0x1p-24f;
      j.a.start_limit = kResidentStartLimit;
      j.a.poll_limit = wait_polls(kResidentPollLimit);
      j.a.one = 1.0f;
      j.result = d.result;
      j.objective = d.objective;
      j.split = p.split ? 1 : 0;
      if (d.maxiters < 1) continue;  // its sampling is its result
      job_xch.push_back(xch_words);
      if (p.blocks > 1) xch_words += 2 * resident_words(p.blocks, d.dim);
      for (int r = 0; r < p.blocks; ++r) table.push_back(make_int2((int)jobs.size(), r));
      jobs.push_back(j);
      smem = std::max(smem, p.smem);
      block = std::max(block, p.threads);
    }
    wave_at.push_back((int)table.size());
    wave_smem.push_back(smem);
    wave_threads.push_back(block);
  }
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  // zeroed: the samplings' words, the exchange words, the error word
  const size_t binit = sizeof(InitCtl) * (size_t)ns;
  const size_t bzero = up(binit + sizeof(unsigned long long) * xch_words + sizeof(unsigned int));
  const size_t bjobs = up(sizeof(ResidentJob) * jobs.size()), need = bzero + bjobs + sizeof(int2) * table.size() + 256;
  if (t->cap < need) {
    if (t->mem) cudaFree(t->mem);
    t->mem = nullptr;
    t->cap = 0;
    PPS_CUDA(cudaMalloc(&t->mem, need));
    t->cap = need;
  }
  char* m = static_cast<char*>(t->mem);
  unsigned long long* xch = reinterpret_cast<unsigned long long*>(m + binit);
  unsigned int* status = reinterpret_cast<unsigned int*>(xch + xch_words);
  for (size_t k = 0; k < jobs.size(); ++k) {
    jobs[k].a.xch = xch + job_xch[k];
    jobs[k].a.status = status;
  }
  ResidentJob* djobs = reinterpret_cast<ResidentJob*>(m + bzero);
  int2* dtable = reinterpret_cast<int2*>(m + bzero + bjobs);
  PPS_CUDA(cudaMemsetAsync(m, 0, bzero, stream));
  if (!jobs.empty()) {
    PPS_CUDA(cudaMemcpyAsync(djobs, jobs.data(), sizeof(ResidentJob) * jobs.size(), cudaMemcpyHostToDevice, stream));
    PPS_CUDA(cudaMemcpyAsync(dtable, table.data(), sizeof(int2) * table.size(), cudaMemcpyHostToDevice, stream));
    PPS_CUDA(cudaFuncSetAttribute(k_batch_resident, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)most_smem(1)));
  }
  int64_t longest = 1;
  for (const auto& d : descs) longest = std::max(longest, d.n);
  const int64_t fill = std::max(8 * sm_count / ns, 1), most = (longest + kBatchInitThreads - 1) / kBatchInitThreads;
  // (y: the waves hold far fewer swarms than a grid's 65,535)
  k_batch_init<<<dim3((unsigned)std::min(fill, most), (unsigned)ns), kBatchInitThreads, 0, stream>>>(
      ddescs, reinterpret_cast<InitCtl*>(m));
  PPS_CUDA(cudaGetLastError());
  for (size_t v = 0; v < waves.size(); ++v) {
    const int nblocks = wave_at[v + 1] - wave_at[v];
    if (nblocks == 0) continue;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)nblocks);
    cfg.blockDim = dim3((unsigned)wave_threads[v]);
    cfg.dynamicSmemBytes = wave_smem[v];
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const cudaError_t e =
        cudaLaunchKernelEx(&cfg, k_batch_resident, (const ResidentJob*)djobs, (const int2*)(dtable + wave_at[v]));
    if (e == cudaErrorCooperativeLaunchTooLarge) {  // nothing but samplings so far: the other form starts over
      cudaGetLastError();
      return PPS_OK;
    }
    if (e != cudaSuccess) return cuda_error(e, "cudaLaunchKernelEx(k_batch_resident)");
  }
  *error_word = status;
  *threads = kBatchInitThreads;  // the sampling's block, where no swarm has an iteration to run
  if (!jobs.empty()) *threads = *std::max_element(wave_threads.begin(), wave_threads.end());
  *taken = true;
  return PPS_OK;
}

}  // namespace pps
