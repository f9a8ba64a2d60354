// The per-mechanism module of the generated variant: the plan's generated
// PTX (codegen.cpp) linked with the relocatable integrator (generated.cu,
// compiled at build time and embedded in this library) by nvJitLink, loaded
// as a CUDA library, kept on disk by content hash.
//
// nvJitLink is opened at run time (dlopen), so the library loads on hosts
// without it; fo_plan_generate then fails with a clear message. Linking runs
// ptxas on the generated code, some seconds on 16 cores for a 210-species /
// 500-reaction mechanism (200,000 multiply-adds); the cache makes that a
// one-time cost per mechanism and host.
#include "jit.h"

#include <cuda_runtime.h>
#include <dlfcn.h>
#include <nvJitLink.h>
#include <sys/stat.h>
#include <unistd.h>

#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <mutex>
#include <numeric>
#include <sstream>
#include <string>
#include <vector>

#include "codegen.h"

// the relocatable integrator (embed.cpp)
extern "C" const unsigned char fo_generated_rdc_begin[];
extern "C" const unsigned char fo_generated_rdc_end[];

namespace fo {
namespace {

struct JitLink {
  bool loaded = false;
  std::string error;
  decltype(&__nvJitLinkCreate_13_0) create = nullptr;
  decltype(&__nvJitLinkDestroy_13_0) destroy = nullptr;
  decltype(&__nvJitLinkAddData_13_0) add_data = nullptr;
  decltype(&__nvJitLinkComplete_13_0) complete = nullptr;
  decltype(&__nvJitLinkGetLinkedCubinSize_13_0) cubin_size = nullptr;
  decltype(&__nvJitLinkGetLinkedCubin_13_0) cubin = nullptr;
  decltype(&__nvJitLinkGetErrorLogSize_13_0) error_log_size = nullptr;
  decltype(&__nvJitLinkGetErrorLog_13_0) error_log = nullptr;
};

std::mutex g_jit_mutex;

const JitLink& jitlink() {
  static JitLink api;
  static bool tried = false;
  std::lock_guard<std::mutex> lock(g_jit_mutex);
  if (tried) return api;
  tried = true;
  const char* names[] = {"libnvJitLink.so.13", "libnvJitLink.so", "/usr/local/cuda/lib64/libnvJitLink.so.13"};
  void* h = nullptr;
  for (const char* nm : names)
    if ((h = dlopen(nm, RTLD_NOW | RTLD_LOCAL)) != nullptr) break;
  if (!h) {
    api.error = "libnvJitLink.so.13 (CUDA 13 nvJitLink) could not be opened: the generated variant needs it";
    return api;
  }
  bool ok = true;
  auto sym = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(dlsym(h, name));
    if (!fn) ok = false;
  };
  sym(api.create, "__nvJitLinkCreate_13_0");
  sym(api.destroy, "__nvJitLinkDestroy_13_0");
  sym(api.add_data, "__nvJitLinkAddData_13_0");
  sym(api.complete, "__nvJitLinkComplete_13_0");
  sym(api.cubin_size, "__nvJitLinkGetLinkedCubinSize_13_0");
  sym(api.cubin, "__nvJitLinkGetLinkedCubin_13_0");
  sym(api.error_log_size, "__nvJitLinkGetErrorLogSize_13_0");
  sym(api.error_log, "__nvJitLinkGetErrorLog_13_0");
  if (!ok) {
    api.error = "libnvJitLink lacks the CUDA 13.0 entry points";
    return api;
  }
  api.loaded = true;
  return api;
}

// The link: sm_103a; at most 128 registers per thread, the integrator
// kernel's budget for sixteen groups per SM, for the generated functions too;
// ptxas optimizes the module's functions (the factorization's pieces among
// them) on all host cores at once.
const char* const kLinkOptions[] = {"-arch=sm_103a", "-O3", "-maxrregcount=128", "-Xptxas=--split-compile=0"};

uint64_t fnv1a(uint64_t h, const void* data, size_t n) {
  const unsigned char* p = static_cast<const unsigned char*>(data);
  for (size_t i = 0; i < n; ++i) {
    h ^= p[i];
    h *= 1099511628211ull;
  }
  return h;
}

std::string default_cache_dir() {
  if (const char* e = std::getenv("FASTODE_GB300_CACHE")) return e;
  if (const char* x = std::getenv("XDG_CACHE_HOME")) return std::string(x) + "/fastode_gb300";
  if (const char* h = std::getenv("HOME")) return std::string(h) + "/.cache/fastode_gb300";
  return "";
}

void make_dirs(const std::string& dir) {
  std::string cur;
  std::stringstream ss(dir);
  std::string part;
  if (!dir.empty() && dir[0] == '/') cur = "/";
  while (std::getline(ss, part, '/')) {
    if (part.empty()) continue;
    cur += part + "/";
    mkdir(cur.c_str(), 0755);
  }
}

bool read_file(const std::string& path, std::vector<char>* out) {
  std::ifstream f(path, std::ios::binary);
  if (!f) return false;
  f.seekg(0, std::ios::end);
  const std::streamoff n = f.tellg();
  if (n <= 0) return false;
  f.seekg(0);
  out->resize((size_t)n);
  f.read(out->data(), n);
  return (bool)f;
}

void write_file_atomic(const std::string& path, const std::vector<char>& data) {
  const std::string tmp = path + ".tmp" + std::to_string(getpid());
  {
    std::ofstream f(tmp, std::ios::binary);
    if (!f) return;
    f.write(data.data(), (std::streamsize)data.size());
    if (!f) {
      std::remove(tmp.c_str());
      return;
    }
  }
  if (std::rename(tmp.c_str(), path.c_str()) != 0) std::remove(tmp.c_str());
}

bool link(const std::string& ptx, std::vector<char>* cubin, std::string* err) {
  const JitLink& api = jitlink();
  if (!api.loaded) {
    *err = api.error;
    return false;
  }
  nvJitLinkHandle h = nullptr;
  if (api.create(&h, (uint32_t)(sizeof(kLinkOptions) / sizeof(kLinkOptions[0])), kLinkOptions) !=
      NVJITLINK_SUCCESS) {
    *err = "nvJitLinkCreate failed";
    return false;
  }
  auto log = [&]() {
    size_t n = 0;
    std::string s;
    if (api.error_log_size(h, &n) == NVJITLINK_SUCCESS && n > 1) {
      s.resize(n);
      api.error_log(h, &s[0]);
      s.resize(n - 1);
    }
    return s;
  };
  bool ok = api.add_data(h, NVJITLINK_INPUT_CUBIN, fo_generated_rdc_begin,
                         (size_t)(fo_generated_rdc_end - fo_generated_rdc_begin), "generated.cu") == NVJITLINK_SUCCESS;
  ok = ok && api.add_data(h, NVJITLINK_INPUT_PTX, ptx.data(), ptx.size(), "mechanism.ptx") == NVJITLINK_SUCCESS;
  ok = ok && api.complete(h) == NVJITLINK_SUCCESS;
  size_t n = 0;
  ok = ok && api.cubin_size(h, &n) == NVJITLINK_SUCCESS && n > 0;
  if (ok) {
    cubin->resize(n);
    ok = api.cubin(h, cubin->data()) == NVJITLINK_SUCCESS;
  }
  if (!ok) *err = "nvJitLink failed: " + log();
  api.destroy(&h);
  return ok;
}

}  // namespace

struct GenModule {
  cudaLibrary_t lib = nullptr;
  cudaKernel_t kernel = nullptr;        // fo_generated_solve_kernel
  cudaKernel_t multi_kernel = nullptr;  // fo_generated_multi_kernel
  cudaKernel_t adjoint_kernel = nullptr;  // fo_generated_adjoint_kernel
  std::mutex mutex;
  int64_t attempt_work = 0;               // FP64 operations of an attempt (the largest mechanism's)
  bool may_cluster = false;
  int clusters[64][4] = {};               // resident clusters of 2^i blocks, plus one (0: not asked yet)
};

int gen_create(const std::vector<const HostTables*>& ts, const std::vector<GenOptions>& opts, const char* cache_dir,
               GenModule** out, fo_gen_info* info, std::string* err) {
  const auto t0 = std::chrono::steady_clock::now();
  *out = nullptr;
  std::string ptx;
  try {
    ptx = generate_ptx(ts, opts);
  } catch (const std::exception& e) {
    *err = std::string("code generation failed: ") + e.what();
    return FO_E_INVALID;
  }
  int runtime = 0;
  cudaRuntimeGetVersion(&runtime);
  uint64_t h = 1469598103934665603ull;
  h = fnv1a(h, ptx.data(), ptx.size());
  h = fnv1a(h, fo_generated_rdc_begin, (size_t)(fo_generated_rdc_end - fo_generated_rdc_begin));
  h = fnv1a(h, &runtime, sizeof(runtime));
  for (const char* o : kLinkOptions) h = fnv1a(h, o, std::strlen(o));
  char key[32];
  std::snprintf(key, sizeof(key), "gen-%016llx.cubin", (unsigned long long)h);
  const std::string dir = cache_dir ? std::string(cache_dir) : default_cache_dir();
  const std::string path = dir.empty() ? "" : dir + "/" + key;
  std::vector<char> cubin;
  bool cached = !path.empty() && read_file(path, &cubin);
  if (!cached) {
    if (!link(ptx, &cubin, err)) return FO_E_UNSUPPORTED;
    if (!path.empty()) {
      make_dirs(dir);
      write_file_atomic(path, cubin);
    }
  }
  GenModule* m = new GenModule;
  cudaError_t e = cudaLibraryLoadData(&m->lib, cubin.data(), nullptr, nullptr, 0, nullptr, nullptr, 0);
  if (e == cudaSuccess) e = cudaLibraryGetKernel(&m->kernel, m->lib, "fo_generated_solve_kernel");
  if (e == cudaSuccess) e = cudaLibraryGetKernel(&m->multi_kernel, m->lib, "fo_generated_multi_kernel");
  if (e == cudaSuccess) e = cudaLibraryGetKernel(&m->adjoint_kernel, m->lib, "fo_generated_adjoint_kernel");
  cudaFuncAttributes attr;
  std::memset(&attr, 0, sizeof(attr));
  if (e == cudaSuccess) e = cudaFuncGetAttributes(&attr, reinterpret_cast<const void*>(m->kernel));
  if (e != cudaSuccess) {
    *err = std::string("loading the generated module: ") + cudaGetErrorString(e);
    if (m->lib) cudaLibraryUnload(m->lib);
    delete m;
    return FO_E_CUDA;
  }
  if (info) {
    std::memset(info, 0, sizeof(*info));
    info->from_cache = cached ? 1 : 0;
    info->registers = attr.numRegs;
    info->tile = opts.empty() ? 0 : opts[0].tile;
    info->local_bytes = (int32_t)attr.localSizeBytes;
    info->ptx_bytes = (int64_t)ptx.size();
    info->cubin_bytes = (int64_t)cubin.size();
    info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  }
  for (const HostTables* t : ts)
    m->attempt_work = std::max(m->attempt_work, t->lu_fma + 3 * t->solve_fma + (int64_t)t->jt_idx.size() +
                                                    2 * (int64_t)t->s_rxn.size());
  // a cluster's blocks exchange a value each through the items of the slot's
  // partial derivatives and rates, of which there are at least R
  m->may_cluster = ts.size() == 1 && ts[0]->R >= kMaxCluster;
  *out = m;
  return FO_OK;
}

int gen_check(const HostTables& t, const GenOptions& opt, bool do_link, fo_gen_info* info, std::string* err) {
  const auto t0 = std::chrono::steady_clock::now();
  std::string ptx;
  try {
    ptx = generate_ptx(t, opt);
  } catch (const std::exception& e) {
    *err = std::string("code generation failed: ") + e.what();
    return FO_E_INVALID;
  }
  std::vector<char> cubin;
  if (do_link && !link(ptx, &cubin, err)) return FO_E_UNSUPPORTED;
  if (info) {
    std::memset(info, 0, sizeof(*info));
    info->tile = opt.tile;
    info->ptx_bytes = (int64_t)ptx.size();
    info->cubin_bytes = (int64_t)cubin.size();
    info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
  }
  return FO_OK;
}

void gen_destroy(GenModule* m) {
  if (!m) return;
  if (m->lib) cudaLibraryUnload(m->lib);
  delete m;
}

namespace {

// Multiprocessors of the current device, or 0.
int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return sms;
}

// Warps per group for a launch of `grid` blocks on the current device: the
// largest power of two, up to kBlockWarps, that still leaves every block
// resident at sixteen warps per SM (the kernels' 128 registers per thread):
// beyond that a larger team only makes groups wait for one another. One warp
// per group and a team, measured on a GB300: eight intervals of TS1 on 64
// cells (2 groups, teams of 16) 142 and 42 ms; two intervals on 8,200 cells
// (257 groups, teams of 8) 27.0 and 9.2 ms; the cold interval of 16,384 cells
// of the 210/500 mechanism (512 groups, teams of 4) 452 and 270 ms.
int team_of(int grid) {
  const int sms = device_sms();
  int team = 1;
  while (2 * team <= kBlockWarps && (int64_t)grid * 2 * team <= (int64_t)sms * 16) team *= 2;
  return team;
}

// Whether lockstep rounds pay for a launch of `grid` blocks: they keep the
// groups of an SM in the same part of the generated code and let them solve
// together, which takes two groups on the fullest SMs and on half of them. With
// and without rounds, ms: one cold interval of 210/500, 6,400 cells (1.3 groups
// per SM) 110.4 and 108.4; 8,192 (1.7) 114 and 122; 9,600 119 and 160; 13,000
// 163 and 218; 16,384 206 and 305; 65,536 716 and 1135; settled, 65,536 cells
// 107 and 137, 100,000 (more groups than slots) 208 and 218; TS1 settled, 8,200
// cells 4.37 and 4.69, 65,536 23.1 and 33.3. The code of a small mechanism
// stays in the instruction cache by itself (9,000 cells cold, ms, synthetic
// mechanisms of seed 3, the larger two with third bodies: 20/40, 1,435
// operations (attempt_work), 1.52 and 1.44; 36/75, 4,130, 2.13 and 2.03; 48/100,
// 7,330, 5.00 and 5.61).
constexpr int64_t kRoundsWork = 5000;

// Blocks per cluster for a launch of `grid` groups on teams of kBlockWarps
// warps: the largest of 8, 4 and 2 with which all clusters are resident at
// once, or one. A cluster's barrier and the operands' way through L2 cost
// about 2,200 cycles a step (a block's barrier 45, its operands come from L1),
// so a mechanism with little work per attempt (attempt_work) stays on one SM:
// 20/40 (1,064 to 1,623 operations by its seed) does, TS1 (20,867) does not.
// One SM and a cluster, measured: a cold interval of one 210/500 group 66.5 and
// 32.0 ms, eight intervals of TS1 on two groups 34.4 and 25.8 ms (both with the
// leading rows' tasks split); two Newton iterations of backward Euler on 42
// groups of 120/260 (clusters of 2) 1.42 and 1.23 ms.
constexpr int64_t kClusterWork = 10000;
constexpr size_t kClusterSmem = sizeof(double) * (32 + 32 * kBlockWarps);

cudaLaunchConfig_t cluster_config(int grid, int blocks, cudaStream_t stream, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid * blocks);
  c.blockDim = dim3(32, kBlockWarps);
  c.dynamicSmemBytes = kClusterSmem;
  c.stream = stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = blocks;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  c.attrs = attr;
  c.numAttrs = 1;
  return c;
}

int cluster_of(GenModule* m, const void* fn, int grid) {
  int dev = 0;
  if (!m->may_cluster || m->attempt_work < kClusterWork || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
  std::lock_guard<std::mutex> lock(m->mutex);
  for (int i = 3; i > 0; --i) {
    int& known = m->clusters[dev][i];
    if (known == 0) {
      int n = 0;
      cudaLaunchAttribute attr;
      const cudaLaunchConfig_t c = cluster_config(1, 1 << i, nullptr, &attr);
      if (cudaOccupancyMaxActiveClusters(&n, fn, &c) != cudaSuccess) {
        (void)cudaGetLastError();
        n = 0;
      }
      known = n + 1;
    }
    if (grid <= known - 1) return 1 << i;
  }
  return 1;
}

}  // namespace

bool gen_rounds_pay(const GenModule* m, int grid) {
  const int sms = device_sms();
  return m->attempt_work >= kRoundsWork && sms > 0 && 2 * (int64_t)grid > 3 * (int64_t)sms;
}

cudaError_t gen_launch(GenModule* m, const SolveParams& p, int grid, size_t smem, cudaStream_t stream) {
  const void* fn = reinterpret_cast<const void*>(m->kernel);
  SolveParams q = p;
  void* args[] = {&q};
  const int team = team_of(grid);
  if (team == kBlockWarps && q.queue == nullptr && q.rounds == nullptr) {
    const int blocks = cluster_of(m, fn, grid);
    if (blocks > 1) {
      cudaLaunchAttribute attr;
      const cudaLaunchConfig_t c = cluster_config(grid, blocks, stream, &attr);
      return cudaLaunchKernelExC(&c, fn, args);
    }
  }
  return cudaLaunchKernel(fn, dim3(grid), dim3(32, team), args, smem, stream);
}

cudaError_t gen_launch_adjoint(GenModule* m, const AdjParams& a, int grid, size_t smem, cudaStream_t stream) {
  const void* fn = reinterpret_cast<const void*>(m->adjoint_kernel);
  AdjParams q = a;
  void* args[] = {&q};
  return cudaLaunchKernel(fn, dim3(grid), dim3(32, team_of(grid)), args, smem, stream);
}

cudaError_t gen_launch_multi(GenModule* m, const SolveParams* batches, int nb, const int32_t* starts,
                             int32_t* queue, double* scratch, int64_t slot_doubles, int grid, size_t smem,
                             cudaStream_t stream) {
  const void* fn = reinterpret_cast<const void*>(m->multi_kernel);
  cudaError_t e = cudaMemsetAsync(queue, 0, sizeof(int32_t), stream);
  if (e != cudaSuccess) return e;
  void* args[] = {&batches, &nb, &starts, &queue, &scratch, &slot_doubles};
  return cudaLaunchKernel(fn, dim3(grid), dim3(32, team_of(grid)), args, smem, stream);
}

}  // namespace fo
