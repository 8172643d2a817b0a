// extern "C" surface of libevoattn.so: argument validation, dispatch, launches.
#include <string.h>

#include <mutex>

#include "common.cuh"
#include "launch.h"

namespace {

thread_local int g_last_path = EVOATTN_PATH_NONE;
thread_local int g_last_launches = 0;
thread_local int g_ctx_bound_device = -1;

// Tensor maps are encoded through the driver API, which needs the device's primary context
// to be current on the calling thread.  A thread that has made no runtime call yet (PyTorch's
// autograd worker on its first backward) gets it bound here, once per thread and device.
void bind_context_once() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  if (g_ctx_bound_device != dev) {
    cudaFree(nullptr);  // the customary no-op that initialises / binds the primary context
    g_ctx_bound_device = dev;
  }
}

bool stride_ok16(const int64_t* s, int esize) {
  for (int i = 0; i < 4; ++i)
    if ((s[i] * esize) % 16 != 0) return false;
  return true;
}

evo::Str4 str4(const int64_t* s) { return evo::Str4{s[0], s[1], s[2], s[3]}; }

int esize_of(int dtype) { return dtype == EVOATTN_FP32 ? 4 : 2; }

int validate_fwd(const evoattn_fwd_params* p) {
  if (!p) return EVOATTN_ERR_NULL;
  if (!p->q || !p->k || !p->v || !p->o || !p->lse) return EVOATTN_ERR_NULL;
  if (p->dtype != EVOATTN_BF16 && p->dtype != EVOATTN_FP16 && p->dtype != EVOATTN_FP32) return EVOATTN_ERR_DTYPE;
  if (p->B <= 0 || p->H <= 0 || p->S <= 0 || p->R <= 0 || p->D <= 0) return EVOATTN_ERR_SHAPE;
  if ((long long)p->B * p->H * p->S > 2147483647LL) return EVOATTN_ERR_SHAPE;
  if (p->R > 65535 * 8) return EVOATTN_ERR_SHAPE;
  if (p->D > 128) return EVOATTN_ERR_UNSUPPORTED;
  if (p->mask_kind < EVOATTN_MASK_NONE || p->mask_kind > EVOATTN_MASK_ADD_SAME) return EVOATTN_ERR_DTYPE;
  if (p->mask_kind != EVOATTN_MASK_NONE && !p->mask) return EVOATTN_ERR_NULL;
  if (p->bias_dtype != EVOATTN_BIAS_F32 && p->bias_dtype != EVOATTN_BIAS_SAME) return EVOATTN_ERR_DTYPE;
  if (!(p->scale == p->scale)) return EVOATTN_ERR_SHAPE;  // NaN scale
  return EVOATTN_OK;
}

void fill_args(const evoattn_fwd_params* p, evo::Args* a) {
  memset(a, 0, sizeof(*a));
  a->B = p->B; a->H = p->H; a->S = p->S; a->R = p->R; a->D = p->D;
  a->scale = p->scale;
  a->q = p->q; a->k = p->k; a->v = p->v; a->o = p->o; a->lse = p->lse;
  a->sq = str4(p->q_stride); a->sk = str4(p->k_stride); a->sv = str4(p->v_stride); a->so = str4(p->o_stride);
  a->mask = p->mask_kind == EVOATTN_MASK_NONE ? nullptr : p->mask;
  a->mask_kind = p->mask_kind;
  a->smask = evo::Str3{p->mask_stride[0], p->mask_stride[1], p->mask_stride[2]};
  a->bias = reinterpret_cast<const float*>(p->bias);
  a->sbias = evo::Str3{p->bias_stride[0], p->bias_stride[1], p->bias_stride[2]};
  a->bias16 = (p->bias && p->bias_dtype == EVOATTN_BIAS_SAME && p->dtype != EVOATTN_FP32) ? 1 : 0;
  a->status = p->status;
  a->gate = p->gate;
  a->sgate = str4(p->gate_stride);
}

int validate_bwd(const evoattn_bwd_params* p) {
  if (!p) return EVOATTN_ERR_NULL;
  int rc = validate_fwd(&p->fwd);
  if (rc) return rc;
  if (!p->d_o || !p->dq || !p->dk || !p->dv) return EVOATTN_ERR_NULL;
  if (p->fwd.gate && !p->dgate) return EVOATTN_ERR_NULL;
  if (p->dbias_cast) {
    if (p->dbias || p->exchange) return EVOATTN_ERR_SHAPE;  // one destination
    if (p->dbias_cast_dtype < EVOATTN_BF16 || p->dbias_cast_dtype > EVOATTN_FP32) return EVOATTN_ERR_DTYPE;
    if (p->dbias_cast_heads_last && (p->fwd.H > 96 || p->fwd.R > 65535 || p->fwd.B > 65535)) return EVOATTN_ERR_SHAPE;
  }
  if (p->exchange) {  // the in-call sum of d(pair_bias) over the node's GPUs works on the caller's exchange buffer
    const evoattn_peer_allreduce_params* x = p->exchange;
    if (!p->fwd.bias || !p->dbias || !x->bufs) return EVOATTN_ERR_NULL;
    if (x->world < 1 || x->world > 8 || x->rank < 0 || x->rank >= x->world) return EVOATTN_ERR_SHAPE;
    if (x->bufs[x->rank] != p->dbias) return EVOATTN_ERR_SHAPE;
    if (x->count != (uint64_t)p->fwd.B * p->fwd.H * p->fwd.R * p->fwd.R) return EVOATTN_ERR_SHAPE;
  }
  return EVOATTN_OK;
}

void fill_bwd_args(const evoattn_bwd_params* p, evo::Args* a) {
  fill_args(&p->fwd, a);
  a->d_o = p->d_o; a->dq = p->dq; a->dk = p->dk; a->dv = p->dv;
  a->dbias = p->fwd.bias ? p->dbias : nullptr;
  a->dbias_ld = a->R;
  if (p->fwd.bias && p->dbias_cast) {
    a->dbias_out = p->dbias_cast;
    a->dbias_out_dtype = p->dbias_cast_dtype;
    a->dbias_out_last = p->dbias_cast_heads_last;
  }
  if (p->fwd.gate) {
    a->dgate = p->dgate;
    a->sdgate = str4(p->dgate_stride);
  }
  a->sdo = str4(p->do_stride); a->sdq = str4(p->dq_stride); a->sdk = str4(p->dk_stride); a->sdv = str4(p->dv_stride);
  a->dmask = p->dmask;
  a->exchange = p->exchange;
}

bool use_sm100_fwd(const evoattn_fwd_params* p, const evo::Args& a) {
  if (p->flags & EVOATTN_FLAG_FORCE_GENERIC) return false;
  if (p->dtype == EVOATTN_FP32) return false;
  if (((uintptr_t)p->q | (uintptr_t)p->k | (uintptr_t)p->v | (uintptr_t)p->o) & 15) return false;
  const int es = esize_of(p->dtype);
  if (p->gate && ((((uintptr_t)p->gate) & 15) || !stride_ok16(p->gate_stride, es))) return false;
  if (!stride_ok16(p->q_stride, es) || !stride_ok16(p->k_stride, es) || !stride_ok16(p->v_stride, es) ||
      !stride_ok16(p->o_stride, es))
    return false;
  return evo::sm100_fwd_supported(p->dtype, a);
}

bool use_sm100_bwd(const evoattn_bwd_params* p, const evo::Args& a) {
  if (!use_sm100_fwd(&p->fwd, a)) return false;
  if (p->dmask) return false;  // the gradient of an additive mask is produced by the CUDA-core kernels
  if (((uintptr_t)p->d_o | (uintptr_t)p->dq | (uintptr_t)p->dk | (uintptr_t)p->dv) & 15) return false;
  const int es = esize_of(p->fwd.dtype);
  if (!stride_ok16(p->do_stride, es) || !stride_ok16(p->dq_stride, es) || !stride_ok16(p->dk_stride, es) ||
      !stride_ok16(p->dv_stride, es))
    return false;
  if (p->fwd.gate && ((((uintptr_t)p->dgate) & 15) || !stride_ok16(p->dgate_stride, es))) return false;
  // dK and dV leave through tensor maps, which know no backward steps.
  for (int i = 0; i < 4; ++i)
    if (p->dk_stride[i] < 0 || p->dv_stride[i] < 0) return false;
  // Of the odd lengths with a d(pair_bias), the smallest calls keep the dispatch that all of them once had:
  // the CUDA cores, with P and dS in fp32.  The line does not separate the faster kernels.  Backward calls in
  // us, tensor / CUDA cores, [B,S,R,H]: D = 8: [1,1,33,1] 15.7 / 9.6, [1,5,51,2] 16.5 / 12.8, [1,1,511,1]
  // 47.0 / 50.9; D = 32: 15.5 / 12.7, 16.8 / 16.2, 40.9 / 75.4; D = 64: 12.2 / 17.4, 13.0 / 21.8,
  // 27.1 / 107.2.  So it gains a few us at one tile of residues and D <= 32 and loses elsewhere; moving a
  // call across it would take its P and dS to 16 bits (errors 1.4 times as large).
  if (p->fwd.bias && (p->dbias || p->dbias_cast) && p->fwd.R % 4 != 0 && (long long)a.B * a.H * a.S * a.R <= 512) return false;
  return evo::sm100_bwd_supported(p->fwd.dtype, a);
}

// Scratch of evoattn_bwd_static_scratch(): part of the library image, so every GPU that loads
// the library holds it until the process exits.  In host code this name is only a stand-in
// for the symbol, never a device address: the address is looked up per device below.
static __device__ __align__(256) unsigned char g_static_scratch[EVOATTN_STATIC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
void* g_static_scratch_addr[kMaxDevices] = {};
std::mutex g_static_scratch_mutex;

// Device address of the static scratch on the current device.  The lookup is repeated on every
// call: it is cheap, it allocates nothing, and it is also what makes the device's primary
// context current on a host thread that has made no CUDA call yet (a fresh worker thread, the
// autograd engine's thread), which the tensor-map encoder needs.  The per-device table is only a
// cross-check that the address never changes.
int static_scratch_address(void** out) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return EVOATTN_ERR_CUDA;
  void* ptr = nullptr;
  if (cudaGetSymbolAddress(&ptr, g_static_scratch) != cudaSuccess || !ptr) return EVOATTN_ERR_CUDA;
  {
    std::lock_guard<std::mutex> lock(g_static_scratch_mutex);
    if (!g_static_scratch_addr[dev]) g_static_scratch_addr[dev] = ptr;
    else if (g_static_scratch_addr[dev] != ptr) return EVOATTN_ERR_CUDA;
  }
  *out = ptr;
  return EVOATTN_OK;
}

// Row stride of the statistics the tensor-core backward reads through tensor maps: whole 16-byte pieces.
int stats_ld(const evo::Args& a) { return (a.R + 3) / 4 * 4; }

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// Scratch of a backward call, in this order: what the kernel family needs (delta first), the effective
// dO of a gated output, and the fp32 buffer d(pair_bias) is summed in where the caller's own cannot be
// it: another type or layout, or (tensor reductions) rows that are not whole 16-byte pieces.
struct Scratch {
  size_t path, gate, dbias;
  size_t total() const { return path + gate + dbias; }
};
Scratch plan_scratch(const evoattn_bwd_params* p, evo::Args* a, bool fast) {
  a->delta_ld = fast ? stats_ld(*a) : a->R;
  Scratch s{};
  if (p->fwd.gate) s.gate = align256((size_t)a->B * a->H * a->S * a->R * a->D * esize_of(p->fwd.dtype));
  if (fast) {
    s.path = evo::sm100_bwd_workspace_bytes(p->fwd.dtype, *a);
  } else {
    evo::Args want = *a;
    if (want.dbias_out) want.dbias = reinterpret_cast<float*>(want.dbias_out);  // (only whether there is one)
    s.path = evo::generic_bwd_workspace_bytes(want);
  }
  s.path = align256(s.path);
  const bool direct = a->dbias && (!fast || (a->R % 4 == 0 && (reinterpret_cast<uintptr_t>(a->dbias) & 15) == 0));
  if (a->dbias && !direct) {
    a->dbias_out = a->dbias;
    a->dbias_out_dtype = EVOATTN_FP32;
    a->dbias_out_last = 0;
  }
  if (a->dbias_out) {
    a->dbias_ld = fast ? stats_ld(*a) : a->R;
    s.dbias = align256((size_t)a->B * a->H * a->R * a->dbias_ld * sizeof(float));
  }
  return s;
}

// The same for scratch that cannot grow.  The CUDA-core kernels speed up with partial sums of
// d(pair_bias), one for each run of MSA rows; they take as many as there is room for, and need none.
Scratch plan_scratch_within(size_t limit, const evoattn_bwd_params* p, evo::Args* a, bool fast) {
  const Scratch all = plan_scratch(p, a, fast);
  if (fast || all.total() <= limit || !(a->dbias || a->dbias_out)) return all;
  a->max_runs = 1;
  const size_t least = plan_scratch(p, a, fast).total();  // (sizes and limit are multiples of 256)
  const size_t partial = (size_t)a->B * a->H * a->R * a->R * sizeof(float);
  if (least < limit && (limit - least) / partial > 1) a->max_runs = (int)((limit - least) / partial);
  return plan_scratch(p, a, fast);
}

// Whether a tensor map could take a call only because something was padded for it: rows of the bias, or
// of the d(pair_bias) that is wanted, that are not whole 16-byte pieces.
bool has_padded_rows(const evoattn_bwd_params* p, const evo::Args& a) {
  if (!a.bias) return false;
  if (a.R * (a.bias16 ? 2 : 4) % 16 != 0) return true;
  return (p->dbias || p->dbias_cast) && (a.R % 4 != 0 || ((uintptr_t)p->dbias & 15) != 0);
}

// The backward with its scratch at `scratch` (caller-provided or the static array).
int run_bwd(const evoattn_bwd_params* p, evo::Args& a, const Scratch& plan, bool fast, void* scratch, cudaStream_t st) {
  unsigned char* base = reinterpret_cast<unsigned char*>(scratch);
  a.delta = reinterpret_cast<float*>(base);  // every kernel family keeps delta at the start of its scratch
  if (plan.gate) a.d_o_eff = base + plan.path;
  if (plan.dbias) a.dbias = reinterpret_cast<float*>(base + plan.path + plan.gate);
  if (a.dmask &&
      cudaMemsetAsync(a.dmask, 0, (size_t)a.B * a.S * a.R * sizeof(float), st) != cudaSuccess)
    return EVOATTN_ERR_CUDA;
  if (fast) {
    g_last_path = EVOATTN_PATH_TCGEN05;
    return evo::launch_sm100_bwd(p->fwd.dtype, a, scratch, plan.path, st, &g_last_launches);
  }
  g_last_path = EVOATTN_PATH_GENERIC;
  if (evo::launch_generic_bwd(p->fwd.dtype, a, st, &g_last_launches) != cudaSuccess) return EVOATTN_ERR_CUDA;
  if (a.dbias_out) {
    const int rc = evo::launch_dbias_out(a, st, &g_last_launches);
    if (rc) return rc;
  }
  if (p->exchange) {  // (the CUDA-core kernels have nothing to run the exchange next to)
    const int rc = evo::launch_peer_allreduce(p->exchange, st);
    if (rc) return rc;
    g_last_launches += 1;
  }
  return EVOATTN_OK;
}

}  // namespace

extern "C" {

int evoattn_abi_version(void) { return EVOATTN_ABI_VERSION; }

const char* evoattn_strerror(int status) {
  switch (status) {
    case EVOATTN_OK: return "ok";
    case EVOATTN_ERR_NULL: return "a required pointer is null";
    case EVOATTN_ERR_SHAPE: return "a dimension or scale is out of range";
    case EVOATTN_ERR_DTYPE: return "unknown dtype or mask kind";
    case EVOATTN_ERR_ALIGN: return "base address or stride is not 16-byte aligned";
    case EVOATTN_ERR_UNSUPPORTED: return "no kernel covers this request (head dimension above 128?)";
    case EVOATTN_ERR_CUDA: return "a CUDA call failed (launch or tensor-map creation)";
    case EVOATTN_ERR_WORKSPACE: return "workspace is null or smaller than evoattn_bwd_workspace_bytes()";
    case EVOATTN_ERR_DEVICE: return "a kernel gave up a bounded wait and set the device status word";
    default: return "unknown status";
  }
}

int evoattn_fwd(const evoattn_fwd_params* p, void* cuda_stream) {
  g_last_path = EVOATTN_PATH_NONE;
  g_last_launches = 0;
  int rc = validate_fwd(p);
  if (rc) return rc;
  evo::Args a;
  fill_args(p, &a);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(cuda_stream);
  bind_context_once();
  if (use_sm100_fwd(p, a)) {
    g_last_path = EVOATTN_PATH_TCGEN05;
    return evo::launch_sm100_fwd(p->dtype, a, st, &g_last_launches);
  }
  g_last_path = EVOATTN_PATH_GENERIC;
  return evo::launch_generic_fwd(p->dtype, a, st, &g_last_launches) == cudaSuccess ? EVOATTN_OK : EVOATTN_ERR_CUDA;
}

size_t evoattn_bwd_workspace_bytes(const evoattn_bwd_params* p) {
  if (validate_bwd(p)) return 0;
  evo::Args a;
  fill_bwd_args(p, &a);
  return plan_scratch(p, &a, use_sm100_bwd(p, a)).total();
}

int evoattn_bwd(const evoattn_bwd_params* p, void* cuda_stream) {
  g_last_path = EVOATTN_PATH_NONE;
  g_last_launches = 0;
  int rc = validate_bwd(p);
  if (rc) return rc;
  evo::Args a;
  fill_bwd_args(p, &a);
  bind_context_once();
  const bool fast = use_sm100_bwd(p, a);
  const Scratch plan = plan_scratch(p, &a, fast);
  const size_t need = plan.total();
  if (need && (!p->workspace || p->workspace_bytes < need)) return EVOATTN_ERR_WORKSPACE;
  if (need && ((uintptr_t)p->workspace & 255)) return EVOATTN_ERR_ALIGN;
  return run_bwd(p, a, plan, fast, p->workspace, reinterpret_cast<cudaStream_t>(cuda_stream));
}

int evoattn_bwd_static_scratch(const evoattn_bwd_params* p, void* cuda_stream) {
  g_last_path = EVOATTN_PATH_NONE;
  g_last_launches = 0;
  int rc = validate_bwd(p);
  if (rc) return rc;
  evo::Args a;
  fill_bwd_args(p, &a);
  bool fast = use_sm100_bwd(p, a);
  Scratch plan = plan_scratch_within(EVOATTN_STATIC_SCRATCH_BYTES, p, &a, fast);
  // The tensor-core kernels need an fp32 dQ accumulator and, for the lengths below, a padded d(pair_bias)
  // (66 MiB at [1,128,501,8,32]); the CUDA-core kernels need one float per score row (2 MiB).  The lengths
  // that reach the tensor cores by padding have always been served from this array and still are; the
  // others have always been refused, and the caller chooses: a workspace, or EVOATTN_FLAG_FORCE_GENERIC.
  if (fast && plan.total() > EVOATTN_STATIC_SCRATCH_BYTES && has_padded_rows(p, a)) {
    fast = false;
    fill_bwd_args(p, &a);
    plan = plan_scratch_within(EVOATTN_STATIC_SCRATCH_BYTES, p, &a, fast);
  }
  if (plan.total() > EVOATTN_STATIC_SCRATCH_BYTES) return EVOATTN_ERR_WORKSPACE;
  // Looking the symbol up (done on every call) also makes the device's primary context current
  // on this thread, which the tensor-map encoder needs; nothing here allocates.
  void* scratch = nullptr;
  rc = static_scratch_address(&scratch);
  if (rc) return rc;
  return run_bwd(p, a, plan, fast, scratch, reinterpret_cast<cudaStream_t>(cuda_stream));
}

int evoattn_last_path(void) { return g_last_path; }
int evoattn_last_launch_count(void) { return g_last_launches; }

}  // extern "C"
