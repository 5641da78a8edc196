// Host side of the C ABI declared in include/sigattn_b200.h: argument checks, TMA tensor
// maps, kernel selection and launches.  No device memory is allocated here.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <algorithm>
#include <atomic>
#include <cmath>
#include <mutex>
#include <stdio.h>
#include <string.h>

#include "../../include/sigattn_b200.h"
#include "bwd_kernel.cuh"
#include "bwd_stream_kernel.cuh"
#include "f32_kernels.cuh"
#include "f32_tc_kernel.cuh"
#include "fwd_kernel.cuh"

namespace {

thread_local char g_err[512] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

#define SIG_CUDA(expr)                                                                            \
  do {                                                                                            \
    cudaError_t e_ = (expr);                                                                      \
    if (e_ != cudaSuccess) return fail(-100, "%s failed: %s", #expr, cudaGetErrorString(e_));     \
  } while (0)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Tensor map over a (B, T, H, D) tensor with element strides {sb, st, sh} and unit stride in
// D.  TMA dimensions are ordered (d, h, t, b); one box is 64 elements of d by `box_rows`
// tokens of one head of one batch, written to shared memory with the 128-byte swizzle.
// Rows at or beyond T read as zeros.
int make_map(CUtensorMap* m, const void* base, int dtype, int B, int T, int H, int D, const int64_t* strides,
             int box_rows, const char* name) {
  // (Encoded on every call: a table of earlier maps, keyed by all that this depends on, took as long to look up - 12.3 us per
  // small forward call either way.)
  EncodeTiledFn enc = get_encode_fn();
  if (!enc) return fail(-101, "cuTensorMapEncodeTiled is not available from this driver");
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return fail(-3, "%s: base pointer must be 16-byte aligned", name);
  for (int i = 0; i < 3; ++i)
    if (strides[i] <= 0 || (strides[i] * 2) % 16 != 0)
      return fail(-3, "%s: stride %d (%lld elements) must be positive and a multiple of 8 elements", name, i,
                  (long long)strides[i]);
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)T, (cuuint64_t)B};
  cuuint64_t gstr[3] = {(cuuint64_t)strides[2] * 2, (cuuint64_t)strides[1] * 2, (cuuint64_t)strides[0] * 2};
  cuuint32_t box[4] = {64, 1, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(m, dtype == SIGATTN_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                   const_cast<void*>(base), dims, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(-102, "%s: cuTensorMapEncodeTiled failed with CUresult %d", name, (int)r);
  return 0;
}

int check_common(const SigAttnParams* p, bool backward) {
  if (!p) return fail(-1, "params is NULL");
  if (p->struct_bytes != sizeof(SigAttnParams))
    return fail(-1, "struct_bytes %u != sizeof(SigAttnParams) %zu (ABI mismatch)", p->struct_bytes,
                sizeof(SigAttnParams));
  if (p->dtype != SIGATTN_FP16 && p->dtype != SIGATTN_BF16 && p->dtype != SIGATTN_FP32)
    return fail(-2, "unsupported dtype %d (fp16=0, bf16=1, fp32=2)", p->dtype);
  if (p->D != 64 && p->D != 128) return fail(-2, "unsupported head dimension %d (64 or 128)", p->D);
  const int per16 = p->dtype == SIGATTN_FP32 ? 4 : 8;
  if (p->head_cols < 0 || p->head_cols > p->D || p->head_cols % per16 != 0)
    return fail(-2, "head_cols %d must be 0 or a multiple of %d up to D = %d", p->head_cols, per16, p->D);
  if (p->B < 0 || p->H < 0 || p->Tq < 0 || p->Tk < 0) return fail(-2, "negative extent");
  if (p->H > 65535 || p->B > 65535) return fail(-2, "B and H must not exceed 65535");
  const bool packed = p->cu_seqlens_q || p->cu_seqlens_k;
  if (packed) {
    if (!p->cu_seqlens_q || !p->cu_seqlens_k) return fail(-1, "packed layout needs both cu_seqlens_q and cu_seqlens_k");
    if (p->seq_lens_q || p->seq_lens_k) return fail(-2, "packed layout: seq_lens_q / seq_lens_k must be NULL");
    if (p->total_q < 0 || p->total_k < 0) return fail(-2, "negative total_q / total_k");
  }
  if (p->B == 0 || p->H == 0) return 1;  // nothing to do
  if (!p->q || !p->k || !p->v) return fail(-1, "q, k, v must not be NULL");
  if (!backward && !p->o) return fail(-1, "o must not be NULL");
  if (backward && (!p->dout || !p->dq || !p->dk || !p->dv)) return fail(-1, "dout, dq, dk, dv must not be NULL");
  return 0;
}

// Columns of the tensors in memory (the kernels' head dimension D is 64 or 128).
int head_cols(const SigAttnParams* p) { return p->head_cols > 0 ? p->head_cols : p->D; }

bool is_contiguous(const int64_t* s, int T, int H, int D) {
  return s[2] == D && s[1] == (int64_t)H * D && s[0] == (int64_t)T * H * D;
}

// Extents of the tensors as the tensor maps, the accumulator and the fills see them: packed tensors are
// one "batch" of total_q / total_k rows.
struct Extents {
  int B, Tq, Tk;
  bool packed;
};
Extents extents(const SigAttnParams* p) {
  const bool packed = p->cu_seqlens_q != nullptr;
  return Extents{packed ? 1 : p->B, packed ? p->total_q : p->Tq, packed ? p->total_k : p->Tk, packed};
}
// {batch, token, head} strides with a usable batch stride when the tensor is packed
struct Strides3 {
  int64_t s[3];
};
Strides3 map_strides(const int64_t* strides, int T, bool packed) {
  Strides3 r{{strides[0], strides[1], strides[2]}};
  if (packed) r.s[0] = (int64_t)(T > 0 ? T : 1) * strides[1];
  return r;
}

// Zero-fill a (B,T,H,D) tensor; only used for degenerate problems (no keys / no queries).
int zero_fill(void* ptr, const int64_t* strides, int B, int T, int H, int D, int dtype, cudaStream_t stream,
              const char* name) {
  if (T == 0) return 0;
  if (!is_contiguous(strides, T, H, D)) return fail(-2, "%s: an empty problem needs a contiguous output", name);
  SIG_CUDA(cudaMemsetAsync(ptr, 0, (size_t)B * T * H * D * (dtype == SIGATTN_FP32 ? 4 : 2), stream));
  return 0;
}

// SIGATTN_ZERO_GAPS: rows of packed outputs that belong to no sequence - before the first one, beyond T within one, behind the
// last one - are zeroed by a kernel that usually finds none, a look at the offsets.  24 causal sequences up to 1500, H=8, D=128,
// forward + backward: 411 -> 368 us without the fills.  (Done by the spare warps of the attention kernels it costs no launch, 361 us, but the
// backward's code moves: a dense causal step of B=8 T=1000 H=16 D=64 took 179 us instead of 174.)
// A warp takes an equal share of the rows, finds the offset behind its first one in a search of 32 ways, and reads on from there
// to its last one.  (With every warp reading all offsets, 4096 sequences of 64 tokens, H=1, D=64: 486 us, 392 so, 390 with fills; 65535 of 8 8400, 5810 and 5900.)
struct GapTensor {
  uint8_t* base;
  int64_t st, sh;  // bytes
};
struct GapSet {  // the tensors that have the same rows
  GapTensor t[2];
  const int* cu;
  int n, T, total;
};
struct GapParams {
  GapSet set[2];
  int B, H, chunks;  // 16-byte pieces of a row of one head
};
constexpr int kGapThreads = 256;
__global__ void __launch_bounds__(kGapThreads) sigattn_zero_gaps_kernel(const GapParams p) {
  const GapSet& s = p.set[blockIdx.y];
  const int lane = threadIdx.x & 31, worker = (int)(blockIdx.x * kGapThreads + threadIdx.x) >> 5;
  const int64_t workers = gridDim.x * (kGapThreads / 32), share = (s.total + workers - 1) / workers;
  const int64_t row0 = worker * share, row1 = min(row0 + share, (int64_t)s.total);
  if (row0 >= row1) return;
  // g = the first sequence that begins behind row0 (B: none)
  int g = 0;
  for (int end = p.B; g < end;) {
    const int step = (end - g + 31) / 32, last = g + lane * step + step - 1;
    const int below = __popc(__ballot_sync(0xffffffffu, last < end && s.cu[min(last, p.B)] <= row0));
    g = min(g + below * step, end);
    end = step == 1 ? g : min(g + step, end);
  }
  for (; g <= p.B; g += 32) {
    const int at = g + lane;  // the gap in front of this sequence
    int64_t lo = 0, hi = 0;
    if (at <= p.B) {
      if (at > 0) lo = s.cu[at - 1] + min(max(s.cu[at] - s.cu[at - 1], 0), s.T);
      hi = at < p.B ? s.cu[at] : s.total;
    }
    const bool beyond = lo >= row1 || at >= p.B;  // no gap behind this one reaches into the share
    lo = max(lo, row0);
    hi = min(hi, row1);
    for (unsigned int m = __ballot_sync(0xffffffffu, lo < hi); m; m &= m - 1) {
      const int src = __ffs(m) - 1;
      const int64_t first = __shfl_sync(0xffffffffu, lo, src), rows = __shfl_sync(0xffffffffu, hi, src) - first;
      // lanes side by side along a row, several rows at a time where it is shorter than 32 pieces
      const int pieces = p.H * p.chunks, at_once = pieces >= 32 ? 1 : 32 / pieces;
      const int r = pieces >= 32 ? 0 : lane / pieces;
      if (r < at_once)
        for (int c = pieces >= 32 ? lane : lane % pieces; c < pieces; c += 32) {
          const int h = c / p.chunks, i = c - h * p.chunks;
          for (int k = 0; k < s.n; ++k) {
            const int64_t step = at_once * s.t[k].st;
            uint8_t* dst = s.t[k].base + (first + r) * s.t[k].st + h * s.t[k].sh + 16 * i;
#pragma unroll 4
            for (int64_t n = r; n < rows; n += at_once, dst += step) *reinterpret_cast<uint4*>(dst) = make_uint4(0, 0, 0, 0);
          }
        }
    }
    if (__any_sync(0xffffffffu, beyond)) break;
  }
}
int zero_gaps(const SigAttnParams* p, bool backward, int n_sm) {
  if (!(p->flags & SIGATTN_ZERO_GAPS) || !p->cu_seqlens_q) return 0;
  const int es = p->dtype == SIGATTN_FP32 ? 4 : 2;
  void* ptr[3] = {backward ? p->dq : p->o, p->dk, p->dv};
  const int64_t* strides[3] = {backward ? p->dq_strides : p->o_strides, p->dk_strides, p->dv_strides};
  GapParams gp = {};
  gp.B = p->B;
  gp.H = p->H;
  gp.chunks = head_cols(p) * es / 16;
  gp.set[0].cu = p->cu_seqlens_q;
  gp.set[0].n = 1;
  gp.set[0].T = p->Tq;
  gp.set[0].total = p->total_q;
  gp.set[1].cu = p->cu_seqlens_k;
  gp.set[1].n = 2;
  gp.set[1].T = p->Tk;
  gp.set[1].total = p->total_k;
  for (int k = 0; k < (backward ? 3 : 1); ++k) {
    if ((reinterpret_cast<uintptr_t>(ptr[k]) & 15u) != 0 || strides[k][1] * es % 16 != 0 || strides[k][2] * es % 16 != 0)
      return fail(-3, "SIGATTN_ZERO_GAPS: outputs and their strides must be 16-byte aligned");
    (k ? gp.set[1].t[k - 1] : gp.set[0].t[0]) = GapTensor{static_cast<uint8_t*>(ptr[k]), strides[k][1] * es, strides[k][2] * es};
  }
  sigattn_zero_gaps_kernel<<<dim3((unsigned int)n_sm, backward ? 2u : 1u), kGapThreads, 0, static_cast<cudaStream_t>(p->stream)>>>(gp);
  SIG_CUDA(cudaGetLastError());
  return 0;
}

struct DeviceGuard {
  int prev = -1;
  bool switched = false;
  cudaError_t enter(int dev) {
    cudaError_t e = cudaGetDevice(&prev);
    if (e != cudaSuccess) return e;
    // Always set the device: on a host thread that has made no runtime call yet (an autograd
    // worker, say) this is what binds the primary context, which the driver-level tensor-map
    // encoder needs.
    e = cudaSetDevice(dev);
    switched = (e == cudaSuccess) && prev != dev;
    return e;
  }
  ~DeviceGuard() {
    if (switched) cudaSetDevice(prev);
  }
};

// Opt-in to the kernel's dynamic shared memory: once per kernel and device (`K` is a distinct type per
// kernel signature only, so the flags are keyed by the kernel's address).
template <typename K>
int set_smem(K kernel, int bytes, int device) {
  constexpr int kMaxKernels = 64, kMaxDevices = 64;
  static std::mutex mu;
  static const void* seen[kMaxKernels] = {};
  static bool done[kMaxKernels][kMaxDevices] = {};
  if (device >= 0 && device < kMaxDevices) {
    std::lock_guard<std::mutex> lock(mu);
    for (int i = 0; i < kMaxKernels; ++i) {
      if (seen[i] == nullptr) seen[i] = reinterpret_cast<const void*>(kernel);
      if (seen[i] == reinterpret_cast<const void*>(kernel)) {
        if (done[i][device]) return 0;
        SIG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        done[i][device] = true;
        return 0;
      }
    }
  }
  SIG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return 0;
}

// Work-item counters of the persistent kernels (forward and backward): a ring of (next item, finished CTAs) pairs.
// Each launch takes the next pair; the kernel leaves its pair at zero when its last CTA finishes,
// so a pair is only in doubt if more launches than the pool holds are in flight at once on one device.
// Launches recorded into a stream capture keep their pair for every replay of the graph, so they draw
// from a pool of their own that eager launches never touch.
constexpr int kTicketSlots = 1024;
constexpr int kEagerTicketSlots = 768;  // the remaining 256 serve launches made under stream capture
__device__ unsigned int g_item_tickets[2 * kTicketSlots];

// Host-visible copies of the devices' health words (see g_status_mirror in ptx.cuh): one page of this
// library's own host data, pinned and mapped once per process.  A kernel writes its device's entry
// only when it abandons a wait; every attention call reads it (a plain host load) before launching.
constexpr int kMaxMirrorDevices = 64;
alignas(4096) volatile int g_host_status[1024];
bool g_host_status_mapped = false;

struct FwdDeviceInfo {
  unsigned int* tickets = nullptr;
  int n_sm = 0;
};

// Device address of the counters and the SM count, looked up once per device (which must be current).
int fwd_device_info(int device, FwdDeviceInfo* out) {
  constexpr int kMaxDevices = 64;
  static FwdDeviceInfo cached[kMaxDevices];
  static std::mutex mu;
  if (device < 0 || device >= kMaxDevices) return fail(-2, "device ordinal %d out of range", device);
  std::lock_guard<std::mutex> lock(mu);
  if (!cached[device].tickets) {
    unsigned int* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_item_tickets);
    if (e != cudaSuccess || !ptr)
      return fail(-100, "cudaGetSymbolAddress(work-item counters) failed on device %d: %s", device,
                  cudaGetErrorString(e));
    int n_sm = 0;
    SIG_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device));
    if (n_sm <= 0) return fail(-100, "device %d reports %d multiprocessors", device, n_sm);
    // health-word mirror: best effort (without it failures are still reported by sigattn_device_status)
    if (!g_host_status_mapped) {
      if (cudaHostRegister(const_cast<int*>(g_host_status), sizeof(g_host_status),
                           cudaHostRegisterPortable | cudaHostRegisterMapped) == cudaSuccess)
        g_host_status_mapped = true;
      else
        (void)cudaGetLastError();
    }
    if (g_host_status_mapped && device < kMaxMirrorDevices) {
      int* dev_view = nullptr;
      if (cudaHostGetDevicePointer(reinterpret_cast<void**>(&dev_view), const_cast<int*>(&g_host_status[device]), 0) ==
              cudaSuccess && dev_view) {
        volatile int* as_volatile = dev_view;
        if (cudaMemcpyToSymbol(sigattn::g_status_mirror, &as_volatile, sizeof(as_volatile)) != cudaSuccess)
          (void)cudaGetLastError();
      } else {
        (void)cudaGetLastError();
      }
    }
    cached[device].n_sm = n_sm;
    cached[device].tickets = ptr;
  }
  *out = cached[device];
  return 0;
}

// Non-zero when a kernel of this library has abandoned a wait on `device` and nobody has read the
// failure yet (sigattn_device_status reads and clears it).
int pending_failure(int device) {
  if (device < 0 || device >= kMaxMirrorDevices) return 0;
  return g_host_status[device];
}
#define SIG_REFUSE_IF_SICK(p)                                                                               \
  do {                                                                                                      \
    if (int site_ = pending_failure((p)->device))                                                           \
      return fail(-5, "device %d: a kernel gave up on a bounded wait (site 0x%x); results since then are "  \
                      "undefined and launches are refused until sigattn_device_status() has been called",   \
                  (p)->device, site_);                                                                      \
  } while (0)

// (batch, head) pairs per scheduling group of the persistent kernels.  Under a causal mask the items of
// one head differ in weight, and handing out the heavy items of many heads first balances the CTAs; the
// group is limited so that what its heads stream per item (`bytes_per_head`) stays within the L2.
// Without a causal mask the plain order is kept.
int schedule_group(bool causal, int64_t n_bh, int64_t bytes_per_head, int64_t l2_budget) {
  if (!causal || n_bh <= 1) return 1;
  int64_t g = l2_budget / (bytes_per_head > 0 ? bytes_per_head : 1);
  if (g < 1) g = 1;
  if (g > n_bh) g = n_bh;
  return (int)g;
}

// The pair of counters for one launch on `stream`.
unsigned int* next_ticket_pair(const FwdDeviceInfo& info, int device, cudaStream_t stream) {
  static std::atomic<unsigned int> next_eager[64], next_captured[64];
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &st) != cudaSuccess) {
    (void)cudaGetLastError();
    st = cudaStreamCaptureStatusNone;
  }
  if (st == cudaStreamCaptureStatusNone) return info.tickets + 2 * (next_eager[device].fetch_add(1u) % kEagerTicketSlots);
  return info.tickets + 2 * (kEagerTicketSlots + next_captured[device].fetch_add(1u) % (kTicketSlots - kEagerTicketSlots));
}

// How the forward divides its work: the persistent form, or, with fewer items than half of the SMs, the split one with clusters of `split`
// CTAs per item; the latter, in one part, also for items of up to 64 queries, if they are few or surely have many keys.
// The key range of each is split, as long as every part keeps two key tiles (a part
// of one costs as much in the cluster's hand-over as it saves) and the clusters still find room at once (they must lie
// within a GPC, whose SM counts are not all multiples of 8: 7/8 of the SMs are counted on).
// B=8 H=8, 64 queries on 1024 .. 4096 keys: 47 -> 29 us; B=1 T=4096 H=2, D = 64 61 -> 33, D = 128 74 -> 37; B=1 T=1024 H=4
// 24.6 -> 20.5; with two parts of two tiles, B=1 T=512 H=4, 20 -> 18.4; unchanged beyond 64 items, B=1 T=8192 H=4.
// At D = 64 with items of 128 rows, whose key tiles the two groups of sigmoid warps take alternately, there are twice as many to split, and up
// to 64 queries fill both halves of a tile (FwdParams::twice): 64 queries as above with a per-key term 26.9 -> 20.7 us, without 23.4 -> 18.7, B=1
// 14.5 -> 12.5; one query on 4096 keys 22.7 -> 18.7.  Frames filled to a third or a twentieth are no slower than with 256 rows: 1.00 - 1.19.
// In one part, its CTAs are not persistent, and every item pays for a set-up that the persistent form overlaps.  Many items therefore need 16 key
// tiles each that are sure to be there: persistent -> one part, us, dense, 512 items of 64 queries on 4096 keys 145 -> 113, 160 on 2048 45 -> 35, 2048
// of one query on 2048 250 -> 232 and on 4096 495 -> 383.  Padded batches, whose lengths the host does not know, stay persistent: 512
// items, frame 4096, full 120 -> 94, filled to a third 52 -> 54, to a twentieth 27 -> 37; 2048 of one query 79 -> 120.
// Few items with too few key tiles to split have 128 rows in the persistent form too: B=2 T=256 H=4 D = 64 10.6 -> 10.1 us, T=384 12.5 -> 10.4,
// D = 128 12.6 -> 10.5, B=16 T=200 12.5 -> 10.4; B=9 T=130 H=8 D = 128 16.6 -> 14.5.
int64_t fwd_items(const SigAttnParams* p, int rows) { return (int64_t)((p->Tq + rows - 1) / rows) * p->H * p->B; }
struct FwdPlan {
  int block_m = sigattn::kFwdBlockM;  // query rows per item
  int split = 0;                      // 0: persistent
  bool twice = false;
};
FwdPlan fwd_plan(const SigAttnParams* p, int n_sm) {
  const int tiles = (p->Tk + sigattn::kTileN - 1) / sigattn::kTileN;
  auto parts = [&](int64_t n_items) {
    int split = 1;
    while (split < 8 && n_items * split * 2 <= n_sm * 7 / 8 && tiles >= 4 * split) split *= 2;
    return split;
  };
  FwdPlan plan;
  const int64_t narrow = fwd_items(p, 128);
  const int split = parts(fwd_items(p, sigattn::kFwdBlockM));
  if (split > 1) plan.split = split;
  // key tiles that an item of up to 64 queries surely has (on average, packed)
  const int sure = p->seq_lens_q || p->seq_lens_k || (p->flags & SIGATTN_CAUSAL) ? 0 : p->cu_seqlens_k ? p->total_k / std::max(p->B, 1) / sigattn::kTileN : tiles;
  if (p->D == 64 && ((narrow <= n_sm && parts(narrow) > 1) || (split == 1 && p->Tq <= 64 && (narrow <= n_sm || sure >= 16)))) {
    plan.block_m = 128;
    plan.split = parts(narrow);
    plan.twice = p->Tq <= 64;
  } else if (split == 1 && narrow <= n_sm) {
    plan.block_m = 128;
  }
  return plan;
}

// Which logits below zero the 16-bit kernels test for (all 1024 of a warp's chunk; see sigmoid2_near), and when.
//  - with a bias of the caller's, the same for the whole batch and above -3, scores would have to be below zero throughout to pass:
//    kDeepWatched tests only while chunks pass.  bf16, bias 0, B=4 T=4096, a test for every chunk -> while it pays, us, forward (H=32 D=64,
//    H=16 D=128) and with the backward: scores of both signs 924 -> 740 and 2560 -> 2340, 582 -> 545 and 1904 -> 1880; about -8, which
//    trained weights may well have, 755 -> 778 and 2260 -> 2310, 507 -> 520 and 1870 -> 1880; about -8 with every 512th key at 0 745 -> 790.
//    (Never tested 725 and 2290, 810 and 2430, and probabilities that are all too small by what the polynomial lacks at 0, see rcp1p_poly.)
//    The far range: what passes is usually far below zero, and the series on packed pairs is shorter (logits about -8, forward, near instead 693 -> 738,
//    D = 128 504 -> 536; fp16 769 -> 786, 543 -> 563).
//  - D = 64, up to 1024 keys: kDeepNear, which scores of deviation 1 pass under the default bias, where kDeepFar, which is two operations
//    shorter per pair, sends them on to the polynomial for all logits.  Far -> near, us, H=16: forward bf16 512 x 512 960 -> 844, 256 x 256
//    158 -> 145, 32 x 1024 214 -> 214, 16 x 2048 380 -> 405; fp16 128 x 512 266 -> 230, 32 x 1000 234 -> 219, 4 x 4096 382 -> 393; backward
//    512 x 512 2345 -> 2286, 32 x 1000 650 -> 600, 32 x 1024 520 -> 518, 16 x 2048 926 -> 933.  The errors are smaller than before: T=512 bf16, dV
//    2.63e-3 -> 2.36e-3, dQ 3.88e-3 -> 3.72e-3; fp16 3.4e-4 -> 3.0e-4, 4.9e-4 -> 4.6e-4.
//    Scores that pass the far test as well, whose chunks are two operations longer now, cost the forward 4 to 5 %, for the smaller errors: H=16,
//    scores of deviation 0.25, bf16 256 x 512 427 -> 448, 512 x 256 265 -> 270, 64 x 1024 395 -> 411; fp16 452 -> 468, 281 -> 293, 430 -> 445; backward
//    up to 1 % (bf16) or nothing.
//    (By the keys and not by the bias, which some callers pass as an array: the result is the same either way.)  At D = 128 the forward does
//    not gain (scores of deviation 0.25, T=512 175 -> 183), and the backward, like the deterministic one, would lose precision.
constexpr int kNearKeys = 1024;
sigattn::DeepForm deep_form(const SigAttnParams* p) {
  if (!p->bias && !p->score_mod && !(p->flags & (SIGATTN_ACCURATE | SIGATTN_BIAS_NEG_LOG_LK)) && p->bias_scalar > -3.0f)
    return sigattn::kDeepWatched;
  return p->D == 64 && p->Tk <= kNearKeys && !(p->flags & SIGATTN_ACCURATE) ? sigattn::kDeepNear : sigattn::kDeepFar;
}

template <int D, bool kBF16, bool kScoreMod, bool kAccurate>
int launch_fwd(const SigAttnParams* p, const CUtensorMap& qm, const CUtensorMap& km, const CUtensorMap& vm) {
  using namespace sigattn;
  constexpr int smem = FwdSmem<D>::kDynBytes;
  FwdParams fp;
  fp.o = p->o;
  fp.o_sb = p->o_strides[0];
  fp.o_st = p->o_strides[1];
  fp.o_sh = p->o_strides[2];
  fp.lens_q = p->seq_lens_q;
  fp.lens_k = p->seq_lens_k;
  fp.cu_q = p->cu_seqlens_q;
  fp.cu_k = p->cu_seqlens_k;
  fp.bias = p->bias;
  fp.score_mod = p->score_mod;
  fp.scale = p->scale;
  fp.bias_scalar = p->bias_scalar;
  if (p->flags & SIGATTN_BIAS_NEG_LOG_LK) { fp.bias = nullptr; fp.bias_scalar = nanf(""); }  // see item_bias()
  fp.B = p->B;
  fp.H = p->H;
  fp.Tq = p->Tq;
  fp.Tk = p->Tk;
  fp.d_cols = head_cols(p);
  fp.causal = (p->flags & SIGATTN_CAUSAL) ? 1 : 0;
  FwdDeviceInfo info;
  if (int rc = fwd_device_info(p->device, &info)) return rc;
  const FwdPlan plan = fwd_plan(p, info.n_sm);
  fp.split = plan.split;
  fp.block_m = plan.block_m;
  fp.twice = plan.twice ? 1 : 0;
  fp.n_qblk = (p->Tq + plan.block_m - 1) / plan.block_m;
  const int64_t n_items = fwd_items(p, plan.block_m);
  if (n_items > INT32_MAX) return fail(-2, "too many (batch, head, query block) items: %lld", (long long)n_items);
  fp.n_items = (int)n_items;
  // K and V of one head, half of the L2 for them
  fp.group = schedule_group(fp.causal != 0, (int64_t)p->B * p->H, (int64_t)p->Tk * D * 2 * 2, 64ll << 20);
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  if (int rc = zero_gaps(p, false, info.n_sm)) return rc;
  if (fp.split) {
    auto pick = [&]() {
      if constexpr (D == 64 && !kAccurate)
        if (p->Tk <= kNearKeys) return sigattn_fwd_kernel<D, kBF16, kScoreMod, false, true, kDeepNear>;
      return sigattn_fwd_kernel<D, kBF16, kScoreMod, kAccurate, true, kDeepFar>;
    };
    auto kernel = pick();
    if (int rc = set_smem(kernel, smem, p->device)) return rc;
    fp.ticket = nullptr;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned int)fp.split;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned int)(n_items * fp.split));
    cfg.blockDim = dim3(kFwdThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (p->ev_main_start) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_start), stream));
    SIG_CUDA(cudaLaunchKernelEx(&cfg, kernel, qm, km, vm, fp));
  } else {
    auto pick = [&]() {
      if constexpr (!kScoreMod && !kAccurate)
        if (deep_form(p) == kDeepWatched) return sigattn_fwd_kernel<D, kBF16, false, false, false, kDeepWatched>;
      if constexpr (D == 64 && !kAccurate)
        if (deep_form(p) == kDeepNear) return sigattn_fwd_kernel<D, kBF16, kScoreMod, false, false, kDeepNear>;
      return sigattn_fwd_kernel<D, kBF16, kScoreMod, kAccurate, false, kDeepFar>;
    };
    auto kernel = pick();
    if (int rc = set_smem(kernel, smem, p->device)) return rc;
    fp.ticket = n_items > info.n_sm ? next_ticket_pair(info, p->device, stream) : nullptr;  // (more items than CTAs)
    // persistent: one CTA per SM (the kernel's shared memory allows no more), fewer when there are fewer items
    dim3 grid((unsigned int)std::min<int64_t>(n_items, info.n_sm));
    if (p->ev_main_start) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_start), stream));
    kernel<<<grid, kFwdThreads, smem, stream>>>(qm, km, vm, fp);
    SIG_CUDA(cudaGetLastError());
  }
  if (p->ev_main_stop) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_stop), stream));
  return 0;
}

// Whether the fused backward gives whole (batch element, head) pairs to CTAs (see kByHead).  The general form fills, reduces
// into, reads and converts an accumulator of 4 bytes per element of Q, passes over memory that this one saves; but its items
// are single key tiles, which balance better, while here the launch ends on somebody's last pair.  So the pairs must be many
// (8 per SM: B=80 T=512 H=16 562 -> 545 us forward + backward) and short.  The lines below are from 22,000 random calls (8 to
// 45 pairs per SM, dense, padded and packed) with both forms forced; figures are the backward alone in this form over the
// general one, means of a class.  By this rule the form is 0.915 of the general one where it is taken and 1.031 where not.
//  - Tq, as the passes' share falls with it and the CTAs' regions outgrow the L2.  D = 64, dense: 0.75 - 0.83 at 129 to 256, 0.84 -
//    0.91 up to 512, 0.75 - 0.97 up to 768, 0.87 - 1.00 up to 1000, 1.06 - 1.16 at 1024 - the high ends at multiples of 128, for which
//    the line is drawn; causal 0.85 - 0.91 up to 1200, 0.94 - 0.97 up to 1536 (there 1.03 - 1.06).  D = 128, half as long: 0.73 - 0.90
//    up to 384, 0.94 up to 500, 0.95 - 1.03 at 512; causal 0.73 - 0.95 up to 768.
//  - Tk, as the gain falls with a pair's number of key tiles and the end's share with the pairs per SM: four tiles, or as many as
//    query tiles, or as many as there are pairs per SM - half as many at D = 128 (0.94 - 1.02 below that, 1.01 - 1.07 above), twice
//    as many at D = 64 with more than one query tile (0.88 - 0.99, 0.97 - 1.04; one query tile 0.96 - 1.00, 1.00 - 1.02).
//    Extremes: Tq=64 on 2048 keys 695 -> 757 us, 256 on 8192 2702 -> 3149, 211 on 2088 2604 -> 1916.  Causal, keys behind the last
//    query have no work (Tq=512 Tk=1024 0.87), but tiles of them pass one after another: D = 64, one query tile, 1.02 - 1.13.
//  - packed sequences, on average: a CTA's share of the rows is at least 2.5 of the longest sequence (with 8 pairs per SM, an
//    average of 0.3 of it; the general form's passes only cover the rows there are).  Some of 768 tokens among many of 128
//    1.12 - 1.21, of 192 1.02 - 1.05, of 256 0.92 - 1.07; of 512 tokens 1.01 - 1.13, 0.95 - 1.09, 0.91 - 0.98.  This also covers that
//    the accumulator must have room for a region per CTA.  (Padded, 768 among 96: 0.71 - 0.89.)
// Both forms have become faster since, the general one more so at D = 64.  Forced again (bf16, by head over general; 640 to 4800 pairs, equal lengths or packed):
//  - Tq, D = 64: 0.82 - 0.89 up to 256, 0.88 - 0.99 up to 512, 0.91 at 700, 1.03 at 768, 0.99 - 1.04 at 900 and 1000, 1.10 - 1.15 at 1024; causal 0.87 - 0.97 up to
//    1200, 1.01 at 1500.  D = 128: 0.60 - 0.87 up to 256, 0.98 at 384, 1.06 - 1.10 at 448 to 512, causal 0.88 at 512, 1.13 at 1000.
//  - Tk, D = 64: 64 queries 0.97 / 1.03 / 1.06 - 1.07 / 1.08 - 1.10 with 2 / 4 / 8 / 16 key tiles, 256 queries 0.94 / 1.01 - 1.02 / 1.07 - 1.09 with 4 / 8 / 16; the rule still takes
//    some of the slower ones.  D = 128: 0.88 / 0.95 / 1.00 - 1.03 / 1.04 - 1.06 and 0.93 / 1.00 / 1.03 - 1.04.  Causal, 128 queries on 512 keys 0.96 and 0.77.
//  - packed, D = 64 0.83 - 0.92; D = 128 0.81 - 0.93 up to 384, causal 0.83 - 0.88 at 512; at 512 and 700 (not taken) 1.01 - 1.06.
// The accurate sigmoid, an option for comparisons, has the general form only.
bool bwd_by_head(const SigAttnParams* p, int n_sm) {
  const bool causal = (p->flags & SIGATTN_CAUSAL) != 0, wide = p->D == 128;
  const Extents ex = extents(p);
  const int64_t n_bh = (int64_t)p->B * p->H, acc_rows = (int64_t)ex.B * ex.Tq * p->H;
  const int64_t q_tiles = ((int64_t)p->Tq + 127) / 128, k_tiles = ((int64_t)p->Tk + 127) / 128;
  const int64_t busy = causal ? std::min(k_tiles, q_tiles) : k_tiles;  // key tiles with work
  if ((p->flags & SIGATTN_ACCURATE) || n_bh < 8 * (int64_t)n_sm || (int64_t)p->Tq * p->D > (causal ? 98304 : 49152)) return false;
  if (busy > 4 && busy > q_tiles && 2 * busy * n_sm > n_bh * (wide ? 1 : q_tiles > 1 ? 4 : 2)) return false;
  if (causal && !wide && q_tiles == 1 && k_tiles > 2) return false;
  return 2 * acc_rows >= 5 * (int64_t)n_sm * p->Tq;
}

// The default backward: the fused 5-GEMM kernel with fp32 dQ reductions into a workspace (bwd_kernel.cuh).
template <int D, bool kBF16, bool kAccurate>
int launch_bwd_fused(const SigAttnParams* p, const CUtensorMap& qm, const CUtensorMap& km, const CUtensorMap& vm,
                     const CUtensorMap& dom) {
  using namespace sigattn;
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  const Extents ex = extents(p);
  const size_t need = sigattn_bwd_workspace_bytes(ex.B, ex.Tq, p->H, p->D);
  if (p->workspace_bytes < need || (need && !p->workspace))
    return fail(-4, "backward workspace too small: %zu bytes given, %zu needed", p->workspace_bytes, need);
  if ((reinterpret_cast<uintptr_t>(p->workspace) & 15u) != 0) return fail(-3, "workspace must be 16-byte aligned");
  float* dq_acc = static_cast<float*>(p->workspace);
  FwdDeviceInfo info;
  if (int rc = fwd_device_info(p->device, &info)) return rc;
  const int64_t n_bh = (int64_t)p->B * p->H;
  const bool by_head = bwd_by_head(p, info.n_sm);
  const int64_t q_tiles = n_bh * ((p->Tq + 127) / 128);
  if (!by_head && q_tiles > INT32_MAX) return fail(-2, "too many (batch, head, query tile) items: %lld", (long long)q_tiles);
  if (!by_head && p->seq_lens_q) {
    sigattn_dq_fill_kernel<D><<<(unsigned int)q_tiles, 256, 0, stream>>>(dq_acc, p->seq_lens_q, (p->Tq + 127) / 128, p->Tq, p->H);
    SIG_CUDA(cudaGetLastError());
  } else if (!by_head) {
    SIG_CUDA(cudaMemsetAsync(dq_acc, 0, need, stream));
  }

  BwdParams bp;
  bp.dq_acc = dq_acc;
  bp.acc_sh = (int64_t)(by_head ? p->Tq : ex.Tq) * D;
  bp.acc_sb = (int64_t)p->H * bp.acc_sh;
  bp.dq = p->dq;
  bp.dq_sb = p->dq_strides[0]; bp.dq_st = p->dq_strides[1]; bp.dq_sh = p->dq_strides[2];
  bp.dk = p->dk;
  bp.dv = p->dv;
  bp.dk_sb = p->dk_strides[0]; bp.dk_st = p->dk_strides[1]; bp.dk_sh = p->dk_strides[2];
  bp.dv_sb = p->dv_strides[0]; bp.dv_st = p->dv_strides[1]; bp.dv_sh = p->dv_strides[2];
  bp.lens_q = p->seq_lens_q;
  bp.lens_k = p->seq_lens_k;
  bp.cu_q = p->cu_seqlens_q;
  bp.cu_k = p->cu_seqlens_k;
  bp.bias = p->bias;
  bp.score_mod = p->score_mod;
  bp.scale = p->scale;
  bp.bias_scalar = p->bias_scalar;
  if (p->flags & SIGATTN_BIAS_NEG_LOG_LK) { bp.bias = nullptr; bp.bias_scalar = nanf(""); }  // see item_bias()
  bp.B = p->B; bp.H = p->H; bp.Tq = p->Tq; bp.Tk = p->Tk;
  bp.d_cols = head_cols(p);
  bp.causal = (p->flags & SIGATTN_CAUSAL) ? 1 : 0;
  bp.n_kvblk = (p->Tk + kBwdTileKV - 1) / kBwdTileKV;
  const int64_t n_items = (int64_t)bp.n_kvblk * p->H * p->B;
  if (n_items > INT32_MAX) return fail(-2, "too many (batch, head, key tile) items: %lld", (long long)n_items);
  bp.n_items = (int)n_items;
  // Q, dO and the fp32 dQ accumulator of one head; a quarter of the L2 (measured: larger groups cost the
  // reductions their locality, a few heads already balance the CTAs)
  bp.group = by_head ? 1 : schedule_group(bp.causal != 0, n_bh, (int64_t)p->Tq * D * (2 + 2 + 4), 32ll << 20);
  if (int rc = zero_gaps(p, true, info.n_sm)) return rc;
  bp.ticket = (by_head ? n_bh : n_items) > info.n_sm ? next_ticket_pair(info, p->device, stream) : nullptr;  // (more items than CTAs)

  {
    // (the accurate sigmoid has one form, and D = 128 one range)
    auto pick = [&]() {
      if constexpr (!kAccurate) {
        if (deep_form(p) == kDeepWatched) return by_head ? sigattn_bwd_kernel<D, kBF16, false, true, kDeepWatched> : sigattn_bwd_kernel<D, kBF16, false, false, kDeepWatched>;
        if constexpr (D == 64)
          if (deep_form(p) == kDeepNear) return by_head ? sigattn_bwd_kernel<D, kBF16, false, true, kDeepNear> : sigattn_bwd_kernel<D, kBF16, false, false, kDeepNear>;
        if (by_head) return sigattn_bwd_kernel<D, kBF16, false, true, kDeepFar>;
      }
      return sigattn_bwd_kernel<D, kBF16, kAccurate, false, kDeepFar>;
    };
    auto kernel = pick();
    constexpr int smem = BwdSmem<D>::kDynBytes;
    if (int rc = set_smem(kernel, smem, p->device)) return rc;
    // persistent: one CTA per SM (the kernel's shared memory allows no more), fewer when there are fewer items
    dim3 grid((unsigned int)std::min<int64_t>(by_head ? n_bh : n_items, info.n_sm));
    if (p->ev_main_start) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_start), stream));
    kernel<<<grid, kBwdThreads, smem, stream>>>(qm, km, vm, dom, bp);
    SIG_CUDA(cudaGetLastError());
    if (p->ev_main_stop) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_stop), stream));
  }
  if (!by_head) {
    // dQ = scale * accumulator, rounded to the 16-bit type
    DqConvertParams cp;
    cp.acc = dq_acc;
    cp.acc_sb = bp.acc_sb; cp.acc_sh = bp.acc_sh;
    cp.dq = p->dq;
    cp.sb = p->dq_strides[0]; cp.st = p->dq_strides[1]; cp.sh = p->dq_strides[2];
    cp.lens_q = p->seq_lens_q;
    cp.cu_q = p->cu_seqlens_q;
    cp.n_tiles = (p->Tq + 127) / 128; cp.T = p->Tq; cp.H = p->H;
    cp.d_cols = head_cols(p);
    cp.scale = p->scale;
    sigattn_dq_convert_kernel<D, kBF16><<<(unsigned int)q_tiles, 256, 0, stream>>>(cp);
    SIG_CUDA(cudaGetLastError());
  }
  return 0;
}

// The split backward (SIGATTN_BWD_SPLIT): the streaming kernel of bwd_stream_kernel.cuh, once in dK/dV mode
// and once in dQ mode.  No workspace, no atomics, deterministic.
template <int D, bool kBF16, bool kDKV, bool kAccurate>
int launch_bwd_stream_mode(const SigAttnParams* p, const CUtensorMap& r1, const CUtensorMap& r2, const CUtensorMap& c1,
                           const CUtensorMap& c2, const FwdDeviceInfo& info) {
  using namespace sigattn;
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  BwdStreamParams bp;
  if (kDKV) {
    bp.out1 = p->dk; bp.o1_sb = p->dk_strides[0]; bp.o1_st = p->dk_strides[1]; bp.o1_sh = p->dk_strides[2];
    bp.out2 = p->dv; bp.o2_sb = p->dv_strides[0]; bp.o2_st = p->dv_strides[1]; bp.o2_sh = p->dv_strides[2];
    bp.lens_r = p->seq_lens_k; bp.lens_c = p->seq_lens_q;
    bp.cu_r = p->cu_seqlens_k; bp.cu_c = p->cu_seqlens_q;
    bp.Tr = p->Tk; bp.Tc = p->Tq;
  } else {
    bp.out1 = p->dq; bp.o1_sb = p->dq_strides[0]; bp.o1_st = p->dq_strides[1]; bp.o1_sh = p->dq_strides[2];
    bp.out2 = nullptr; bp.o2_sb = bp.o2_st = bp.o2_sh = 0;
    bp.lens_r = p->seq_lens_q; bp.lens_c = p->seq_lens_k;
    bp.cu_r = p->cu_seqlens_q; bp.cu_c = p->cu_seqlens_k;
    bp.Tr = p->Tq; bp.Tc = p->Tk;
  }
  bp.bias = p->bias;
  bp.score_mod = p->score_mod;
  bp.scale = p->scale;
  bp.bias_scalar = p->bias_scalar;
  if (p->flags & SIGATTN_BIAS_NEG_LOG_LK) { bp.bias = nullptr; bp.bias_scalar = nanf(""); }  // see item_bias()
  bp.B = p->B; bp.H = p->H; bp.Tk = p->Tk;
  bp.d_cols = head_cols(p);
  bp.causal = (p->flags & SIGATTN_CAUSAL) ? 1 : 0;
  bp.n_rblk = (bp.Tr + kBsTile - 1) / kBsTile;
  const int64_t n_items = (int64_t)bp.n_rblk * p->H * p->B;
  if (n_items > INT32_MAX) return fail(-2, "too many (batch, head, tile) items: %lld", (long long)n_items);
  bp.n_items = (int)n_items;
  // what one head streams per item (the two streamed tensors), half of the L2 for a group
  bp.group = schedule_group(bp.causal != 0, (int64_t)p->B * p->H, (int64_t)bp.Tc * D * 2 * 2, 64ll << 20);
  bp.ticket = next_ticket_pair(info, p->device, stream);
  auto kernel = sigattn_bwd_stream_kernel<D, kBF16, kDKV, kAccurate>;
  constexpr int smem = BsSmem<D, kDKV>::kDynBytes;
  if (int rc = set_smem(kernel, smem, p->device)) return rc;
  dim3 grid((unsigned int)std::min<int64_t>(n_items, info.n_sm));
  kernel<<<grid, kBsThreads, smem, stream>>>(r1, r2, c1, c2, bp);
  SIG_CUDA(cudaGetLastError());
  return 0;
}

template <int D, bool kBF16, bool kAccurate>
int launch_bwd_stream(const SigAttnParams* p, const CUtensorMap& qm, const CUtensorMap& km, const CUtensorMap& vm,
                      const CUtensorMap& dom) {
  FwdDeviceInfo info;
  if (int rc = fwd_device_info(p->device, &info)) return rc;
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  if (int rc = zero_gaps(p, true, info.n_sm)) return rc;
  if (p->ev_main_start) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_start), stream));
  if (int rc = launch_bwd_stream_mode<D, kBF16, true, kAccurate>(p, km, vm, qm, dom, info)) return rc;
  if (int rc = launch_bwd_stream_mode<D, kBF16, false, kAccurate>(p, qm, dom, km, vm, info)) return rc;
  if (p->ev_main_stop) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_stop), stream));
  return 0;
}

// Scratch of sigattn_bwd_static_scratch: lives in the device image of this library.
static __device__ __align__(256) float g_static_dq_scratch[SIGATTN_STATIC_SCRATCH_ELEMS];

// In host code the name above is only a handle for the runtime, not a device address; the
// address valid on `device` is looked up once per device (with that device current) and cached.
int static_scratch_ptr(int device, float** out) {
  constexpr int kMaxDevices = 64;
  static float* cached[kMaxDevices] = {};
  static std::mutex mu;
  if (device < 0 || device >= kMaxDevices) return fail(-2, "device ordinal %d out of range", device);
  std::lock_guard<std::mutex> lock(mu);
  if (!cached[device]) {
    int cur = -1;
    SIG_CUDA(cudaGetDevice(&cur));
    if (cur != device) return fail(-100, "internal: device %d is not current (current is %d)", device, cur);
    float* ptr = nullptr;
    cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_static_dq_scratch);
    if (e != cudaSuccess || !ptr)
      return fail(-100, "cudaGetSymbolAddress(static dQ scratch) failed on device %d: %s", device, cudaGetErrorString(e));
    cached[device] = ptr;
  }
  *out = cached[device];
  return 0;
}

// float32 tensors on the FMA pipe (no tensor maps, no workspace).
template <int D, int kR, int kC>
int launch_f32_shape(const SigAttnParams* p, const sigattn::F32Params& fp, bool backward) {
  using namespace sigattn;
  using S = F32Shape<D, kR, kC>;
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  const int n_q = (p->Tq + S::kRows - 1) / S::kRows;
  const int n_k = (p->Tk + S::kRows - 1) / S::kRows;
  const int64_t n_bh = (int64_t)p->B * p->H;
  if (n_bh * std::max(n_q, n_k) > INT32_MAX) return fail(-2, "too many (batch, head, tile) items: %lld", (long long)(n_bh * std::max(n_q, n_k)));
  if (!backward) {
    auto kernel = sigattn_fwd_f32_kernel<D, kR, kC>;
    if (int rc = set_smem(kernel, S::kFwdBytes, p->device)) return rc;
    kernel<<<(unsigned int)(n_bh * n_q), S::kThreads, S::kFwdBytes, stream>>>(fp, n_q);
    SIG_CUDA(cudaGetLastError());
  } else {
    auto kernel = sigattn_bwd_f32_kernel<D, kR, kC>;
    constexpr int smem = std::max(S::kDkdvBytes, S::kDqBytes);
    if (int rc = set_smem(kernel, smem, p->device)) return rc;
    const bool both = n_bh * ((int64_t)n_k + n_q) <= INT32_MAX;
    kernel<<<(unsigned int)(n_bh * (n_k + (both ? n_q : 0))), S::kThreads, smem, stream>>>(fp, n_k, n_q);
    SIG_CUDA(cudaGetLastError());
    if (!both) {
      kernel<<<(unsigned int)(n_bh * n_q), S::kThreads, smem, stream>>>(fp, 0, n_q);
      SIG_CUDA(cudaGetLastError());
    }
  }
  return 0;
}

// float32 tensors on the tensor cores (no tensor maps, no workspace either).
// CTAs per tile of the float32 tensor-core kernels: with fewer tiles than half of the SMs, the jobs of each are split over a cluster, as long as
// a part keeps four jobs of 64 rows (clusters of two find room on every SM, larger ones on 7/8 of them, see fwd_plan()).
// D = 64, us, forward and backward: B=1 H=1 T=4096 103 -> 41 and 159 -> 95; B=1 H=4 T=1024 31 -> 21 and 51 -> 37, T=2048 54 -> 36 and 89 -> 87 (136 tiles
// of the backward: not split); D = 128 H=1 T=8192 300 -> 170 and 947 -> 939.
// The last wave of more tiles, forward: B=4 T=2048 H=8 (3.46 waves, 68 tiles in two parts each) 208 -> 195, D = 128 367 -> 349; B=5 T=1024 H=8 (24 in
// four) 90 -> 82.
int tc_split(int64_t ctas, int jobs, int n_sm) {
  int split = 1;
  while (split < 8 && ctas * split * 2 <= (split == 1 ? n_sm : n_sm * 7 / 8) && jobs >= 8 * split) split *= 2;
  return split;
}
int64_t f32_tc_tiles(const SigAttnParams* p, bool backward) {
  const int64_t n_q = ((int64_t)p->Tq + sigattn::kTcRows - 1) / sigattn::kTcRows, n_k = ((int64_t)p->Tk + sigattn::kTcRows - 1) / sigattn::kTcRows;
  return (int64_t)p->B * p->H * (backward ? n_q + n_k * (p->D == 64 ? 1 : 2) : n_q);
}
// CTAs per tile, of all tiles or (all = 1) of those of the last wave.
struct F32TcParts {
  int all, last;
};
F32TcParts f32_tc_parts(const SigAttnParams* p, bool backward, int n_sm) {
  const int64_t ctas = f32_tc_tiles(p, backward);
  F32TcParts parts = {tc_split(ctas, (int)(((int64_t)(backward ? std::min(p->Tq, p->Tk) : p->Tk) + sigattn::kTcJob - 1) / sigattn::kTcJob), n_sm), 1};
  if (backward || parts.all > 1) return parts;
  // A last wave that half of the SMs would sit out is split as well, in two or four, where all tiles take the same time (a ragged last one
  // does too, but was not measured).
  const int64_t rest = ctas % n_sm;
  const bool even = !(p->flags & SIGATTN_CAUSAL) && !p->seq_lens_q && !p->seq_lens_k && !p->cu_seqlens_q && p->Tq % sigattn::kTcRows == 0;
  if (even && ctas > n_sm && rest > 0 && p->Tk >= 16 * sigattn::kTcJob) parts.last = tc_split(rest, 16, n_sm);
  return parts;
}
template <typename K, typename... Args>
int launch_clusters(K kernel, int64_t ctas, int split, int threads, int smem, cudaStream_t stream, Args... args) {
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned int)split;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned int)(ctas * split));
  cfg.blockDim = dim3((unsigned int)threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  SIG_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  return 0;
}

template <int D>
int launch_f32_tc(const SigAttnParams* p, const sigattn::F32Params& fp, bool backward, int n_sm) {
  using namespace sigattn;
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  const int n_q = (p->Tq + kTcRows - 1) / kTcRows, n_k = (p->Tk + kTcRows - 1) / kTcRows;
  const int64_t ctas = f32_tc_tiles(p, backward);
  if (ctas > INT32_MAX) return fail(-2, "too many (batch, head, tile) items: %lld", (long long)ctas);
  const F32TcParts parts_of = f32_tc_parts(p, backward, n_sm);
  const int split = parts_of.all, last = parts_of.last;
  if (!backward) {
    constexpr int smem = TcShape<D, kTcFwd>::kDynBytes;
    auto whole = sigattn_f32_tc_fwd_kernel<D, false>;
    auto parts = sigattn_f32_tc_fwd_kernel<D, true>;
    if (int rc = set_smem(whole, smem, p->device)) return rc;
    if (int rc = set_smem(parts, smem, p->device)) return rc;
    if (split > 1) return launch_clusters(parts, ctas, split, kTcThreads, smem, stream, fp, n_q, split, 0);
    const int64_t rest = last > 1 ? ctas % n_sm : 0;
    whole<<<(unsigned int)(ctas - rest), kTcThreads, smem, stream>>>(fp, n_q, 1, 0);
    SIG_CUDA(cudaGetLastError());
    return last > 1 ? launch_clusters(parts, rest, last, kTcThreads, smem, stream, fp, n_q, last, (int)(ctas - rest)) : 0;
  }
  constexpr int smem = tc_bwd_bytes<D>();
  if (split > 1) {
    auto parts = sigattn_f32_tc_bwd_kernel<D, true>;
    if (int rc = set_smem(parts, smem, p->device)) return rc;
    return launch_clusters(parts, ctas, split, kTcThreads, smem, stream, fp, n_k, n_q, split);
  }
  auto whole = sigattn_f32_tc_bwd_kernel<D, false>;
  if (int rc = set_smem(whole, smem, p->device)) return rc;
  whole<<<(unsigned int)ctas, kTcThreads, smem, stream>>>(fp, n_k, n_q, 1);
  SIG_CUDA(cudaGetLastError());
  return 0;
}

// Whether float32 tensors take the tensor-core kernels.  Their tiles have 128 rows, and setting one up takes as long as two of
// its steps of 64: so they need enough 64-row tiles to occupy half of the SMs (in a forward of the queries, in a backward of
// queries and keys on average), or sequences that are long enough for the faster steps to pay even where 16-row tiles of the
// FMA kernels would occupy more of the chip.  Device time of these over FMA kernels, from 477 shapes (means over those that
// differ in B H only):
//  - D = 64 forward: T=256, 64 tiles or more 0.42 - 0.77, fewer 1.08; T=512 0.31 - 0.88, T=1024 0.25 - 0.75; backward T=384 0.30 - 0.80,
//    T=1024 0.22 - 0.63.  Heads of 32 columns, which get the same kernels (and the same bits as heads filled up with zeros):
//    T=512 0.37 - 1.01, backward T=384 0.40 - 1.04.
//  - D = 128 forward: T=256 0.36 - 0.69 from 148 tiles on, 0.88 at 64 and 1.05 there with a causal mask, 1.3 below; Tk = 512 0.98;
//    backward (three kernels): 0.35 - 0.71 from 96 tiles on, 0.76 - 0.89 at 64 with T >= 512 (causal 0.94 - 1.06), 1.1 - 1.6 below.
//  - below 256 rows on both sides 0.5 - 2.2, and below 64 keys or 16 queries mostly padding: FMA kernels.
//  - packed sequences that are shorter on average than a tile is worth, whatever the longest one, once the rows are so many that the FMA
//    kernels are not waiting for that one alone (as many per SM as it has).  Forward D = 64, mean length 32 and 64 1.9 - 2.0, 96
//    0.95 - 1.03 and 128 0.98 - 1.09, causal 96 1.17, 128 1.2, 192 1.00 - 1.04, 256 0.76; D = 128 0.87 - 0.97 from 32 on; backward 64
//    1.25 - 1.39 and 1.23, 96 0.66 - 0.69 and 0.73 (causal 0.82).  With one of 1024 among few of 64, 0.66 and 0.61 (step).
//    (Padded ones, whose lengths the host does not know, go by the padded extents.  Where a tenth or less of those is filled they are slower than
//    the FMA kernels: T=1024 B=128 H=8 filled to 48, D = 64 forward 1.28, with the backward 1.09, D = 128 0.88 and 0.97; T=512 B=256 to 40 1.65
//    and 1.37, 1.09 and 1.23; to 200 of 1024 0.56 and 0.47, 0.43 and 0.49; full 0.26, 0.26, 0.21 and 0.28.)
bool f32_tc(const SigAttnParams* p, bool backward, int n_sm) {
  const int64_t Tq = p->Tq, Tk = p->Tk, longer = std::max(Tq, Tk);
  if (Tk < 64 || Tq < 16 || longer < 256) return false;
  // (the kernels' factor of the score is 2^-31.5 scale, which must not be a subnormal number)
  if (p->scale != 0.0f && !(std::abs(p->scale) >= 1e-25f)) return false;
  if (p->cu_seqlens_q && (backward || p->D == 64)) {
    const int64_t rows = std::max(p->total_q, p->total_k);  // B sequences of `line` would have more
    const int64_t line = backward ? 80 : (p->flags & SIGATTN_CAUSAL) ? 192 : 96;
    if (rows < line * p->B && rows * p->H >= n_sm * longer) return false;
  }
  const int64_t tiles = (int64_t)p->B * p->H * (((backward ? (Tq + Tk) / 2 : Tq) + 63) / 64);
  if (p->D == 128) return backward ? tiles >= 96 || (tiles >= 64 && longer >= 512) : tiles >= 72 || Tk >= 512;
  return tiles >= 64 || longer >= (backward ? 384 : 512);
}

// Rows per CTA: 64 once such tiles occupy half of the SMs; below that 16, with four times the threads per row, which take
// 1.9 times the SM time per row and a quarter of the latency (B=2 T=256 H=4: 15 against 30 us forward).
int f32_tile_rows(const SigAttnParams* p, int n_sm) {
  const int64_t tiles64 = (int64_t)p->B * p->H * ((std::min(p->Tq, p->Tk) + 63) / 64);
  return 2 * tiles64 >= n_sm ? 64 : 16;
}

template <int D>
int launch_f32_d(const SigAttnParams* p, bool backward) {
  using namespace sigattn;
  F32Params fp = {};
  fp.q = static_cast<const float*>(p->q);
  fp.k = static_cast<const float*>(p->k);
  fp.v = static_cast<const float*>(p->v);
  fp.dout = static_cast<const float*>(p->dout);
  fp.o = static_cast<float*>(p->o);
  fp.dq = static_cast<float*>(p->dq);
  fp.dk = static_cast<float*>(p->dk);
  fp.dv = static_cast<float*>(p->dv);
  fp.q_sb = p->q_strides[0]; fp.q_st = p->q_strides[1]; fp.q_sh = p->q_strides[2];
  fp.k_sb = p->k_strides[0]; fp.k_st = p->k_strides[1]; fp.k_sh = p->k_strides[2];
  fp.v_sb = p->v_strides[0]; fp.v_st = p->v_strides[1]; fp.v_sh = p->v_strides[2];
  fp.o_sb = p->o_strides[0]; fp.o_st = p->o_strides[1]; fp.o_sh = p->o_strides[2];
  fp.do_sb = p->do_strides[0]; fp.do_st = p->do_strides[1]; fp.do_sh = p->do_strides[2];
  fp.dq_sb = p->dq_strides[0]; fp.dq_st = p->dq_strides[1]; fp.dq_sh = p->dq_strides[2];
  fp.dk_sb = p->dk_strides[0]; fp.dk_st = p->dk_strides[1]; fp.dk_sh = p->dk_strides[2];
  fp.dv_sb = p->dv_strides[0]; fp.dv_st = p->dv_strides[1]; fp.dv_sh = p->dv_strides[2];
  fp.lens_q = p->seq_lens_q;
  fp.lens_k = p->seq_lens_k;
  fp.cu_q = p->cu_seqlens_q;
  fp.cu_k = p->cu_seqlens_k;
  fp.bias = p->bias;
  fp.score_mod = p->score_mod;
  fp.scale = p->scale;
  fp.bias_scalar = p->bias_scalar;
  if (p->flags & SIGATTN_BIAS_NEG_LOG_LK) { fp.bias = nullptr; fp.bias_scalar = nanf(""); }  // see item_bias()
  fp.B = p->B; fp.H = p->H; fp.Tq = p->Tq; fp.Tk = p->Tk;
  fp.d_cols = head_cols(p);
  fp.causal = (p->flags & SIGATTN_CAUSAL) ? 1 : 0;
  cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
  FwdDeviceInfo info;
  if (int rc = fwd_device_info(p->device, &info)) return rc;
  if (int rc = zero_gaps(p, backward, info.n_sm)) return rc;
  if (p->ev_main_start) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_start), stream));
  int rc = 0;
  if (f32_tc(p, backward, info.n_sm)) {
    rc = launch_f32_tc<D>(p, fp, backward, info.n_sm);
  } else
    rc = f32_tile_rows(p, info.n_sm) == 64 ? launch_f32_shape<D, 4, D / 64>(p, fp, backward) : launch_f32_shape<D, 1, 4>(p, fp, backward);
  if (rc) return rc;
  if (p->ev_main_stop) SIG_CUDA(cudaEventRecord(static_cast<cudaEvent_t>(p->ev_main_stop), stream));
  return 0;
}

int launch_f32(const SigAttnParams* p, bool backward) {
  struct Tensor { const void* ptr; const int64_t* strides; const char* name; };
  const Tensor fwd_t[] = {{p->q, p->q_strides, "q"}, {p->k, p->k_strides, "k"}, {p->v, p->v_strides, "v"}, {p->o, p->o_strides, "o"}};
  const Tensor bwd_t[] = {{p->q, p->q_strides, "q"}, {p->k, p->k_strides, "k"}, {p->v, p->v_strides, "v"},
                          {p->dout, p->do_strides, "dout"}, {p->dq, p->dq_strides, "dq"}, {p->dk, p->dk_strides, "dk"},
                          {p->dv, p->dv_strides, "dv"}};
  const Tensor* ts = backward ? bwd_t : fwd_t;
  const int n = backward ? 7 : 4;
  for (int t = 0; t < n; ++t) {
    if ((reinterpret_cast<uintptr_t>(ts[t].ptr) & 15u) != 0) return fail(-3, "%s: base pointer must be 16-byte aligned", ts[t].name);
    for (int i = 0; i < 3; ++i)
      if (ts[t].strides[i] % 4 != 0) return fail(-3, "%s: strides must be multiples of 4 elements (16 bytes)", ts[t].name);
  }
  return p->D == 64 ? launch_f32_d<64>(p, backward) : launch_f32_d<128>(p, backward);
}

// Self-test of the bounded waits: one warp waits on a barrier that nothing ever arrives on, with a
// limit of a few milliseconds, exactly as a kernel of the library would on a lost signal: the wait
// gives up, records its site in the health word, and the kernel returns normally.
constexpr int kSelfTestSite = 0x30001;
__global__ void sigattn_selftest_wait_kernel(unsigned long long limit_ns, int* gave_up) {
  __shared__ __align__(8) unsigned long long bar_storage;
  __shared__ int abort_flag;
  const uint32_t bar = sigattn::smem_u32(&bar_storage);
  if (threadIdx.x == 0) {
    abort_flag = 0;
    sigattn::mbar_init(bar, 1);
    sigattn::fence_mbar_init();
  }
  __syncthreads();
  const bool ok = sigattn::mbar_wait(bar, 0, &abort_flag, kSelfTestSite, limit_ns);
  if (threadIdx.x == 0) *gave_up = ok ? 0 : 1;
}

}  // namespace

extern "C" {

const char* sigattn_last_error(void) { return g_err; }

int sigattn_query(int what) {
  switch (what) {
    case SIGATTN_Q_ABI_VERSION: return SIGATTN_ABI_VERSION;
    case SIGATTN_Q_SM_ARCH: return 100;
    case SIGATTN_Q_MAX_HEAD_DIM: return 128;
    case SIGATTN_Q_PARAMS_SIZE: return (int)sizeof(SigAttnParams);
    case SIGATTN_Q_HEAD_COLS: return 1;
    default: return -1;
  }
}

int sigattn_form(const SigAttnParams* p, int backward, int n_sm) {
  g_err[0] = 0;
  if (!p) return fail(-1, "params is NULL");
  if (p->struct_bytes != sizeof(SigAttnParams)) return fail(-1, "struct_bytes %u != sizeof(SigAttnParams) %zu (ABI mismatch)", p->struct_bytes, sizeof(SigAttnParams));
  if (n_sm < 1) return fail(-2, "n_sm must be positive, got %d", n_sm);
  if (p->dtype == SIGATTN_FP32) {
    if (f32_tc(p, backward != 0, n_sm)) return SIGATTN_FORM_F32_TC;
    return f32_tile_rows(p, n_sm) == 64 ? SIGATTN_FORM_F32_64 : SIGATTN_FORM_F32_16;
  }
  if (!backward) return fwd_plan(p, n_sm).split > 1 ? SIGATTN_FORM_FWD_SPLIT : SIGATTN_FORM_FWD;
  if (p->flags & SIGATTN_BWD_SPLIT) return SIGATTN_FORM_BWD_STREAM;
  return bwd_by_head(p, n_sm) ? SIGATTN_FORM_BWD_BY_HEAD : SIGATTN_FORM_BWD;
}

int sigattn_parts(const SigAttnParams* p, int backward, int n_sm) {
  const int form = sigattn_form(p, backward, n_sm);
  if (form < 0) return form;
  if (form == SIGATTN_FORM_FWD || form == SIGATTN_FORM_FWD_SPLIT) return fwd_plan(p, n_sm).split;
  if (form != SIGATTN_FORM_F32_TC) return 1;
  const F32TcParts parts = f32_tc_parts(p, backward != 0, n_sm);
  return std::max(parts.all, parts.last);
}

size_t sigattn_bwd_workspace_bytes(int32_t B, int32_t Tq, int32_t H, int32_t D) {
  if (B <= 0 || Tq <= 0 || H <= 0 || D <= 0) return 0;
  return (size_t)B * (size_t)Tq * (size_t)H * (size_t)D * sizeof(float);
}

int sigattn_device_status(int device) {
  DeviceGuard g;
  SIG_CUDA(g.enter(device));
  SIG_CUDA(cudaDeviceSynchronize());
  int v = 0;
  SIG_CUDA(cudaMemcpyFromSymbol(&v, sigattn::g_status_word, sizeof(int)));
  if (v != 0) {
    // A kernel that gave up may have left its work-item counters half used: clear them together
    // with the status, so that the library is usable again after the caller has seen the failure.
    int zero = 0;
    SIG_CUDA(cudaMemcpyToSymbol(sigattn::g_status_word, &zero, sizeof(int)));
    void* tickets = nullptr;
    SIG_CUDA(cudaGetSymbolAddress(&tickets, g_item_tickets));
    SIG_CUDA(cudaMemset(tickets, 0, sizeof(unsigned int) * 2 * kTicketSlots));
  }
  if (device >= 0 && device < kMaxMirrorDevices) g_host_status[device] = 0;
  return v;
}


int sigattn_selftest_bounded_wait(int device, int limit_ms) {
  g_err[0] = 0;
  if (limit_ms < 1 || limit_ms > 1000) return fail(-2, "limit_ms must be in [1, 1000], got %d", limit_ms);
  DeviceGuard g;
  SIG_CUDA(g.enter(device));
  {
    FwdDeviceInfo info;  // first use of the device: also installs the host-visible copy of the health word
    if (int rc = fwd_device_info(device, &info)) return rc;
  }
  int* flag = nullptr;
  SIG_CUDA(cudaMalloc(&flag, sizeof(int)));
  cudaError_t e = cudaMemset(flag, 0xff, sizeof(int));
  int gave_up = -1;
  if (e == cudaSuccess) {
    sigattn_selftest_wait_kernel<<<1, 32>>>((unsigned long long)limit_ms * 1000000ull, flag);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(&gave_up, flag, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(flag);
  if (e != cudaSuccess) return fail(-100, "self-test: %s", cudaGetErrorString(e));
  return gave_up;
}

int sigattn_fwd(const SigAttnParams* p) {
  g_err[0] = 0;
  int rc = check_common(p, false);
  if (rc < 0) return rc;
  if (rc == 1) return 0;
  SIG_REFUSE_IF_SICK(p);
  DeviceGuard g;
  SIG_CUDA(g.enter(p->device));
  const Extents ex = extents(p);
  if (ex.Tq == 0) return 0;
  if (p->Tq == 0) {  // every row is outside a sequence
    FwdDeviceInfo info;
    if ((rc = fwd_device_info(p->device, &info))) return rc;
    return zero_gaps(p, false, info.n_sm);
  }
  if (ex.Tk == 0 || p->Tk == 0) {  // no keys at all: the output is all zeros
    const Strides3 os = map_strides(p->o_strides, ex.Tq, ex.packed);
    return zero_fill(p->o, os.s, ex.B, ex.Tq, p->H, head_cols(p), p->dtype, static_cast<cudaStream_t>(p->stream), "o");
  }
  if (p->dtype == SIGATTN_FP32) return launch_f32(p, false);
  CUtensorMap qm, km, vm;
  FwdDeviceInfo info;
  if ((rc = fwd_device_info(p->device, &info))) return rc;
  const int q_rows = fwd_plan(p, info.n_sm).twice ? 64 : 128;  // of a load
  if ((rc = make_map(&qm, p->q, p->dtype, ex.B, ex.Tq, p->H, head_cols(p), map_strides(p->q_strides, ex.Tq, ex.packed).s, q_rows, "q"))) return rc;
  if ((rc = make_map(&km, p->k, p->dtype, ex.B, ex.Tk, p->H, head_cols(p), map_strides(p->k_strides, ex.Tk, ex.packed).s, 128, "k"))) return rc;
  if ((rc = make_map(&vm, p->v, p->dtype, ex.B, ex.Tk, p->H, head_cols(p), map_strides(p->v_strides, ex.Tk, ex.packed).s, 128, "v"))) return rc;
  if ((reinterpret_cast<uintptr_t>(p->o) & 15u) != 0) return fail(-3, "o: base pointer must be 16-byte aligned");
  for (int i = ex.packed ? 1 : 0; i < 3; ++i)
    if (p->o_strides[i] % 8 != 0) return fail(-3, "o: strides must be multiples of 8 elements");

  const bool bf = p->dtype == SIGATTN_BF16;
  const bool sm = p->score_mod != nullptr;
  const bool acc = (p->flags & SIGATTN_ACCURATE) != 0;
#define SIG_FWD(DD, BF, SM)                                             \
  do {                                                                  \
    if (acc) return launch_fwd<DD, BF, SM, true>(p, qm, km, vm);        \
    return launch_fwd<DD, BF, SM, false>(p, qm, km, vm);                \
  } while (0)
  if (p->D == 64) {
    if (bf) { if (sm) SIG_FWD(64, true, true); else SIG_FWD(64, true, false); }
    else    { if (sm) SIG_FWD(64, false, true); else SIG_FWD(64, false, false); }
  } else {
    if (bf) { if (sm) SIG_FWD(128, true, true); else SIG_FWD(128, true, false); }
    else    { if (sm) SIG_FWD(128, false, true); else SIG_FWD(128, false, false); }
  }
#undef SIG_FWD
  return fail(-2, "unreachable");
}

int sigattn_bwd(const SigAttnParams* p) {
  g_err[0] = 0;
  int rc = check_common(p, true);
  if (rc < 0) return rc;
  if (rc == 1) return 0;
  SIG_REFUSE_IF_SICK(p);
  DeviceGuard g;
  SIG_CUDA(g.enter(p->device));
  const Extents ex = extents(p);
  if (ex.Tq == 0 || ex.Tk == 0 || p->Tq == 0 || p->Tk == 0) {
    // no query or no key: every gradient is zero
    cudaStream_t stream = static_cast<cudaStream_t>(p->stream);
    if ((rc = zero_fill(p->dq, map_strides(p->dq_strides, ex.Tq, ex.packed).s, ex.B, ex.Tq, p->H, head_cols(p), p->dtype, stream, "dq"))) return rc;
    if ((rc = zero_fill(p->dk, map_strides(p->dk_strides, ex.Tk, ex.packed).s, ex.B, ex.Tk, p->H, head_cols(p), p->dtype, stream, "dk"))) return rc;
    return zero_fill(p->dv, map_strides(p->dv_strides, ex.Tk, ex.packed).s, ex.B, ex.Tk, p->H, head_cols(p), p->dtype, stream, "dv");
  }
  if (p->dtype == SIGATTN_FP32) return launch_f32(p, true);
  CUtensorMap qm, km, vm, dom;
  if ((rc = make_map(&qm, p->q, p->dtype, ex.B, ex.Tq, p->H, head_cols(p), map_strides(p->q_strides, ex.Tq, ex.packed).s, 128, "q"))) return rc;
  if ((rc = make_map(&km, p->k, p->dtype, ex.B, ex.Tk, p->H, head_cols(p), map_strides(p->k_strides, ex.Tk, ex.packed).s, 128, "k"))) return rc;
  if ((rc = make_map(&vm, p->v, p->dtype, ex.B, ex.Tk, p->H, head_cols(p), map_strides(p->v_strides, ex.Tk, ex.packed).s, 128, "v"))) return rc;
  if ((rc = make_map(&dom, p->dout, p->dtype, ex.B, ex.Tq, p->H, head_cols(p), map_strides(p->do_strides, ex.Tq, ex.packed).s, 128, "dout"))) return rc;
  const void* outs[3] = {p->dq, p->dk, p->dv};
  const int64_t* ostr[3] = {p->dq_strides, p->dk_strides, p->dv_strides};
  for (int t = 0; t < 3; ++t) {
    if ((reinterpret_cast<uintptr_t>(outs[t]) & 15u) != 0) return fail(-3, "gradient pointers must be 16-byte aligned");
    for (int i = ex.packed ? 1 : 0; i < 3; ++i)
      if (ostr[t][i] % 8 != 0) return fail(-3, "gradient strides must be multiples of 8 elements");
  }
  const bool bf = p->dtype == SIGATTN_BF16;
  const bool acc = (p->flags & SIGATTN_ACCURATE) != 0;
  const bool split = (p->flags & SIGATTN_BWD_SPLIT) != 0;
#define SIG_BWD(DD, BF)                                                                   \
  do {                                                                                    \
    if (split) {                                                                          \
      if (acc) return launch_bwd_stream<DD, BF, true>(p, qm, km, vm, dom);                \
      return launch_bwd_stream<DD, BF, false>(p, qm, km, vm, dom);                        \
    }                                                                                     \
    if (acc) return launch_bwd_fused<DD, BF, true>(p, qm, km, vm, dom);                   \
    return launch_bwd_fused<DD, BF, false>(p, qm, km, vm, dom);                           \
  } while (0)
  if (p->D == 64) { if (bf) SIG_BWD(64, true); else SIG_BWD(64, false); }
  else            { if (bf) SIG_BWD(128, true); else SIG_BWD(128, false); }
#undef SIG_BWD
  return fail(-2, "unreachable");
}

int sigattn_bwd_static_scratch(const SigAttnParams* p) {
  g_err[0] = 0;
  int rc = check_common(p, true);
  if (rc < 0) return rc;
  if (rc == 1) return 0;
  const Extents ex = extents(p);
  const unsigned long long elems = (unsigned long long)ex.B * (unsigned long long)ex.Tq * (unsigned long long)p->H *
                                   (unsigned long long)p->D;
  // float32 tensors run kernels of their own, which use no accumulator: no limit applies to them
  if (p->dtype == SIGATTN_FP32) return sigattn_bwd(p);
  if (elems > SIGATTN_STATIC_SCRATCH_ELEMS)
    return fail(-4, "problem too large for the built-in scratch: B*Tq*H*D = %llu elements, limit %u; "
                    "use sigattn_bwd with a caller-provided workspace", elems, (unsigned)SIGATTN_STATIC_SCRATCH_ELEMS);
  float* scratch = nullptr;
  {
    DeviceGuard g;  // makes p->device current for the address lookup
    SIG_CUDA(g.enter(p->device));
    if ((rc = static_scratch_ptr(p->device, &scratch))) return rc;
  }
  // Same path as sigattn_bwd from here on; no form of it reads the accumulator before it has written it.
  SigAttnParams q = *p;
  q.flags &= ~(uint32_t)SIGATTN_BWD_SPLIT;  // the kernel that accumulates dQ in scratch memory
  q.workspace = scratch;
  q.workspace_bytes = (size_t)SIGATTN_STATIC_SCRATCH_ELEMS * sizeof(float);
  return sigattn_bwd(&q);
}

}  // extern "C"
