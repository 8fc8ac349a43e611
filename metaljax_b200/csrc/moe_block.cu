// The gathered SwiGLU expert block in one call (eterevsky/metaljax src/metaljax/moe.py:1283-1461: pairs sorted by
// expert, three grouped products, the routed weighted sum), every launch on the caller's stream, nothing read
// back by the host: sort -> gate, up -> silu(gate) * up -> down -> weighted sum. (qmm_moe_experts_checked looks at one word of
// the sort's once everything is enqueued.)
//
// A few decoded tokens through such a block used to be a sort, a bincount (which waits for the device), half a
// dozen index kernels and three products whose 64-row tiles were one or two rows full: 8 tokens, 2 of 8 experts each,
// d 4096, ffn 14336 took 700 us for 713 MB of weights.
#include <cuda_runtime.h>
#include <sched.h>

#include <mutex>
#include <vector>

#include "../../include/qmm.h"
#include "qmm_internal.h"

namespace qmm {
namespace {

constexpr int kSortWarps = 32;

// Pairs p = t * k + j sorted by expert, stable: a counting sort by one CTA. A warp owns a stretch of pairs, counts its
// experts, and places its pairs behind those of the warps before it. Bound by latency: P / 1024 rounds of a
// match and a shared-memory update, twice (8192 pairs: 2 x 8 rounds).
//   sizes [E] pairs per expert; token_of_row [P]; row_of_pair [P]; *report (host memory, or NULL) becomes 2 ticket + (some index was
//   out of range) as soon as every index has been seen
template <typename IT>
__global__ void __launch_bounds__(kSortWarps * 32)
moe_sort_kernel(const IT* __restrict__ experts, int pairs, int k, int nexp, int32_t* __restrict__ sizes, int32_t* __restrict__ token_of_row,
                int64_t* __restrict__ row_of_pair, int* status, volatile unsigned* report, unsigned ticket) {
  extern __shared__ int counts[];                  // [warps][E]
  __shared__ unsigned out_of_range;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  for (int i = threadIdx.x; i < warps * nexp; i += blockDim.x) counts[i] = 0;
  if (threadIdx.x == 0) out_of_range = 0u;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  __syncthreads();
  const int per = (pairs + warps * 32 - 1) / (warps * 32) * 32, lo = warp * per, hi = min(lo + per, pairs);
  int* mine = counts + warp * nexp;
  auto expert_of = [&](int p) -> int {
    if (p >= hi) return -1;
    const int64_t e = static_cast<int64_t>(experts[p]);
    if (e >= 0 && e < nexp) return static_cast<int>(e);
    if (report) out_of_range = 1u;                 // never followed: reported, and the pair goes to expert 0
    else atomicCAS(status, 0, QMM_DEVICE_BAD_INDEX);
    return 0;
  };
  for (int p0 = lo; p0 < hi; p0 += 32) {
    const int e = expert_of(p0 + lane);
    const unsigned same = __match_any_sync(0xffffffffu, e);
    if (e >= 0 && (same & below) == 0) mine[e] += __popc(same);
    __syncwarp();
  }
  __syncthreads();
  if (report && threadIdx.x == 0) *report = 2u * ticket + out_of_range;
  // counts -> where a warp's pairs of an expert start: after the experts before it and the warps before it
  if (warp == 0) {
    int before = 0;
    for (int e0 = 0; e0 < nexp; e0 += 32) {
      const int e = e0 + lane;
      int own = 0;
      if (e < nexp)
        for (int w = 0; w < warps; ++w) own += counts[w * nexp + e];
      int run = own;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
      }
      if (e < nexp) {
        sizes[e] = own;
        int at = before + run - own;
        for (int w = 0; w < warps; ++w) {
          const int c = counts[w * nexp + e];
          counts[w * nexp + e] = at;
          at += c;
        }
      }
      before += __shfl_sync(0xffffffffu, run, 31);
    }
  }
  __syncthreads();
  for (int p0 = lo; p0 < hi; p0 += 32) {
    const int p = p0 + lane, e = expert_of(p);
    const unsigned same = __match_any_sync(0xffffffffu, e);
    int row = 0;
    if (e >= 0) row = mine[e] + __popc(same & below);
    __syncwarp();
    if (e >= 0) {
      if ((same & below) == 0) mine[e] += __popc(same);
      token_of_row[row] = p / k;
      row_of_pair[p] = row;
    }
    __syncwarp();
  }
}

// out[r, :] = x[token_of_row[r], :], 16 bytes a thread (bound by HBM: the rows are written once and read from L2).
__global__ void gather_rows_kernel(const uint4* __restrict__ x, const int32_t* __restrict__ token_of_row, uint4* __restrict__ out, int64_t rows, int pieces) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  for (int64_t r = blockIdx.x; r < rows; r += gridDim.x) {
    const uint4* src = x + static_cast<int64_t>(token_of_row[r]) * pieces;
    for (int i = threadIdx.x; i < pieces; i += blockDim.x) out[r * pieces + i] = __ldg(src + i);
  }
}

size_t align256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

struct Workspace {
  size_t sizes, tokens, rows, xs, gate, up, down, total;
};

// `gathered`: the products read their rows of x by index, no sorted copy of x is made.
Workspace layout(const qmm_moe_block& b, bool gathered) {
  const size_t pairs = static_cast<size_t>(b.tokens) * b.k, es = elem_size(b.x_dtype);
  Workspace w;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += align256(bytes);
    return here;
  };
  w.sizes = take(static_cast<size_t>(b.experts) * 4);
  w.tokens = take(pairs * 4);
  w.rows = take(pairs * 8);
  w.xs = take(gathered ? 0 : pairs * b.d * es);
  w.gate = take(pairs * b.ffn * es);
  w.up = take(pairs * b.ffn * es);
  w.down = take(pairs * b.d * es);
  w.total = at;
  return w;
}

int sort_warps(int64_t pairs, int experts) {
  int64_t w = (pairs + 31) / 32;
  if (w > kSortWarps) w = kSortWarps;
  while (w > 1 && w * experts * 4 > 96 * 1024) w /= 2;
  return static_cast<int>(w);
}

qmm_problem product(const qmm_moe_block& b, const qmm_moe_weight& w, const void* x, void* y, const int32_t* sizes, int64_t k, int64_t n) {
  qmm_problem p = {};
  p.struct_size = sizeof(p);
  p.mode = b.mode; p.bits = b.bits; p.group_size = b.group_size;
  p.x_dtype = p.y_dtype = b.x_dtype; p.table_dtype = b.table_dtype;
  p.batch = b.experts; p.M = b.tokens * b.k; p.K = k; p.N = n;
  p.x = x; p.w = static_cast<const uint32_t*>(w.w); p.scales = w.scales; p.biases = w.biases; p.y = y;
  p.w_batch_stride = n;
  p.group_sizes = sizes;
  return p;
}

int check_block(const qmm_moe_block& b) {
  if (b.struct_size != sizeof(qmm_moe_block)) return fail(QMM_ERR_UNSUPPORTED, "qmm_moe_block.struct_size=%u, library expects %zu", b.struct_size, sizeof(b));
  if (b.x_dtype != QMM_BF16 && b.x_dtype != QMM_F16) return fail(QMM_ERR_DTYPE, "moe_experts: bf16 or f16 activations");
  if (b.tokens < 0 || b.k < 1 || b.experts < 1 || b.experts > 1024 || b.d < 8 || b.d % 8 || b.ffn < 8 || b.ffn % 8 || b.tokens * b.k >= (1LL << 31))
    return fail(QMM_ERR_SHAPE, "moe_experts: d and ffn are multiples of 8, 1..1024 experts");
  if (b.index_bytes != 4 && b.index_bytes != 8) return fail(QMM_ERR_DTYPE, "moe_experts: expert indices are 32- or 64-bit");
  return QMM_OK;
}

// Words of page-locked memory that the sort reports to, one per call that is waiting for its own; they stay for later calls.
struct Report {
  volatile unsigned* word;
  unsigned ticket;
};
std::mutex g_reports_mutex;
std::vector<Report> g_reports;

bool take_report(Report* out) {
  {
    std::lock_guard<std::mutex> lock(g_reports_mutex);
    if (!g_reports.empty()) {
      *out = g_reports.back();
      g_reports.pop_back();
      ++out->ticket;
      return true;
    }
  }
  void* p = nullptr;
  if (cudaHostAlloc(&p, 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  out->word = static_cast<volatile unsigned*>(p);
  *out->word = 0u;
  out->ticket = 1u;
  return true;
}

void give_back(const Report& r) {
  std::lock_guard<std::mutex> lock(g_reports_mutex);
  g_reports.push_back(r);
}

bool takes_rows(const qmm_moe_block& b) {
  return grouped_takes_rows(product(b, b.w1, nullptr, nullptr, reinterpret_cast<const int32_t*>(16), b.d, b.ffn));
}

}  // namespace
}  // namespace qmm

using namespace qmm;

extern "C" int64_t qmm_moe_workspace_bytes(const qmm_moe_block* block) {
  if (!block || check_block(*block)) return -1;
  return static_cast<int64_t>(layout(*block, takes_rows(*block)).total);
}

static int enqueue_block(const qmm_moe_block* block, void* stream, const Report& report) {
  if (!block) return fail(QMM_ERR_NULL, "moe_experts: block is NULL");
  const qmm_moe_block& b = *block;
  int rc = check_block(b);
  if (rc || b.tokens == 0) return rc;
  if (!b.x || !b.indices || !b.weights || !b.out || !b.workspace) return fail(QMM_ERR_NULL, "moe_experts: null pointer");
  const bool gathered = takes_rows(b);
  const Workspace ws = layout(b, gathered);
  if (b.workspace_bytes < static_cast<int64_t>(ws.total)) return fail(QMM_ERR_TOO_LARGE, "moe_experts: workspace of %lld bytes, %zu needed", (long long)b.workspace_bytes, ws.total);
  if ((reinterpret_cast<uintptr_t>(b.x) | reinterpret_cast<uintptr_t>(b.out) | reinterpret_cast<uintptr_t>(b.workspace)) & 15)
    return fail(QMM_ERR_LAYOUT, "moe_experts: pointers must be 16-byte aligned");
  int* status = device_status_word();
  if (!status) return fail(QMM_ERR_CUDA, "could not allocate the device status word");
  uint8_t* base = static_cast<uint8_t*>(b.workspace);
  int32_t* sizes = reinterpret_cast<int32_t*>(base + ws.sizes);
  int32_t* tokens = reinterpret_cast<int32_t*>(base + ws.tokens);
  int64_t* rows = reinterpret_cast<int64_t*>(base + ws.rows);
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t pairs = b.tokens * b.k;

  const RowsGather pick = {tokens, b.tokens};
  const qmm_problem gate = product(b, b.w1, gathered ? b.x : base + ws.xs, base + ws.gate, sizes, b.d, b.ffn);
  const qmm_problem up = product(b, b.w3, gathered ? b.x : base + ws.xs, base + ws.up, sizes, b.d, b.ffn);
  const qmm_problem down = product(b, b.w2, base + ws.gate, base + ws.down, sizes, b.ffn, b.d);
  if ((rc = check_problem(gate)) || (rc = check_problem(up)) || (rc = check_problem(down))) return rc;

  const int warps = sort_warps(pairs, b.experts);
  const size_t smem = static_cast<size_t>(warps) * b.experts * 4;
  static bool configured[kMaxDevices] = {};        // the attribute is per device
  const int dev = current_device();
  if (dev < 0) return QMM_ERR_DEVICE;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(moe_sort_kernel<int64_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024 + 4096);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(moe_sort_kernel<int32_t>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024 + 4096);
    if (e != cudaSuccess) return fail(QMM_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    configured[dev] = true;
  }
  if (b.index_bytes == 8)
    launch_early(moe_sort_kernel<int64_t>, 1, warps * 32, smem, st, static_cast<const int64_t*>(b.indices), static_cast<int>(pairs), b.k, b.experts, sizes, tokens, rows, status, report.word, report.ticket);
  else
    launch_early(moe_sort_kernel<int32_t>, 1, warps * 32, smem, st, static_cast<const int32_t*>(b.indices), static_cast<int>(pairs), b.k, b.experts, sizes, tokens, rows, status, report.word, report.ticket);
  count_launch();
  if (!gathered) {
    const int pieces = static_cast<int>(b.d * elem_size(b.x_dtype) / 16);
    const int64_t cap = static_cast<int64_t>(device_sm_count()) * 8;
    launch_early(gather_rows_kernel, static_cast<unsigned>(pairs < cap ? pairs : cap), pieces >= 256 ? 256 : 128, 0, st, static_cast<const uint4*>(b.x), tokens,
                 reinterpret_cast<uint4*>(base + ws.xs), pairs, pieces);
    count_launch();
  }
  if ((rc = check_launch("moe_sort_kernel"))) return rc;
  const bool paired = gathered && rows_pair_pays(gate);
  if (paired) {                                    // both products and the gate as one launch
    const RowsPair second = {up.w, up.scales, up.biases};
    if ((rc = launch_rows(gate, st, &pick, false, &second))) return rc;
  } else if (gathered) {
    if ((rc = launch_rows(gate, st, &pick)) || (rc = launch_rows(up, st, &pick))) return rc;
  } else {
    if ((rc = run_problem(gate, st)) || (rc = run_problem(up, st))) return rc;
  }
  if (!paired && (rc = qmm_moe_silu_mul(base + ws.gate, base + ws.up, base + ws.gate, pairs * b.ffn, b.x_dtype, stream))) return rc;
  if ((rc = run_problem(down, st))) return rc;
  return qmm_moe_routed_sum(base + ws.down, rows, b.weights, b.out, b.tokens, b.k, b.d, pairs, b.x_dtype, stream);
}

extern "C" int qmm_moe_experts(const qmm_moe_block* block, void* stream) { return enqueue_block(block, stream, Report{}); }

// The wait is for the first kernel of the block alone, and it is waited for behind the last enqueue: the host is back, and enqueues what
// comes next, while the products run (8 tokens, 2 of 8 experts, d 4096, ffn 14336: 202.2 us a call without the look, 202.4 with it, when gate and up were two launches; 182 with it now).
extern "C" int qmm_moe_experts_checked(const qmm_moe_block* block, void* stream) {
  const cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess) cudaGetLastError();
  Report report = {};
  if (capturing != cudaStreamCaptureStatusNone || !block || block->tokens <= 0 || !take_report(&report)) return qmm_moe_experts(block, stream);
  int rc = enqueue_block(block, stream, report);
  if (rc) return rc;                               // (the word is left out of the pool: the sort may have been launched)
  auto arrived = [&] { return *report.word >> 1 == (report.ticket & 0x7fffffffu); };
  for (unsigned spins = 1; !arrived(); ++spins) {
    if (spins % 64) continue;
    sched_yield();
    const cudaError_t e = cudaStreamQuery(st);
    if (e != cudaErrorNotReady && !arrived()) return fail(QMM_ERR_CUDA, "moe_experts: the sort did not report: %s", cudaGetErrorString(e));
  }
  const bool out_of_range = *report.word & 1u;
  give_back(report);
  return out_of_range ? fail(QMM_ERR_SHAPE, "moe_experts: an expert index is outside [0, %d)", block->experts) : QMM_OK;
}
