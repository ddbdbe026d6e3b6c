// Host plumbing of the C ABI: thread-local error text, device queries, TMA tensor-map construction.
#include <cudaTypedefs.h>

#include <atomic>
#include <mutex>

#include "common.cuh"

namespace b2 {
namespace {
thread_local std::string g_last_error;
}

void set_last_error(const std::string& msg) { g_last_error = msg; }

int fail_status(int status, const char* op, const std::string& msg) {
  g_last_error = std::string("owoinfer_b200::") + op + ": " + msg;
  return status;
}
int fail_invalid(const char* op, const std::string& msg) { return fail_status(B2_ERR_INVALID_ARGUMENT, op, msg); }
int fail_cuda(const char* op, cudaError_t e) {
  return fail_status(B2_ERR_CUDA, op, std::string("CUDA error: ") + cudaGetErrorName(e) + " (" + cudaGetErrorString(e) + ")");
}

namespace {
struct Chain {
  cudaStream_t stream = nullptr;
  bool open = false;
  int launches = 0;
};
thread_local Chain g_chain;
}  // namespace

LaunchChain::LaunchChain(cudaStream_t stream) : outer_(!g_chain.open) {
  if (outer_) g_chain = Chain{stream, true, 0};
}
LaunchChain::~LaunchChain() {
  if (outer_) g_chain = Chain{};
}
bool in_chain(cudaStream_t stream) { return g_chain.open && g_chain.stream == stream; }
bool chain_follows(cudaStream_t stream) { return in_chain(stream) && g_chain.launches++ > 0; }

int sm_count() {
  static std::atomic<int> cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  int n = cached[dev].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

bool make_tensor_map_2d(CUtensorMap* map, const void* base, std::uint64_t inner, std::uint64_t rows,
                        std::uint64_t row_stride, std::uint32_t inner_box, std::uint32_t row_box, const char* op,
                        int swizzle_bytes) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
  });
  if (encode == nullptr) {
    fail_status(B2_ERR_CUDA, op, "cuTensorMapEncodeTiled is not available from this driver");
    return false;
  }
  const cuuint64_t dims[2] = {inner, rows};
  const cuuint64_t strides[1] = {row_stride};
  const cuuint32_t box[2] = {inner_box, row_box};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, elem,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                            CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fail_status(B2_ERR_CUDA, op, "cuTensorMapEncodeTiled failed with code " + std::to_string(static_cast<int>(r)) +
                                     " (inner " + std::to_string(inner) + ", rows " + std::to_string(rows) + ", stride " +
                                     std::to_string(row_stride) + ")");
    return false;
  }
  return true;
}

}  // namespace b2

extern "C" {

const char* b2_last_error_message(void) { return b2::g_last_error.c_str(); }

uint32_t b2_numerics_version(int which) {
  // 0, 1, 3: bit-identical to the reference kernels of these versions. 2: the attention output follows the reference's
  // version-1 contract inside its tolerances but is produced by a different kernel (P is rounded against a lazily raised
  // maximum), so the high half carries this library's own revision of that kernel.
  constexpr std::uint32_t kInt8 = 1, kInt4 = 1, kAttention = (2u << 16) | 1u, kGroupedDecode = 1;
  switch (which) {
    case 0: return kInt8;
    case 1: return kInt4;
    case 2: return kAttention;
    case 3: return kGroupedDecode;
    default: return 0;
  }
}

}  // extern "C"
