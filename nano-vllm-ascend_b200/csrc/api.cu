// api.cu -- library-level entry points of libb200attn.so (version, errors, launch counter).
#include "common.cuh"

namespace b200 {
long long g_launch_count = 0;

int* wait_status() {
  static int* const word = [] {
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {   // nothing can be launched: the host side alone
      cudaGetLastError();
      static int host_only = 0;
      return &host_only;
    }
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;       // the first call may come while a stream is captured
    cudaThreadExchangeStreamCaptureMode(&mode);
    int* p = nullptr;
    if (cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) *p = 0;
    else cudaGetLastError(), p = nullptr;
    cudaThreadExchangeStreamCaptureMode(&mode);
    return p;
  }();
  return word;
}

bool take_wait_status() {
  int* word = wait_status();
  return word != nullptr && __atomic_load_n(word, __ATOMIC_RELAXED) != 0 && __atomic_exchange_n(word, 0, __ATOMIC_RELAXED) != 0;
}
}  // namespace b200

extern "C" int b200_version(void) { return B200ATTN_VERSION; }

extern "C" int64_t b200_launch_count(void) { return b200::g_launch_count; }
extern "C" void b200_reset_launch_count(void) { b200::g_launch_count = 0; }

extern "C" int b200_take_wait_status(void) { return b200::take_wait_status() ? B200_ERR_WAIT : B200_OK; }
extern "C" int32_t* b200_wait_status_word(void) { return b200::wait_status(); }

extern "C" const char* b200_error_string(int code) {
  switch (code) {
    case B200_OK: return "success";
    case B200_ERR_NULL_POINTER: return "b200attn: required pointer argument is NULL";
    case B200_ERR_BAD_SHAPE: return "b200attn: inconsistent or non-positive shape/stride argument";
    case B200_ERR_UNSUPPORTED:
      return "b200attn: unsupported configuration (head_dim must be 64/128, GQA group <= 8, "
             "kv heads in {1,2,4,8k}, block_size % 16 == 0)";
    case B200_ERR_MISALIGNED: return "b200attn: pointer or stride violates the alignment contract";
    case B200_ERR_WORKSPACE: return "b200attn: workspace too small";
    case B200_ERR_DRIVER: return "b200attn: cuTensorMapEncodeTiled unavailable or failed";
    case B200_ERR_BAD_DTYPE: return "b200attn: dtype must be B200_DTYPE_BF16 or B200_DTYPE_F16";
    case B200_ERR_WAIT: return "b200attn: a wait inside a kernel of an earlier call ran out; that call's output is not valid";
    default: break;
  }
  if (code > 0) return cudaGetErrorString((cudaError_t)code);
  return "b200attn: unknown error code";
}
