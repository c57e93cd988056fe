// Status words for the calls without a handle (hodlr_gemm_broadcast,
// hodlr_gemm_reduce and its variant that allocates nothing): the digit products
// they run wait on mbarriers, and a wait that expired has to reach the caller.
//
// A file-scope array, since one of the callers may not allocate and the others
// are short: a word of its own for every call in progress, handed out under a
// mutex.  The array's address is looked up on every call (a table lookup), so a
// device that was reset in between is no trouble.
#include <condition_variable>
#include <mutex>
#include <string>

#include "kernels.cuh"

namespace hodlr {

constexpr int kWords = 64;
static __device__ DevStatus g_words[kWords];

static std::mutex g_mu;
static std::condition_variable g_freed;
static unsigned long long g_taken = 0;  // bit i: word i, on whichever device

static thread_local long long g_waiting_launches = 0;
void note_waiting_launch() { ++g_waiting_launches; }

CallStatus::CallStatus() {
  std::unique_lock<std::mutex> lock(g_mu);
  g_freed.wait(lock, [] { return ~g_taken != 0; });
  slot_ = 0;
  while (g_taken >> slot_ & 1) ++slot_;
  g_taken |= 1ull << slot_;
}

// A free word is zero: whoever finds it set, or leaves with work on the stream, clears it.
CallStatus::~CallStatus() {
  if (word_) {
    (void)cudaMemsetAsync(word_, 0, sizeof(DevStatus), 0);
    (void)cudaStreamSynchronize(0);
  }
  {
    std::lock_guard<std::mutex> lock(g_mu);
    g_taken &= ~(1ull << slot_);
  }
  g_freed.notify_one();
}

cudaError_t CallStatus::find() {
  void *p = nullptr;
  launches_ = g_waiting_launches;
  const cudaError_t e = cudaGetSymbolAddress(&p, g_words);
  if (e == cudaSuccess) word_ = static_cast<DevStatus *>(p) + slot_;
  return e;
}

int CallStatus::finish(const char *call) {
  DevStatus s{};
  cudaError_t e = cudaSuccess;
  if (launches_ != g_waiting_launches) e = cudaMemcpyAsync(&s, word_, sizeof s, cudaMemcpyDeviceToHost, 0);
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  if (e != cudaSuccess) return set_last_error(HODLR_ERR_CUDA, cudaGetErrorString(e));
  if (s.code == HODLR_OK) {
    word_ = nullptr;
    return HODLR_OK;
  }
  const std::string what = std::string(call) + ": device wait timed out (index " + std::to_string(s.index) + ")";
  return set_last_error(s.code, what.c_str());
}

}  // namespace hodlr
