// Host-side copies of the host-buffer calls.
//
// A call with numpy frames (the reference's own call pattern) moves each frame into a
// pinned staging buffer before its asynchronous upload and each result out of one after
// its download.  One core's memcpy moves ~16 GB/s, so four 4 MB planes cost ~1 ms per
// 1024^2 pair, more than the uploads themselves.  of_host_copy splits a large copy over a
// small persistent pool of threads (the caller copies one slice itself).  Python reaches
// it through ctypes, which releases the interpreter lock for the call.
//
// of_host_stage is the copy into an upload's staging buffer.  Its stores go past the caches:
// the upload reads what was just written, and reading lines that are dirty in the caches of
// several cores is slow: a 4 MB plane staged by 1, 2, 4, 8 threads with ordinary stores
// uploads in 98, 244, 523, 717 us, with streaming stores in 88 us whatever their number.
#if defined(__x86_64__)
#include <emmintrin.h>
#endif
#include <stdint.h>
#include <string.h>
#include <unistd.h>

#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"

namespace {

// memcpy with streaming stores.
void copy_streaming(char* dst, const char* src, size_t n) {
#if defined(__x86_64__)
  const size_t head = (16 - ((uintptr_t)dst & 15)) & 15;
  if (n >= 256) {
    memcpy(dst, src, head);
    size_t i = head;
    for (; i + 64 <= n; i += 64) {
      const __m128i* s = reinterpret_cast<const __m128i*>(src + i);
      __m128i* d = reinterpret_cast<__m128i*>(dst + i);
      const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1), c = _mm_loadu_si128(s + 2),
                    e = _mm_loadu_si128(s + 3);
      _mm_stream_si128(d, a);
      _mm_stream_si128(d + 1, b);
      _mm_stream_si128(d + 2, c);
      _mm_stream_si128(d + 3, e);
    }
    memcpy(dst + i, src + i, n - i);
    _mm_sfence();  // streaming stores are ordered by the storing thread
    return;
  }
#endif
  memcpy(dst, src, n);
}

class CopyPool {
 public:
  static CopyPool& get() {
    static CopyPool* p = new CopyPool();  // never destroyed: workers may outlive static teardown
    return *p;
  }
  bool usable() const { return getpid() == pid_; }  // a forked child has none of the workers
  void copy(char* dst, const char* src, size_t bytes, bool streaming) {
    std::lock_guard<std::mutex> one(call_mu_);  // one pooled copy at a time
    {
      std::lock_guard<std::mutex> g(mu_);
      dst_ = dst;
      src_ = src;
      bytes_ = bytes;
      streaming_ = streaming;
      pending_ = (int)workers_.size();
      ++gen_;
    }
    cv_.notify_all();
    part(0);
    std::unique_lock<std::mutex> g(mu_);
    done_.wait(g, [&] { return pending_ == 0; });
  }

 private:
  CopyPool() : pid_(getpid()) {
    unsigned hc = std::thread::hardware_concurrency();
    int n = hc > 1 ? (int)(hc / 2) : 1;
    if (n > 8) n = 8;
    parts_ = n;
    for (int i = 1; i < n; i++) workers_.emplace_back([this, i] { loop(i); });
    for (auto& t : workers_) t.detach();
  }
  void part(int i) const {
    size_t per = (bytes_ + parts_ - 1) / parts_;
    per = (per + 4095) & ~(size_t)4095;  // page-aligned slices
    const size_t b = (size_t)i * per;
    if (b >= bytes_) return;
    const size_t e = b + per < bytes_ ? b + per : bytes_;
    if (streaming_)
      copy_streaming(dst_ + b, src_ + b, e - b);
    else
      memcpy(dst_ + b, src_ + b, e - b);
  }
  void loop(int i) {
    unsigned seen = 0;
    for (;;) {
      std::unique_lock<std::mutex> g(mu_);
      cv_.wait(g, [&] { return gen_ != seen; });
      seen = gen_;
      g.unlock();
      part(i);
      g.lock();
      if (--pending_ == 0) done_.notify_one();
    }
  }

  const pid_t pid_;
  int parts_ = 1;
  std::vector<std::thread> workers_;
  std::mutex call_mu_, mu_;
  std::condition_variable cv_, done_;
  char* dst_ = nullptr;
  const char* src_ = nullptr;
  size_t bytes_ = 0;
  bool streaming_ = false;
  int pending_ = 0;
  unsigned gen_ = 0;
};

}  // namespace

static int host_copy(const char* what, void* dst, const void* src, size_t bytes, bool streaming) {
  OF_REQUIRE(bytes == 0 || (dst && src), "%s: null buffer", what);
  OF_REQUIRE(bytes == 0 || (const char*)dst + bytes <= (const char*)src || (const char*)src + bytes <= (const char*)dst,
             "%s: the buffers overlap", what);
  char* d = static_cast<char*>(dst);
  const char* s = static_cast<const char*>(src);
  if (bytes >= ((size_t)1 << 20) && CopyPool::get().usable())
    CopyPool::get().copy(d, s, bytes, streaming);
  else if (bytes && streaming)
    copy_streaming(d, s, bytes);
  else if (bytes)
    memcpy(d, s, bytes);
  return OF_OK;
}

extern "C" int of_host_copy(void* dst, const void* src, size_t bytes) {
  return host_copy("of_host_copy", dst, src, bytes, false);
}

extern "C" int of_host_stage(void* dst, const void* src, size_t bytes) {
  return host_copy("of_host_stage", dst, src, bytes, true);
}
