// qd_staging.h -- the host side of the copies between the caller's arrays and
// the device: worker threads, the NaN/Inf scan and the page-locked staging
// buffers.  No device code: it compiles as plain C++.
#pragma once
#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>
#include <sys/mman.h>
#include <unistd.h>
#ifdef __SSE2__
#include <emmintrin.h>
#endif

// Host worker threads for the input checks and the staging copies: created
// once per process (up to 16, the calling thread included; fewer where the
// system refuses more) and reused, so a 32 MiB chunk costs no thread creation.
// run(fn) calls fn(t) for every worker t and returns when all are done; callers
// take turns.  In a process forked after the pool was made (its workers do not
// exist there) the calling thread does every part itself.
class HostPool {
 public:
  static HostPool &get()
  {
    static HostPool *p = new HostPool();   // never destroyed: workers may outlive exit
    return *p;
  }
  unsigned size() const { return (unsigned)th_.size() + 1; }
  template <typename F> void run(const F &fn)
  {
    std::lock_guard<std::mutex> turn(run_mu_);
    if (th_.empty() || getpid() != pid_) {
      for (unsigned t = 0; t < size(); t++) fn(t);
      return;
    }
    const std::function<void(unsigned)> job = fn;
    {
      std::lock_guard<std::mutex> l(m_);
      job_ = &job;
      pending_ = th_.size();
      gen_++;
    }
    cv_.notify_all();
    fn(0);
    std::unique_lock<std::mutex> l(m_);
    done_.wait(l, [&] { return pending_ == 0; });
    job_ = nullptr;
  }

 private:
  HostPool() : pid_(getpid())
  {
    const unsigned hw = std::thread::hardware_concurrency();
    const unsigned n = std::max(1u, std::min(16u, hw ? hw : 1u));
    try {
      th_.reserve(n);
      for (unsigned t = 1; t < n; t++) th_.emplace_back([this, t] { loop(t); });
    } catch (const std::exception &) {
      // the system refuses more threads: the ones there are and the caller do the work
    }
  }
  void loop(unsigned t)
  {
    uint64_t seen = 0;
    for (;;) {
      const std::function<void(unsigned)> *f;
      {
        std::unique_lock<std::mutex> l(m_);
        cv_.wait(l, [&] { return gen_ != seen; });
        seen = gen_;
        f = job_;
      }
      (*f)(t);
      std::lock_guard<std::mutex> l(m_);
      if (--pending_ == 0) done_.notify_one();
    }
  }
  std::vector<std::thread> th_;
  pid_t pid_;
  std::mutex run_mu_, m_;
  std::condition_variable cv_, done_;
  const std::function<void(unsigned)> *job_ = nullptr;
  uint64_t gen_ = 0;
  size_t pending_ = 0;
};

// Inf and NaN are the doubles whose exponent field is all ones.  The scan
// ORs that test over the words without an early exit (so it stays a stream
// of independent loads), and splits arrays of a million or more words over
// the host pool: the check reads the whole input once per call and is bound
// by host memory bandwidth.
inline bool finite_words(const double *a, size_t n)
{
  constexpr uint64_t E = 0x7ff0000000000000ull;
  uint64_t b0 = 0, b1 = 0, b2 = 0, b3 = 0;
  size_t i = 0;
  for (; i + 4 <= n; i += 4) {
    uint64_t u[4];
    std::memcpy(u, a + i, sizeof u);
    b0 |= (u[0] & E) == E;
    b1 |= (u[1] & E) == E;
    b2 |= (u[2] & E) == E;
    b3 |= (u[3] & E) == E;
  }
  for (; i < n; i++) {
    uint64_t u;
    std::memcpy(&u, a + i, sizeof u);
    b0 |= (u & E) == E;
  }
  return (b0 | b1 | b2 | b3) == 0;
}

inline bool all_finite(const double *a, size_t n)
{
  if (n < (size_t(1) << 20)) return finite_words(a, n);
  HostPool &pool = HostPool::get();
  const unsigned nt = pool.size();
  const size_t chunk = (n + nt - 1) / nt;
  std::vector<char> ok(nt, 1);
  pool.run([&](unsigned t) {
    const size_t b = std::min(n, t * chunk), e = std::min(n, b + chunk);
    if (b < e) ok[t] = finite_words(a + b, e - b);
  });
  return std::all_of(ok.begin(), ok.end(), [](char c) { return c != 0; });
}

// Copies between the caller's (pageable) arrays and the device through
// page-locked staging buffers, allocated once per process and reused: host
// threads copy one chunk at a time into a staging buffer -- checking the
// words for NaN/Inf on the way when asked, while they are in cache -- and the
// copy engine moves each chunk as soon as it is staged, so the host copy of
// chunk c overlaps the transfer of chunk c - 1.  One transfer at a time per
// process; without page-locked memory the copies fall back to plain
// cudaMemcpyAsync from the caller's arrays.  The buffers serve every device; the
// events that guard them belong to one each, as an event can only be recorded on
// a stream of its own device.
class Staging {
 public:
  static constexpr size_t CHUNK = size_t(32) << 20;   // bytes per staging buffer
  static constexpr int NBUF = 4;
  static constexpr size_t LARGE = size_t(4) << 20;    // transfers from this size on use it
  // results of the set-up calls: staged from FETCH on where the array's pages are fresh,
  // as the copy threads share their faults, and from FETCH_WARM on where they are in memory
  // (a LEPS grid, us a call, plain and staged.  Fresh pages: 1.2 MB 260 and 405, 4.2 MB
  // 1500 and 1230, 8.4 MB 2400 and 1900, 33.6 MB 7600 and 4600; in memory: 2.1 MB 190
  // and 460, 8.4 MB 560 and 1440, 31.5 MB 1850 and 3500, 41.9 MB 2300 and 2700, 67 MB
  // 3900 and 2800)
  static constexpr size_t FETCH = size_t(2) << 20, FETCH_WARM = size_t(48) << 20;

  static Staging &get()
  {
    static Staging s;
    return s;
  }
  // an upload of `bytes` goes through the staging buffers, so upload() checks
  // its words while it copies them (inputs that are not staged are checked
  // before any device work)
  bool staged(size_t bytes)
  {
    std::lock_guard<std::mutex> lock(mu_);
    return bytes >= LARGE && ready();
  }
  // One host array of doubles for upload(): copied as doubles (their words
  // checked for NaN/Inf when `check`), or rounded to floats (`narrow`: always
  // checked for NaN, Inf and values beyond the FP32 range).
  struct Up {
    void *dst;            // device
    const double *src;    // host
    size_t n;             // doubles
    bool narrow = false;
    bool check = false;
  };
  // host -> device of several arrays as one stream of whole staging buffers
  // (a buffer holds the end of one array and the start of the next), so a
  // batch of mid-size arrays moves in as few chunks as its bytes need;
  // bad[i] = array i failed its check.  The staging buffers are taken in
  // turn across calls, so the host copy of one call's first chunk overlaps
  // the transfer of the previous call's last.
  cudaError_t upload(const Up *pc, int np, cudaStream_t st, std::vector<char> &bad)
  {
    bad.assign(np, 0);
    std::lock_guard<std::mutex> lock(mu_);
    if (!ready()) {
      for (int i = 0; i < np; i++) {
        if (pc[i].narrow) return cudaErrorMemoryAllocation;
        if (pc[i].check && !all_finite(pc[i].src, pc[i].n)) bad[i] = 1;
        cudaError_t e = cudaMemcpyAsync(pc[i].dst, pc[i].src, sizeof(double) * pc[i].n,
                                        cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return e;
      }
      return cudaSuccess;
    }
    int i = 0;
    size_t done = 0;                             // doubles of array i already staged
    while (i < np) {
      const int b = (int)(next_++ % NBUF);
      cudaError_t e = wait(b);   // the buffer's last transfer is done
      if (e != cudaSuccess) return e;
      size_t co = 0;                             // bytes of the buffer in use
      while (i < np) {
        const size_t w = pc[i].narrow ? sizeof(float) : sizeof(double);
        const size_t m = std::min(pc[i].n - done, (CHUNK - co) / w);
        if (m == 0 && done < pc[i].n) break;     // the buffer is full
        char *sb = static_cast<char *>(buf_[b]) + co;
        const bool ok = pc[i].narrow ? narrow_copy(reinterpret_cast<float *>(sb), pc[i].src + done, m)
                                     : copy_scan(sb, pc[i].src + done, m * w, pc[i].check);
        if (!ok) bad[i] = 1;
        if (m > 0) {
          e = cudaMemcpyAsync(static_cast<char *>(pc[i].dst) + done * w, sb, m * w,
                              cudaMemcpyHostToDevice, st);
          if (e != cudaSuccess) return e;
        }
        done += m;
        if (done == pc[i].n) {
          i++;
          done = 0;
        }
        co = (co + m * w + 63) & ~size_t(63);    // each part starts 64-byte aligned
        if (co >= CHUNK) break;
      }
      e = mark(b, st);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  // device -> host of one array; returns once dst holds the data
  cudaError_t download(void *dst, const void *src, size_t bytes, cudaStream_t st)
  {
    const Piece one{dst, src, bytes};
    return download(&one, 1, st);
  }
  // device -> host of several arrays as one stream of chunks (a chunk may
  // span the end of one array and the start of the next), so the transfers
  // of a batch of small arrays overlap the host copies as well
  struct Piece {
    void *dst;
    const void *src;
    size_t bytes;         // device bytes
    bool widen = false;   // src holds floats, dst receives them as doubles (2 x bytes)
  };
  cudaError_t download(const Piece *pc, int np, cudaStream_t st, size_t least = LARGE)
  {
    size_t total = 0;
    bool widen = false;
    for (int i = 0; i < np; i++) {
      total += pc[i].bytes;
      widen = widen || pc[i].widen;
    }
    // a small array alone needs no staging buffers: it makes none, and takes no turn at them
    std::unique_lock<std::mutex> turn(mu_, std::defer_lock);
    const bool small = !widen && np == 1 && total < least;
    if (!small) turn.lock();
    if (small || !ready()) {
      if (widen) return cudaErrorMemoryAllocation;
      for (int i = 0; i < np; i++) {
        cudaError_t e = cudaMemcpyAsync(pc[i].dst, pc[i].src, pc[i].bytes, cudaMemcpyDeviceToHost,
                                        st);
        if (e != cudaSuccess) return e;
      }
      return cudaStreamSynchronize(st);
    }
    const size_t nch = (total + CHUNK - 1) / CHUNK;
    // chunk c covers bytes [c*CHUNK, ...) of the concatenation; walk the pieces
    auto each_part = [&](size_t c, auto &&fn) {
      const size_t lo = c * CHUNK, hi = std::min(total, lo + CHUNK);
      size_t base = 0;
      for (int i = 0; i < np && base < hi; base += pc[i].bytes, i++) {
        const size_t a = std::max(lo, base), z = std::min(hi, base + pc[i].bytes);
        if (a < z) fn(i, a - base, a - lo, z - a);   // piece, offset in piece, in chunk, bytes
      }
    };
    auto issue = [&](size_t c) -> cudaError_t {
      const int b = (int)(c % NBUF);
      cudaError_t e = wait(b);
      each_part(c, [&](int i, size_t po, size_t co, size_t n) {
        if (e == cudaSuccess)
          e = cudaMemcpyAsync(static_cast<char *>(buf_[b]) + co,
                              static_cast<const char *>(pc[i].src) + po, n,
                              cudaMemcpyDeviceToHost, st);
      });
      if (e == cudaSuccess) e = mark(b, st);
      return e;
    };
    for (size_t c = 0; c < nch && c < (size_t)NBUF - 1; c++) {
      cudaError_t e = issue(c);
      if (e != cudaSuccess) return e;
    }
    for (size_t c = 0; c < nch; c++) {
      const int b = (int)(c % NBUF);
      cudaError_t e = wait(b);
      if (e != cudaSuccess) return e;
      each_part(c, [&](int i, size_t po, size_t co, size_t n) {
        if (pc[i].widen)
          widen_copy(static_cast<double *>(pc[i].dst) + po / sizeof(float),
                     reinterpret_cast<const float *>(static_cast<const char *>(buf_[b]) + co),
                     n / sizeof(float));
        else
          copy_scan(static_cast<char *>(pc[i].dst) + po, static_cast<const char *>(buf_[b]) + co,
                    n, false);
      });
      if (c + NBUF - 1 < nch) {
        e = issue(c + NBUF - 1);
        if (e != cudaSuccess) return e;
      }
    }
    next_ = 0;   // every buffer's event has completed
    return cudaSuccess;
  }

  // result of a set-up call, device -> host on the default stream; the wait for
  // the kernel leaves the staging buffers to other threads' copies
  cudaError_t fetch(void *dst, const void *src, size_t bytes)
  {
    if (bytes < FETCH || (bytes < FETCH_WARM && in_memory(dst, bytes)))
      return cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost);
    const cudaError_t e = cudaStreamSynchronize(nullptr);
    const Piece one{dst, src, bytes};
    return e == cudaSuccess ? download(&one, 1, nullptr, FETCH) : e;
  }

 private:
  Staging() = default;
  // most pages of [p, p + n) are in memory: 32 of them are looked at
  static bool in_memory(const void *p, size_t n)
  {
    constexpr int SAMPLES = 32;
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), at = reinterpret_cast<uintptr_t>(p);
    int in = 0;
    for (int i = 0; i < SAMPLES; i++) {
      unsigned char v = 0;
      if (mincore(reinterpret_cast<void *>((at + n / SAMPLES * i) & ~(page - 1)), 1, &v) == 0)
        in += v & 1;
    }
    return 2 * in > SAMPLES;
  }
  // the buffers, and the current device's events, exist (made on first use)
  bool ready()
  {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= MAXDEV) {
      cudaGetLastError();
      return false;
    }
    if (!tried_) {
      tried_ = ok_ = true;
      for (int b = 0; b < NBUF && ok_; b++)
        ok_ = cudaHostAlloc(&buf_[b], CHUNK, cudaHostAllocPortable) == cudaSuccess;
    }
    if (ok_ && !dev_tried_[dev]) {
      dev_tried_[dev] = dev_ok_[dev] = true;
      for (int b = 0; b < NBUF && dev_ok_[dev]; b++)
        dev_ok_[dev] = cudaEventCreateWithFlags(&ev_[dev][b], cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok_ || !dev_ok_[dev]) {
      cudaGetLastError();
      return false;
    }
    return true;
  }
  // buffer b's last transfer, whichever device it was on, is done
  cudaError_t wait(int b) { return last_[b] ? cudaEventSynchronize(last_[b]) : cudaSuccess; }
  // buffer b's last transfer is the one issued on st, a stream of the current device
  cudaError_t mark(int b, cudaStream_t st)
  {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    last_[b] = ev_[dev][b];
    return cudaEventRecord(last_[b], st);
  }
  // memcpy over the host pool, the stores streamed past the caches where the
  // destination is 16-byte aligned (no read of the destination lines); with
  // scan, also the NaN/Inf test of the copied words, on the loaded values
  static bool copy_scan(void *dst, const void *src, size_t n, bool scan)
  {
    HostPool &pool = HostPool::get();
    const unsigned nt = pool.size();
    const size_t part = (n / nt + 63) & ~size_t(63);
    std::vector<char> ok(nt, 1);
    pool.run([&](unsigned t) {
      const size_t a = std::min(n, t * part), z = t + 1 == nt ? n : std::min(n, a + part);
      if (a >= z) return;
      char *d = static_cast<char *>(dst) + a;
      const char *s = static_cast<const char *>(src) + a;
      const size_t len = z - a;
      size_t i = 0;
      uint64_t bad = 0;
#ifdef __SSE2__
      if ((reinterpret_cast<uintptr_t>(d) & 15) == 0) {
        constexpr uint64_t E = 0x7ff0000000000000ull;
        for (; i + 64 <= len; i += 64) {
          const __m128i *p = reinterpret_cast<const __m128i *>(s + i);
          const __m128i v0 = _mm_loadu_si128(p), v1 = _mm_loadu_si128(p + 1);
          const __m128i v2 = _mm_loadu_si128(p + 2), v3 = _mm_loadu_si128(p + 3);
          __m128i *q = reinterpret_cast<__m128i *>(d + i);
          _mm_stream_si128(q, v0);
          _mm_stream_si128(q + 1, v1);
          _mm_stream_si128(q + 2, v2);
          _mm_stream_si128(q + 3, v3);
          if (scan) {
            uint64_t u[8];
            std::memcpy(u, s + i, sizeof u);
            for (int k = 0; k < 8; k++) bad |= (u[k] & E) == E;
          }
        }
        _mm_sfence();
      }
#endif
      std::memcpy(d + i, s + i, len - i);
      if (scan)
        ok[t] = bad == 0 && finite_words(reinterpret_cast<const double *>(d + i), (len - i) / 8);
    });
    return std::all_of(ok.begin(), ok.end(), [](char c) { return c != 0; });
  }
  // dst[i] = (float)src[i] over the host pool; false if some src[i] is NaN,
  // Inf or beyond the FP32 range
  static bool narrow_copy(float *dst, const double *src, size_t n)
  {
    HostPool &pool = HostPool::get();
    const unsigned nt = pool.size();
    const size_t part = (n / nt + 15) & ~size_t(15);
    std::vector<char> ok(nt, 1);
    pool.run([&](unsigned t) {
      const size_t a = std::min(n, t * part), z = t + 1 == nt ? n : std::min(n, a + part);
      // |v| above FLT_MAX, Inf and NaN are the magnitudes above FLT_MAX's bits
      constexpr uint64_t MAGN = 0x7fffffffffffffffull, FMAX = 0x47efffffe0000000ull;
      uint64_t bad = 0;
      size_t i = a;
#ifdef __SSE2__
      // four values a round, streamed past the caches into the staging buffer
      // (dst + a is 16-byte aligned: a is a multiple of 16 and dst a page-locked buffer)
      for (; i + 4 <= z; i += 4) {
        const __m128d v0 = _mm_loadu_pd(src + i), v1 = _mm_loadu_pd(src + i + 2);
        _mm_stream_ps(dst + i, _mm_movelh_ps(_mm_cvtpd_ps(v0), _mm_cvtpd_ps(v1)));
        uint64_t u[4];
        std::memcpy(u, src + i, sizeof u);
        bad |= ((u[0] & MAGN) > FMAX) | ((u[1] & MAGN) > FMAX) | ((u[2] & MAGN) > FMAX) |
               ((u[3] & MAGN) > FMAX);
      }
      _mm_sfence();
#endif
      for (; i < z; i++) {
        uint64_t u;
        std::memcpy(&u, src + i, sizeof u);
        bad |= (u & MAGN) > FMAX;
        dst[i] = (float)src[i];
      }
      ok[t] = bad == 0;
    });
    return std::all_of(ok.begin(), ok.end(), [](char c) { return c != 0; });
  }
  // dst[i] = src[i] widened to double, over the host pool
  static void widen_copy(double *dst, const float *src, size_t n)
  {
    HostPool &pool = HostPool::get();
    const unsigned nt = pool.size();
    const size_t part = (n / nt + 15) & ~size_t(15);
    pool.run([&](unsigned t) {
      const size_t a = std::min(n, t * part), z = t + 1 == nt ? n : std::min(n, a + part);
      size_t i = a;
#ifdef __SSE2__
      // two values a round, streamed to the caller's array when it is 16-byte aligned
      if ((reinterpret_cast<uintptr_t>(dst + a) & 15) == 0) {
        for (; i + 2 <= z; i += 2) {
          const __m128 f = _mm_castsi128_ps(_mm_loadl_epi64(reinterpret_cast<const __m128i *>(src + i)));
          _mm_stream_pd(dst + i, _mm_cvtps_pd(f));
        }
        _mm_sfence();
      }
#endif
      for (; i < z; i++) dst[i] = (double)src[i];
    });
  }
  std::mutex mu_;
  static constexpr int MAXDEV = 64;
  bool tried_ = false, ok_ = false, dev_tried_[MAXDEV] = {}, dev_ok_[MAXDEV] = {};
  void *buf_[NBUF] = {};
  cudaEvent_t ev_[MAXDEV][NBUF] = {}, last_[NBUF] = {};
  size_t next_ = 0;               // the upload's next staging buffer (round robin)
};
