"""The host side of the staged copies (csrc/qd_staging.h), compiled against the
stand-in runtime of tests/fake_runtime: one program per property.
"""
import os
import subprocess

import pytest

from conftest import PKG, REPO

PRELUDE = r"""
#include "qd_staging.h"
#include <cstdio>
#define CHECK(x) do { if (!(x)) { std::printf("failed: %s\n", #x); return 1; } } while (0)
typedef std::vector<double> V;
static V ramp(size_t n) { V a(n); for (size_t i = 0; i < n; i++) a[i] = 0.5 * i; return a; }
"""


def run(tmp_path, body, *flags):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PRELUDE + body)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", *flags,
                    f"-I{os.path.join(REPO, 'tests', 'fake_runtime')}",
                    f"-I{os.path.join(PKG, 'csrc')}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("first,second", [(0, 1), (1, 0), (3, 2)])
def test_devices_in_turn(tmp_path, first, second):
    # several chunks up and down on one device, then on another, then on the first again
    run(tmp_path, """
    int main() {
      Staging &s = Staging::get();
      const V a = ramp((size_t(40) << 20) / 8);
      for (int dev : {%d, %d, %d}) {
        CHECK(cudaSetDevice(dev) == cudaSuccess);
        V up(a.size()), down(a.size());
        const Staging::Up u{up.data(), a.data(), a.size(), false, true};
        std::vector<char> bad;
        FakeHandle st{dev};
        CHECK(s.staged(8 * a.size()));
        CHECK(s.upload(&u, 1, &st, bad) == cudaSuccess);
        CHECK(!bad[0] && up == a);
        CHECK(s.download(down.data(), up.data(), 8 * a.size(), &st) == cudaSuccess);
        CHECK(down == a);
        V dflt(a.size());
        CHECK(s.download(dflt.data(), up.data(), 8 * a.size(), nullptr) == cudaSuccess);
        CHECK(dflt == a);
      }
      return 0;
    }""" % (first, second, first))


def test_small_fetch_pins_nothing(tmp_path):
    run(tmp_path, """
    int main() {
      Staging &s = Staging::get();
      const V a = ramp(1000);
      V b(a.size());
      CHECK(s.download(b.data(), a.data(), 8 * a.size(), nullptr) == cudaSuccess);
      CHECK(b == a);
      CHECK(fake::pinned == 0);
      const V big = ramp(Staging::LARGE / 8);       // the smallest array that is staged
      V c(big.size());
      CHECK(s.download(c.data(), big.data(), 8 * big.size(), nullptr) == cudaSuccess);
      CHECK(c == big);
      CHECK(fake::pinned == (long)(Staging::NBUF * Staging::CHUNK));
      return 0;
    }""")


@pytest.mark.parametrize("mib", [1, 3, 8])
def test_waiting_for_a_kernel_delays_no_other_copy(tmp_path, mib):
    # a fetch whose kernel is still running (the stream's synchronise does not return)
    # leaves the staging buffers to another thread's copies
    run(tmp_path, """
    #include <chrono>
    int main() {
      Staging &s = Staging::get();
      const V a = ramp((size_t(%d) << 20) / 8), up = ramp((size_t(8) << 20) / 8);
      std::mutex m;
      std::condition_variable cv;
      bool waiting = false, uploaded = false, in_time = false;
      fake::on_stream_sync = [&] {
        std::unique_lock<std::mutex> l(m);
        if (waiting) return;                       // the fetch's first wait: its kernel
        waiting = true;
        cv.notify_all();
        in_time = cv.wait_for(l, std::chrono::seconds(10), [&] { return uploaded; });
      };
      V got(a.size()), dst(up.size());
      cudaError_t e = cudaErrorInvalidValue;
      std::thread t([&] { e = s.fetch(got.data(), a.data(), 8 * a.size()); });
      {
        std::unique_lock<std::mutex> l(m);
        CHECK(cv.wait_for(l, std::chrono::seconds(10), [&] { return waiting; }));
      }
      const Staging::Up u{dst.data(), up.data(), up.size(), false, true};
      std::vector<char> bad;
      CHECK(s.upload(&u, 1, nullptr, bad) == cudaSuccess);
      { std::lock_guard<std::mutex> l(m); uploaded = true; }
      cv.notify_all();
      t.join();
      CHECK(in_time && e == cudaSuccess && got == a && dst == up);
      return 0;
    }""" % mib)


@pytest.mark.parametrize("threads", [0, 1, 5])
def test_fewer_worker_threads_than_asked_for(tmp_path, threads):
    # the system gives `threads` threads and refuses the others
    run(tmp_path, """
    #include <cerrno>
    #include <dlfcn.h>
    #include <pthread.h>
    static int given = 0;
    extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *p) {
      typedef int (*Fn)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
      static Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
      return given < %d ? (given++, real(t, a, f, p)) : EAGAIN;
    }
    int main() {
      const V a = ramp((size_t(5) << 20) / 8);
      V b(a.size());
      CHECK(Staging::get().download(b.data(), a.data(), 8 * a.size(), nullptr) == cudaSuccess);
      CHECK(b == a && given <= %d && all_finite(a.data(), a.size()));
      return 0;
    }""" % (threads, threads), "-rdynamic", "-D_GNU_SOURCE")


def test_results_into_warm_pages_are_not_staged(tmp_path):
    # an array whose pages are in memory: a plain copy up to FETCH_WARM; a fresh mapping of
    # the same size: staged
    run(tmp_path, """
    #include <sys/mman.h>
    int main() {
      Staging &s = Staging::get();
      const size_t n = size_t(8) << 20;
      const V a = ramp(n / 8);
      V warm(n / 8);
      CHECK(s.fetch(warm.data(), a.data(), n) == cudaSuccess && warm == a);
      CHECK(s.fetch(warm.data() + 1, a.data(), n - 8) == cudaSuccess && warm[1] == a[0]);
      CHECK(fake::pinned == 0);
      double *f = (double *)mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
      CHECK(f != MAP_FAILED && s.fetch(f, a.data(), n) == cudaSuccess);
      CHECK(std::equal(a.begin(), a.end(), f) && fake::pinned > 0);
      return 0;
    }""")
