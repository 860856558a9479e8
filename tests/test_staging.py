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
