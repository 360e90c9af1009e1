"""The tables of the state-tile kernels (crs_fx_build.cpp), built on the host
from mechanisms' table images (CPU)."""
import ctypes
import os
import shutil
import subprocess

import pytest

from conftest import GOLDEN_CASES, REPO
from create_rate_subs_gb300 import _lib

CSRC = os.path.join(REPO, "create_rate_subs_gb300", "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include "crs_fx_tab.cuh"
static std::vector<unsigned char> read(const std::string &name) {
  std::vector<unsigned char> v;
  FILE *f = fopen(name.c_str(), "rb");
  for (int c; (c = fgetc(f)) != EOF;) v.push_back((unsigned char)c);
  fclose(f);
  return v;
}
int main(int, char **argv) {
  const std::vector<unsigned char> img = read(argv[1]), lay = read(argv[2]);
  crs::ImgLayout L;
  memcpy(&L, lay.data(), sizeof L);
  const crs::Tab t = crs::make_tab(img.data(), L);
  crs::fx::FxTab f;
  std::vector<unsigned char> out;
  crs::fx::build(t, f, out);
  printf("%d %d %zu", f.usable, f.mixed, out.size());
  const size_t n = out.size();
  for (int64_t limit : {(int64_t)n - 1, 2 * (int64_t)n + (1 << 17)}) {
    crs::fx::build(t, f, out, limit);
    printf(" %d %zu", f.usable || f.mixed, out.size());
  }
  printf("\n");
}
"""


@pytest.fixture(scope="module")
def tool(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("fx_tables")
    (d / "t.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, str(d / "t.cpp"),
                    os.path.join(CSRC, "crs_fx_build.cpp"), "-o", str(d / "t")], check=True)

    def run(mech):
        lib = _lib.load()
        blob, s = mech.blob, (ctypes.c_size_t * 2)()
        _lib.check(lib.crs_mech_image(blob, len(blob), None, 0, None, 0, s))
        img, lay = ctypes.create_string_buffer(s[0]), (ctypes.c_int32 * s[1])()
        _lib.check(lib.crs_mech_image(blob, len(blob), img, s[0], lay, s[1], s))
        (d / "img").write_bytes(img.raw)
        (d / "lay").write_bytes(bytes(lay))
        out = subprocess.run([str(d / "t"), str(d / "img"), str(d / "lay")], check=True,
                             capture_output=True, text=True).stdout
        return [int(v) for v in out.split()]
    return run


@pytest.mark.parametrize("name", GOLDEN_CASES + ("large561",))
def test_no_table_beyond_the_limit(name, tool, golden, synth_mech):
    """The bound that keeps the tables' 32-bit offsets in range: tables that
    might pass a limit are not built, those that stay well below it are."""
    mech = synth_mech(name) if name == "large561" else golden(name)[0]
    usable, mixed, size, on_below, size_below, on_above, size_above = tool(mech)
    assert (on_below, size_below) == (0, 0)
    assert size_above == size and on_above == (usable or mixed)
    if not name.startswith("features"):
        assert usable and mixed


@pytest.mark.parametrize("change,usable", [
    (lambda a, b, e: (a, b, e), True),
    # log2 of the constant beyond 800 at the middle of an interval: the sum of a
    # rate's exponents might leave 64 bits
    (lambda a, b, e: (1e-290, b, e), False),
    (lambda a, b, e: (1e-60, -95.0, e), False),
    # terms beyond 500
    (lambda a, b, e: (a, b, 4e5), False)])
def test_constants_outside_the_range_are_general(change, usable, tool, tmp_path):
    """Rate constants that the fixed-point sums do not hold are left to the
    general arithmetic; with all of them outside, the tables are not used."""
    from create_rate_subs_gb300 import synth
    from create_rate_subs_gb300.mechanism import Mechanism
    text, therm = synth.make_mechanism(**synth.CONFIGS["small"])
    lines = []
    for line in text.split("\n"):
        w = line.split()
        if "=" in line:
            line = "%-40s %13.6E %8.3f %10.1f" % ((w[0],) + change(*map(float, w[1:])))
        lines.append(line)
    mp, tp = tmp_path / "mech.inp", tmp_path / "therm.dat"
    mp.write_text("\n".join(lines))
    tp.write_text(therm)
    assert tool(Mechanism.from_chemkin(str(mp), str(tp)))[0] == usable
