"""The per-thread store of projection plans (csrc/recent.h): the sizes of a model's pass stay in it from one pass to the next.
The header is plain C++, so it is compiled here with the host compiler."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "distributed-llm-inferencing_b200", "csrc")
PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include "recent.h"
struct Key { int M, N, K; bool operator==(const Key& o) const { return M == o.M && N == o.N && K == o.K; } };
int main(int argc, char** argv) {  // argv: M, then N K pairs; prints how many of a second pass's look-ups miss
  dli::RecentResults<Key, int, 32> store;
  int misses[2] = {0, 0};
  for (int pass = 0; pass < 2; ++pass)
    for (int i = 2; i + 1 < argc; i += 2) {
      const Key k{atoi(argv[1]), atoi(argv[i]), atoi(argv[i + 1])};
      const int* v = store.find(k);
      if (v == nullptr) { ++misses[pass]; store.put(k, i); }
      else if (*v != i) return 2;
    }
  printf("%d %d\n", misses[0], misses[1]);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("recent")
    (d / "t.cc").write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(d / "t.cc"), "-o", str(d / "t")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("name", ["llama-3-8b", "mistral-7b", "tinyllama-1.1b", "llama-3-70b", "gpt2"])
@pytest.mark.parametrize("M", [3, 19, 301, 1024])
def test_a_second_pass_finds_every_plan(program, name, M):
    from dli_b200.engine import NAMED_SPECS

    s = NAMED_SPECS[name]
    d, hd = s.d_model, s.head_dim
    up = (2 if s.arch == "llama" else 1) * s.d_ff
    sizes = [((s.n_heads + 2 * s.n_kv_heads) * hd, d), (d, s.n_heads * hd), (up, d), (d, s.d_ff), (s.vocab, d)]
    out = subprocess.run([program, str(M)] + [str(v) for nk in sizes for v in nk], check=True, capture_output=True, text=True)
    first, second = map(int, out.stdout.split())
    assert first == len(set(sizes)) and second == 0


def test_the_oldest_goes_first(program):
    """33 sizes in a store of 32: each pass drives out what the next one asks for first, none is answered wrongly."""
    args = [str(v) for i in range(33) for v in (64 * i, 64)]
    out = subprocess.run([program, "7"] + args, check=True, capture_output=True, text=True)
    assert out.stdout.split() == ["33", "33"]
