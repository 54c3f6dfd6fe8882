"""The copy threads of the host-pointer calls (csrc/staging.h), compiled by itself and run on the CPU."""
import os
import re
import subprocess

from theano_b200 import build

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include <sys/resource.h>
#include <algorithm>
#include <vector>
%s
#include "staging.h"
using namespace b200;
static int check(int threads) {
  CopyPool pool(threads);
  const size_t sizes[] = {1, 63, 64, 4095, 4096, 131071, 131072, 131073, 1 << 20, (2 << 20) - 1, (2 << 20) + 1, (16 << 20) + 12345};
  std::vector<char> src(17 << 20), raw(17 << 20), back(17 << 20);
  for (size_t i = 0; i < src.size(); ++i) src[i] = static_cast<char>(i * 2654435761u >> 13);
  char* pinned = raw.data() + (64 - reinterpret_cast<uintptr_t>(raw.data()) %% 64) %% 64;      // as a ring slot: aligned
  for (size_t n : sizes)
    for (size_t off : {0, 1, 5000}) {
      std::fill(back.begin(), back.end(), 'x');
      std::fill(raw.begin(), raw.end(), 'y');
      pool.copy(pinned, src.data() + off, n, true);
      if (memcmp(pinned, src.data() + off, n) || pinned[n] != 'y') return 1;
      pool.touch(back.data() + off, n);
      for (char c : back)
        if (c != 'x') return 2;
      pool.copy(back.data() + off, pinned, n, false);
      if (memcmp(back.data() + off, pinned, n) || back[off + n] != 'x' || (off && back[off - 1] != 'x')) return 3;
      pool.touch(back.data() + off, n);
      if (memcmp(back.data() + off, pinned, n)) return 4;
    }
  return 0;
}
int main(int argc, char**) {
  if (argc > 1) {                     // no room for the stacks of more threads
    std::vector<char> room(64 << 20);
    rlimit lim = {1 << 20, 1 << 20};
    if (setrlimit(RLIMIT_AS, &lim)) return 1;
    CopyPool pool(8);
    std::fill(room.begin(), room.begin() + (16 << 20), 'z');
    pool.copy(room.data() + (32 << 20), room.data(), 16 << 20, true);
    puts(memcmp(room.data() + (32 << 20), room.data(), 16 << 20) ? "wrong" : "ok");
    return 0;
  }
  for (int threads : {1, 2, 8})
    if (int rc = check(threads)) { printf("%%d threads: %%d\n", threads, rc); return 1; }
  puts("ok");
}
"""


def run(tmp_path, before="", args=()):
    src, exe = tmp_path / "staging.cpp", tmp_path / "staging"
    src.write_text(PROGRAM % before)
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-pthread", "-I", build.CSRC, str(src), "-o", str(exe)])
    return subprocess.run([str(exe)] + list(args), stdout=subprocess.PIPE, timeout=120).stdout.decode().strip()


def test_copies_and_touches_over_sizes_and_offsets(tmp_path):
    assert run(tmp_path) == "ok"


def test_other_processors_copy_with_memcpy(tmp_path):
    """Without x86 (its macro taken away once the system's headers are in), no x86 header or instruction is needed."""
    headers = ["stdint.h", "string.h", "sys/mman.h", "atomic", "chrono", "condition_variable", "mutex", "system_error", "thread"]
    before = "".join("#include <%s>\n" % h for h in headers) + "#undef __x86_64__\n"
    assert run(tmp_path, before) == "ok"
    staging = open(os.path.join(build.CSRC, "staging.h")).read()
    guarded = staging[staging.index("#if defined(__x86_64__)\ninline"):staging.index("#else")]
    rest = staging.replace(guarded, "").replace("#if defined(__x86_64__)\n#include <immintrin.h>\n#endif\n", "")
    assert not re.search(r"_mm_|_mm256_|immintrin|cpuid|__asm__", rest)


def test_threads_that_cannot_be_made_are_done_without(tmp_path):
    assert run(tmp_path, args=["no-threads"]) == "ok"
