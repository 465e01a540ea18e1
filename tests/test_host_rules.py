"""Rules of the host code and the kernels that are plain C++: compiled here with
the host compiler and run (no GPU needed)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run(tmp_path, header, body):
    src = tmp_path / "rule.cpp"
    src.write_text('#include <cstdio>\n#include "%s"\nint main() {\n%s\n}\n' % (header, body))
    exe = str(tmp_path / "rule")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "dust_b200", "csrc"),
                    str(src), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [int(x) for x in out.split()]


def test_near_list_sizes(tmp_path):
    """The list never asks for more than its limit, holds no more than all
    pairs, and stays as it is where the pairs would not fit."""
    limit = 40 * 2 ** 30 // 8
    seen = 1_500_000 * 14_600  # 175 GB of pairs
    got = run(tmp_path, "near_list.h", """
      const size_t lim = %dull;
      printf("%%zu %%zu %%zu %%zu\\n", near_list_first(2000000, 14596, lim),
             near_list_first(1000, 40, lim), near_list_first(2000000, 14596, 1000),
             near_list_first(1000000000, 14596, lim));
      printf("%%zu %%zu %%zu %%zu\\n", near_list_next(1000, 1000, lim),
             near_list_next(1000, 1001, lim), near_list_next(192000000, %dull, lim),
             near_list_next(1000, lim - 1, lim));""" % (limit, seen))
    assert got == [192_000_000, 40_000, 1000, limit, 1000, 1001 + 250 + 1024, 192_000_000, limit]
