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


def test_p2p_items_cover_every_pair(tmp_path):
    """The items of a leaf hold each of its targets' sources once, also where
    longer pieces keep a large leaf to its share of the list."""
    cases = [(nt, S, it, cap) for nt in (1, 31, 32, 33, 70, 128) for S in (1, 64, 65, 700, 20001)
             for it, cap in ((64, 1 << 18), (3, 80), (64, 16))]
    body = "const unsigned c[][4] = {%s};\n" % ",".join("{%d,%d,%d,%d}" % c for c in cases)
    body += """for (auto &q : c) {
      const P2PCut k = p2p_cut(q[0], q[1], q[2], q[3]);
      printf("%llu\\n", (unsigned long long)k.ni);
      for (uint64_t e = 0; e < k.ni; ++e) {
        uint32_t tb, lo, hi;
        p2p_item(k, q[1], e, tb, lo, hi);
        printf("%u %u %u\\n", tb, lo, hi);
      }
    }"""
    got = iter(run(tmp_path, "p2p_items.h", body))
    for nt, S, it, cap in cases:
        ni = next(got)
        items = [(next(got), next(got), next(got)) for _ in range(ni)]
        blocks = -(-nt // 32)
        assert ni <= cap // 8 + blocks  # (pieces are rounded up once a block)
        for b in range(blocks):
            at = 0
            for lo, hi in (i[1:] for i in items if i[0] == 32 * b):
                assert lo == at and hi > lo
                at = hi
            assert at == S
        assert all(i[0] % 32 == 0 and i[0] < nt for i in items)


def test_p2p_items_of_a_huge_leaf(tmp_path):
    """Counts beyond 32 bits: 3.1 million particles in one leaf (4.7e9 pieces of
    64 sources) and the largest leaf there can be."""
    got = run(tmp_path, "p2p_items.h", """
      const unsigned n[] = {23000u, 3100000u, 2147483647u};
      for (unsigned x : n) {
        const P2PCut c = p2p_cut(x, x, 64, 1u << 18);
        uint32_t tb, lo, hi;
        p2p_item(c, x, c.ni - 1, tb, lo, hi);
        printf("%llu %u %u %u %u\\n", (unsigned long long)c.ni, c.it, tb, lo < hi, hi);
      }""")
    for k, n in enumerate((23000, 3100000, 2147483647)):
        ni, it, tb, some, hi = got[5 * k:5 * k + 5]
        assert ni == n // 32 * -(-n // it) + (1 if n % 32 else 0) * -(-n // min(it * (32 // max(n % 32, 1)), n))
        assert tb == (n - 1) // 32 * 32 and some and hi == n
        assert ni <= (1 << 15) + -(-n // 32)
