"""Index arithmetic of the launches at the limits of 32 bits: csrc/launch_math.h compiled for the host with checks for
overflow (no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, body):
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text('#include <cstdio>\n#include <cstdlib>\n#include <initializer_list>\n#include "launch_math.h"\nusing namespace pce;\n'
                   "static void need(bool ok, int line) { if (!ok) { std::printf(\"line %d\\n\", line); std::exit(1); } }\n"
                   "#define NEED(x) need((x), __LINE__)\nint main() {\n" + body + "\nreturn 0; }\n")
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=all", "-I",
                    os.path.join(ROOT, "pcengine_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], capture_output=True, text=True)
    assert done.returncode == 0, done.stdout + done.stderr


def test_blocks_of_the_tiled_fp32_kernel(tmp_path):
    """Row blocks beyond 65535 (the end of gridDim.y and z) and up to the last int32 row, channel slices beyond 65535: the
    blocks' rows and channels cover the output once, the last rows first, parts of a cluster next to each other."""
    _run(tmp_path, """
      const int rows[] = {1, 32, 33, 2097120, 2097121, 8388480, 8388481, 2147483647};
      const int widths[] = {1, 48, 49, 65535 * 48, 65535 * 48 + 1, 2147483647};
      for (int n : rows) for (int bm : {32, 128}) for (int lg : {0, 2, 3}) for (int c : widths) {
        if (lg > 0 && n > 100000000) continue;  // (clusters are for small maps)
        const F32Grid g = f32_grid(n, bm, c, 48, 1 << lg);
        const unsigned row_blocks = static_cast<unsigned>((static_cast<long long>(n) + bm - 1) / bm);
        NEED(g.x == row_blocks << lg && g.x <= 2147483647u && g.y >= 1 && g.y <= 65535u && g.z >= 1 && g.z <= 65535u);
        NEED(static_cast<long long>(g.y) * g.z * 48 >= c && (static_cast<long long>(g.y) * g.z - g.z) * 48 < c);
        const unsigned xs[] = {0u, 1u, (1u << lg) - 1u, 1u << lg, 65535u << lg, g.x - 1u};
        for (unsigned x : xs) {
          if (x >= g.x) continue;
          const F32Block p = f32_block(x, 0, 0, g, lg, bm, 48);
          NEED(p.part == static_cast<int>(x % (1u << lg)));
          NEED(p.row0 == static_cast<int>((row_blocks - 1 - x / (1u << lg)) * static_cast<unsigned>(bm)) && p.row0 < n && p.row0 + (bm - 1) >= 0);
        }
        const F32Block last = f32_block(0, g.y - 1, g.z - 1, g, lg, bm, 48), next = f32_block(0, 0, g.z - 1, g, lg, bm, 48);
        NEED(last.channel0 == (static_cast<long long>(g.y) * g.z - 1) * 48);
        if (g.z > 1) NEED(next.channel0 == f32_block(0, g.y - 1, g.z - 2, g, lg, bm, 48).channel0 + 48);
      }""")


def test_pieces_of_a_cooperative_grid(tmp_path):
    """Contiguous pieces cover every entry once, up to 2^31 - 1 entries, and a piece's walk in strides of a block's 2048
    entries (512 threads, four each) does not wrap around behind the last one."""
    _run(tmp_path, """
      const unsigned sizes[] = {1, 2, 4095, 4096, 4097, 2147479552u, 2147483639u, 2147483646u, 2147483647u};
      for (unsigned n : sizes) for (unsigned parts : {1u, 2u, 295u, 296u, 1024u}) {
        unsigned covered = 0;
        for (unsigned p = 0; p < parts; ++p) {
          const Piece a = piece_of(n, p, parts);
          NEED(a.first == covered && a.end >= a.first && a.end <= n);
          covered = a.end;
          const unsigned past = a.end + 2048u + 2048u;
          NEED(past > a.end);
        }
        NEED(covered == n);
      }""")
