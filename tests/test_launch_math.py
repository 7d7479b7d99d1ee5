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
    """Row blocks beyond 65535 (the end of gridDim.y) and up to the last int32 row: every block has one place, in the
    order parts, row blocks, slices, and the rows it names stay within int32."""
    _run(tmp_path, """
      const int rows[] = {1, 32, 33, 2097120, 2097121, 8388480, 8388481, 2147483647};
      for (int n : rows) for (int bm : {32, 128}) for (int parts : {1, 4, 8}) for (int slices : {1, 3}) {
        if (parts > 1 && n > 100000000) continue;  // (clusters are for small maps)
        const long long blocks = f32_blocks(n, bm, slices * 48, 48, parts);
        const int row_blocks = static_cast<int>((static_cast<long long>(n) + bm - 1) / bm);
        NEED(blocks == static_cast<long long>(row_blocks) * slices * parts && blocks <= 2147483647ll);
        const long long probes[] = {0, 1, parts, 65535ll * parts, 65536ll * parts, 1ll * row_blocks * parts - 1, 1ll * row_blocks * parts, blocks - 1};
        for (long long b : probes) {
          if (b >= blocks) continue;
          const F32Block p = f32_block(static_cast<unsigned>(b), parts, row_blocks);
          NEED(p.part >= 0 && p.part < parts && p.row_block >= 0 && p.row_block < row_blocks && p.slice >= 0 && p.slice < slices);
          NEED((static_cast<long long>(p.slice) * row_blocks + p.row_block) * parts + p.part == b);
          const int row0 = (row_blocks - 1 - p.row_block) * bm;
          NEED(row0 >= 0 && row0 < n && row0 + (bm - 1) >= 0);
        }
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
