"""Host-side rules of the matmul by CTA pairs (qm_kernel_args.h), compiled with the host compiler: no GPU needed."""
import os
import subprocess

import lib_b200

CSRC = os.path.join(os.path.dirname(lib_b200.__file__), "csrc")


def compiled(tmp_path, body):
    """What a program with this body of main() prints."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <cstdio>\n#include "qm_kernel_args.h"\nint main() {\n%s\nreturn 0;\n}\n' % body)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-I/usr/local/cuda/include", "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe)], check=True, stdout=subprocess.PIPE, text=True).stdout


def test_instruction_width_is_a_documented_one(tmp_path):
    out = compiled(tmp_path, """for (int ctas = 1; ctas <= 2; ctas++)
        for (int t = 1; t <= 256; t++) printf("%d %d %d\\n", ctas, t, qm_pair_mma_n(t, ctas));""")
    lines = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert len(lines) == 512
    for ctas, tokens, n in lines:
        step = 32 if ctas == 2 else 16      # a pair: multiples of 32; one CTA: multiples of 16
        assert n % step == 0 and step <= n <= 256
        assert tokens <= n <= (tokens + 31) // 32 * 32      # all tokens, and no more than a tile of 32s holds
