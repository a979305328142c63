"""Host-side rules of the matmul by CTA pairs, compiled with the host compiler: no GPU needed."""
import os
import subprocess

import lib_b200

CSRC = os.path.join(os.path.dirname(lib_b200.__file__), "csrc")


def compiled(tmp_path, body, header="qm_kernel_args.h"):
    """What a program with this body of main() prints."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <cstdio>\n#include "%s"\nint main() {\n%s\nreturn 0;\n}\n' % (header, body))
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


# A B200 runs 148 single CTAs of this kernel at once, 74 pairs and 33 clusters of four.
CLUSTERS = "const QmPairClusters at_once = {{0, 148, 74, 0, 33}, {0, 74, 33, 0, 0}};"


def test_token_tiles_of_expert_lists_are_bounded_tightly(tmp_path):
    """The bound that sizes grouped launches against the lists that make the most tiles: no list beyond `longest`, `rows`
    tokens in all. (A K-shared launch computes only the tiles that it has a cluster for.)"""
    cases = [(longest, rows, experts, bn) for longest in (1, 31, 32, 33, 100) for rows in (1, 7, 64, 100, 333)
             for experts in (1, 2, 5, 16) for bn in (32, 96) if rows >= longest]
    out = compiled(tmp_path, "\n".join('printf("%%d\\n", (int)qm_grouped_token_tiles(%d, %d, %d, %d));' % c for c in cases),
                   "qm_pair_plan.h")
    for (longest, rows, experts, bn), bound in zip(cases, map(int, out.split())):
        # the most tiles: best[r] over lists so far with r tokens
        best = [0] + [-1] * rows
        for _ in range(experts):
            best = [max([best[r]] + [best[r - l] + (l + bn - 1) // bn for l in range(1, min(longest, r) + 1)
                                     if best[r - l] >= 0]) for r in range(rows + 1)]
        most = max(best)
        assert most <= bound <= most + 1, (longest, rows, experts, bn, most, bound)


def test_shared_k_launches_fit_at_once(tmp_path):
    """Grouped down launches share K only where a cluster per possible tile fits on the device at once."""
    cases = [(hidden, longest, typical, rows, experts) for hidden in (512, 1024, 2048, 4096) for experts in (1, 2, 4, 8, 16, 64)
             for rows in (3, 64, 300, 600, 1024, 8192) for longest in (rows, (rows + experts - 1) // experts)
             for typical in ((rows + experts - 1) // experts,)]
    body = CLUSTERS + "\nQmPairPlan p;\n" + "\n".join(
        'p = qm_plan_grouped(at_once, %d, false, %d, %d, %d, %d, 16, true); printf("%%d %%d %%d %%d\\n", p.cg, p.bn, p.splitk, '
        '(int)p.tiles);' % c for c in cases)
    shared = 0
    for c, line in zip(cases, compiled(tmp_path, body, "qm_pair_plan.h").splitlines()):
        cg, bn, splitk, tiles = map(int, line.split())
        assert cg == 2 and bn % 32 == 0 and 32 <= bn <= 160 and tiles >= 1
        assert splitk == (2 if tiles <= 33 else 1), c
        shared += splitk == 2
    assert 0 < shared < len(cases)
