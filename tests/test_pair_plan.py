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
    """Grouped down launches over lists that stay on the device share K only where a cluster for every tile that the lists
    may hold fits on the device at once; where the host knows the lists of the same pairs, it decides alike."""
    cases = [(hidden, rows, experts) for hidden in (512, 1024, 2048, 4096) for experts in (1, 2, 4, 8, 16, 64)
             for rows in (3, 64, 300, 600, 1024, 8192)]
    body = CLUSTERS + "\nQmPairPlan p;\n"
    for hidden, rows, experts in cases:
        for longest, typical in ((rows, "qm_typical_list(%d, %d)" % (rows, experts)), ((rows + experts - 1) // experts,) * 2):
            body += ('p = qm_plan_grouped(at_once, %d, false, %d, %s, %d, %d, 16, true, %d, %d); '
                     'printf("%%d %%d %%d %%d\\n", p.cg, p.bn, p.splitk, (int)p.tiles);\n'
                     % (hidden, longest, typical, rows, experts, rows, rows))
    lines = [tuple(map(int, line.split())) for line in compiled(tmp_path, body, "qm_pair_plan.h").splitlines()]
    for case, unknown, known in zip(cases, lines[::2], lines[1::2]):
        for cg, bn, splitk, tiles in (unknown, known):
            assert cg == 2 and bn % 32 == 0 and 32 <= bn <= 160 and tiles >= 1
        assert unknown[2] == (2 if unknown[3] <= 33 else 1) == known[2], case
    assert {p[2] for p in lines} == {1, 2}


# One shape per form of the single-matrix matmul: rows, K, tokens -> CTAs per tile, tokens per tile, K shares, tiles.
# Ragged rows; token tiles that are full, that end one token past a multiple of 16 or 32, and short last ones.
FORMS = [
    ((10129, 256, 103), (2, 128, 1, 40)), ((4862, 1536, 103), (2, 128, 2, 19)), ((6144, 4096, 391), (2, 160, 1, 72)),
    ((10129, 256, 145), (2, 160, 1, 40)), ((4862, 2816, 139), (2, 160, 2, 19)), ((12934, 512, 169), (2, 192, 1, 51)),
    ((775, 3840, 1411), (2, 192, 2, 32)), ((12934, 768, 205), (2, 224, 1, 51)), ((4862, 9216, 205), (2, 224, 2, 19)),
    ((1739, 2304, 1908), (2, 192, 1, 70)), ((14336, 1024, 2048), (2, 128, 1, 896)),
    ((64, 1024, 2), (1, 32, 4, 1)), ((4302, 1536, 2), (1, 32, 2, 34)), ((536, 256, 962), (1, 64, 1, 80)),
    ((4862, 1536, 36), (1, 64, 2, 38)), ((64, 1024, 1059), (1, 64, 4, 17)), ((10129, 256, 69), (1, 96, 1, 80)),
    ((4862, 1536, 69), (1, 96, 2, 38)), ((137, 1024, 1059), (1, 96, 4, 24)), ((1616, 256, 1282), (1, 128, 1, 143)),
    ((536, 2048, 1411), (1, 128, 2, 60)), ((137, 1536, 1553), (1, 128, 4, 26)), ((2638, 256, 962), (1, 160, 1, 147)),
    ((775, 3840, 1553), (1, 160, 2, 70)), ((289, 2048, 1553), (1, 160, 4, 30)), ((6210, 2816, 490), (1, 192, 1, 147)),
    ((6210, 768, 655), (1, 224, 1, 147)),
]


def test_matmul_plans(tmp_path):
    body = CLUSTERS + "\nQmPairPlan p;\n" + "\n".join(
        'p = qm_plan_matmul(at_once, %d, %d, %d); printf("%%d %%d %%d %%d\\n", p.cg, p.bn, p.splitk, (int)p.tiles);'
        % (n, m, k // 256) for (n, k, m), _ in FORMS)
    out = compiled(tmp_path, body, "qm_pair_plan.h")
    assert [tuple(map(int, line.split())) for line in out.splitlines()] == [plan for _, plan in FORMS]
