"""GPU parity of the kernels that run in thread-block clusters, at the sizes where they can go wrong: the matmul by CTA
pairs (row tiles, token tiles, K shares), the eight-row Q4_0 / Q8_0 matvecs and the decode step whose CTAs share the
staging of x; and of the one-row Q8_1 matvecs with the activations in registers."""
import numpy as np
import pytest

import lib_b200
from lib_b200 import _capi, synth
from oracle import oracle
from tests import q8_1_cases as cases
from tests.capture import launches
from tests.test_pair_plan import FORMS
from tests.test_gpu_matmul import TOL as MATMUL_TOL, run as run_matmul
from tests.test_gpu_stack import build_stack, nre, oracle_chain

pytestmark = pytest.mark.gpu


# Few rows or tokens, which run as single CTAs with tiles of 32 and 64 tokens: rows around a CTA's 128, tokens around the
# rounding to 16 and a tile of 32; one K unit, fewer units than K shares, more units than the ring of weight items.
@pytest.mark.parametrize("n,k,m", [(1, 256, 1), (127, 256, 15), (129, 512, 17), (255, 768, 32), (257, 1024, 33), (256, 2560, 127),
                                   (640, 5120, 129), (272, 256, 255), (520, 512, 257), (144, 2304, 481), (20000, 256, 31),
                                   (9500, 512, 161)])
def test_matmul_edges(ctx, devbuf, n, k, m):
    assert run_matmul(ctx, devbuf, n, k, m, seed=3 * n + m) <= MATMUL_TOL


# Every form of the matmul — pairs and single CTAs, tiles of up to 224 tokens, one to four K shares, several tiles per
# CTA — with the launch that the plan says. The last 100 rows against the oracle, where the rows are ragged.
@pytest.mark.parametrize("shape,plan", FORMS)
def test_matmul_forms(ctx, devbuf, shape, plan):
    (n, k, m), (cg, bn, splitk, tiles) = shape, plan
    assert run_matmul(ctx, devbuf, n, k, m, seed=n + m, check_rows=(max(0, n - 100), n)) <= MATMUL_TOL
    w = ctx.store_create(12, n, k)
    a, c = devbuf(nbytes=2 * m * k), devbuf(nbytes=4 * m * n)
    made, = launches(ctx, lambda: ctx.matmul_bf16(w, a.ptr, m, k, c.ptr, n))
    assert made.name == ("qm_gemm_q4k_pair" if cg == 2 else "qm_gemm_q4k_solo")
    assert made.grid == cg * (tiles * splitk if splitk > 1 else min(tiles, 148 // cg))
    w.free()


# Two limbs per activation row from three rows on: 14 bits of the unit's maximum, 3e-4 normwise (as in the matvec
# tests). K of one unit, a partial unit, an odd number of units, and a long K that runs in parts: below the sizes that
# share a staging.
@pytest.mark.parametrize("fmt", [2, 8])
@pytest.mark.parametrize("m", [6, 7, 8])
@pytest.mark.parametrize("rows,cols,xop", [(16, 256, 0), (33, 288, 1), (2400, 2336, 1), (4736, 1280, 0), (96, 8192, 1)])
def test_matvec_without_sharing(ctx, devbuf, fmt, m, rows, cols, xop):
    raw = synth.weights(fmt, rows, cols, seed=rows + m)
    w = ctx.store_upload(fmt, rows, cols, raw)
    x = synth.activations(m, cols, 9)
    xd, yd = devbuf(x), devbuf(np.full((m, rows), np.nan, np.float32))
    assert not any(k.name.endswith("_x2") for k in launches(ctx, lambda: ctx.matvec(w, xd.ptr, m, cols, yd.ptr, rows, xop)))
    ctx.matvec(w, xd.ptr, m, cols, yd.ptr, rows, xop)
    got = yd.get((m, rows))
    assert ctx.last_status() == (0, 0)
    want = oracle.MatVec(fmt, raw, rows, cols, oracle.RMSNorm(x) if xop else x)
    assert nre(got, want) <= 3e-4
    w.free()


# Two CTAs share the staging from seven rows and 96 (row, unit) pairs on: the fewest units, a last unit with one block, an
# odd number of units and the most (one unit less than runs in parts; Q8_0: the most that fit), rows that are no whole
# tiles and fewer tiles than CTAs, and every input transform (the sums of squares cross the CTAs).
@pytest.mark.parametrize("fmt,m,rows,cols,xop", [
    (fmt, m, rows, cols, xop) for fmt in (2, 8) for m in (7, 8) for xop in range(4)
    for rows, cols in [(33, 3584 if m == 7 else 3072), (2387, 3360), (4737, 4096), (17, 7936 if fmt == 2 else 4096)]])
def test_matvec_shared_staging(ctx, devbuf, fmt, m, rows, cols, xop):
    raw = synth.weights(fmt, rows, cols, seed=rows + m)
    w = ctx.store_upload(fmt, rows, cols, raw)
    x, x2 = synth.activations(m, cols, 9), synth.activations(m, cols, 10)
    xd, x2d, yd = devbuf(x), devbuf(x2), devbuf(np.full((m, rows), np.nan, np.float32))
    call = lambda: ctx.matvec(w, xd.ptr, m, cols, yd.ptr, rows, xop, x2d.ptr if xop >= 2 else 0)
    assert [k.name[:17] + k.name[-3:] for k in launches(ctx, call)] == ["qm_gemv_q%d0_lean__x2" % (4 if fmt == 2 else 8)]
    call()
    got = yd.get((m, rows))
    assert ctx.last_status() == (0, 0)
    x64 = x.astype(np.float64)
    inputs = [x, oracle.RMSNorm(x), oracle.RMSNorm(x + x2), (x64 / (1 + np.exp(-x64)) * x2).astype(np.float32)]
    assert nre(got, oracle.MatVec(fmt, raw, rows, cols, inputs[xop])) <= 3e-4
    w.free()


# Eight Q8_0 rows of 17 units: the shared memory of a CTA holds them only without the second CTA's sums of squares. Sixteen
# units, and Q4_0, share.
@pytest.mark.parametrize("fmt,cols,kernel", [(8, 4352, "qm_gemv_q80_lean_c2n2d2"), (8, 4128, "qm_gemv_q80_lean_c2n2d2"),
                                             (8, 4096, "qm_gemv_q80_lean_c2n2d2_x2"), (2, 4352, "qm_gemv_q40_lean_c2n2d2_x2")])
def test_matvec_that_fits_only_without_sharing(ctx, devbuf, fmt, cols, kernel):
    rows, m = 80, 8
    raw = synth.weights(fmt, rows, cols, seed=cols)
    w = ctx.store_upload(fmt, rows, cols, raw)
    x = synth.activations(m, cols, 9)
    xd, yd = devbuf(x), devbuf(np.full((m, rows), np.nan, np.float32))
    call = lambda: ctx.matvec(w, xd.ptr, m, cols, yd.ptr, rows, 1)
    assert [k.name for k in launches(ctx, call)] == [kernel]
    call()
    assert nre(yd.get((m, rows)), oracle.MatVec(fmt, raw, rows, cols, oracle.RMSNorm(x))) <= 3e-4
    assert ctx.last_status() == (0, 0)
    w.free()


# Hidden sizes of fewer units than the cluster has warps, an odd number of units, and a down projection that cannot be
# cut into four parts (5 and 7 units) or can (8).
@pytest.mark.parametrize("m", [3, 4, 6, 7, 8])
@pytest.mark.parametrize("hidden,kv,ffn", [(256, 32, 1280), (768, 96, 1792), (1280, 160, 2048)])
def test_step_shared_staging(ctx, m, hidden, kv, ffn):
    st, raws = build_stack(ctx, 2, hidden, kv, ffn, 12, seed=41)
    check_step(ctx, st, raws, m, hidden, kv, ffn)
    st.close()


# The kernels whose CTAs share the staging, by their rules on rows and hidden units: one and two column tiles, each number
# of ring stages, an odd number of units, the down projection whole and in parts; and just below the rules.
@pytest.mark.parametrize("m,hidden,ffn,kernel", [
    (4, 3072, 512, "c2d4_x4"), (4, 3328, 1024, "c2d4_x4"), (4, 8192, 512, "c2d3_x4"), (4, 2816, 512, "c2d4"),
    (5, 2560, 512, "n2d3_x4"), (5, 2304, 512, "n2d3"), (6, 2048, 1024, "n2d3_x4"), (7, 1280, 1280, "n2d3_x4"),
    (8, 1280, 512, "n2d3_x4"), (8, 1024, 512, "n2d3"), (8, 5120, 512, "n2d2_x4")])
def test_step_forms(ctx, devbuf, m, hidden, ffn, kernel):
    kv = 32
    st, raws = build_stack(ctx, 2 if hidden <= 4096 else 1, hidden, kv, ffn, 12, seed=43)
    check_step(ctx, st, raws, m, hidden, kv, ffn)
    xd = devbuf(synth.activations(m, hidden, 8))
    assert "qm_fused_q4k_dd_" + kernel in [k.name for k in launches(ctx, lambda: st.step(xd.ptr, m, hidden))]
    st.close()


def check_step(ctx, st, raws, m, hidden, kv, ffn):
    x = synth.activations(m, hidden, 8)
    h, kvs = st.step_host(x, want_kv=True)
    want_h, want_kv, _ = oracle_chain(12, raws, x, hidden, kv, ffn)
    assert nre(h, want_h) <= 1e-3 and nre(kvs, want_kv) <= 1e-3
    assert np.array_equal(h, st.step_host(x))
    assert ctx.last_status() == (0, 0)


# Steps of four super-blocks: a single one, whole steps, a remainder, the largest K in registers and the first beyond.
# (Rows of Q2_K / IQ2_XXS are whole 16-byte pieces, which the staged form needs, at multiples of four / eight units.)
@pytest.mark.parametrize("fmt", [10, 16])
@pytest.mark.parametrize("cols", [256, 1024, 2048, 3072, 4096, 6144])
def test_q8_1_row(ctx, devbuf, fmt, cols):
    experts, rows = 3, 41
    raw = synth.weights(fmt, experts * rows, cols, seed=fmt + cols)
    w = ctx.store_upload(fmt, experts * rows, cols, raw)
    ids = np.array([2, 7, 0], dtype=np.int32)
    x, _ = cases.random_rows(1, cols, seed=cols)
    xq = oracle.RMSNormQ8_1(x, None, 1, cols, 1e-6, False)
    xd, yd = devbuf(np.frombuffer(xq, dtype=np.uint8)), devbuf(nbytes=len(ids) * rows * 4)
    ctx.matvec_selected(w, experts, devbuf(ids).ptr, len(ids), xd.ptr, 0, yd.ptr, _capi.FLAG_X_Q8_1)
    got = yd.get((len(ids), rows))
    want = oracle.SelectedMatVecQ8_1(fmt, raw, experts, rows, cols, [2, -1, 0], xq)
    # exact integer sums per group, float32 across groups: 2e-5 of the largest output, as for the other Q8_1 matvecs
    assert np.abs(got[[0, 2]] - want[[0, 2]]).max() <= 2e-5 * np.abs(want[[0, 2]]).max()
    assert np.all(got[1].view(np.uint32) == 0x7fffffff)
    w.free()


# Those kernels hold more registers than the others: a launch starts no more CTAs than run at once.
@pytest.mark.parametrize("fmt,name,ctas", [(10, "qm_gemv_q2k_q81_row", 3), (16, "qm_gemv_iq2xxs_q81_row", 4)])
@pytest.mark.parametrize("cols", [1024, 2048, 4096])
@pytest.mark.parametrize("slots", [1, 8])
def test_q8_1_row_launch_fits_at_once(ctx, devbuf, fmt, name, ctas, cols, slots):
    if fmt == 16 and cols == 1024:
        name, ctas = "qm_gemv_iq2xxs_q81_m1", 8     # rows of 264 bytes: the direct form
    w = ctx.store_create(fmt, 8 * 14336, cols)
    b = devbuf(nbytes=4 * 8 * 14336)
    made, = launches(ctx, lambda: ctx.matvec_selected(w, 8, b.ptr, slots, b.ptr, 0, b.ptr, _capi.FLAG_X_Q8_1))
    assert made.name == name and 148 * ctas // 2 <= made.grid <= 148 * ctas
    w.free()


# Launches overlap the end of the kernel before them: weights written in stream order right before a product, and a
# product whose input the launch before it writes, have to be as good as with a wait in between (equal bits).
@pytest.mark.parametrize("fmt", [2, 8, 10, 12, 16])
@pytest.mark.parametrize("m", [1, 8])
def test_overlapping_launches_keep_stream_order(ctx, devbuf, fmt, m):
    n = 1024
    raws = [devbuf(np.frombuffer(bytes(synth.weights(fmt, n, n, seed=60 + i)), dtype=np.uint8)) for i in range(2)]
    size = len(bytes(synth.weights(fmt, n, n, seed=60)))
    x = devbuf(synth.activations(m, n, 5))

    def chain(wait):
        w = ctx.store_create(fmt, n, n)
        ys = [devbuf(np.zeros((m, n), np.float32)) for _ in range(8)]
        for i, y in enumerate(ys):
            if i % 3 != 2:   # written before two of three products
                w.write_rows_device(0, n, raws[i % 2].ptr, size)
                if wait:
                    ctx.sync()
            ctx.matvec(w, (ys[i - 1] if i else x).ptr, m, n, y.ptr, n)
            if wait:
                ctx.sync()
        ctx.sync()
        got = [y.get((m, n)) for y in ys]
        w.free()
        return got

    for a, b in zip(chain(True), chain(False)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert ctx.last_status() == (0, 0)


# A product reads its weights before it waits for the kernel before it, so that kernel must not be the one that writes
# them: whatever another context, on another stream, has multiplied with them in the meantime.
@pytest.mark.parametrize("fmt", [2, 8, 12])
@pytest.mark.parametrize("flags", [0, _capi.FLAG_PDL])
def test_no_product_overlaps_the_kernel_that_writes_its_weights(ctx, devbuf, fmt, flags):
    n = 1024
    raw = devbuf(np.frombuffer(bytes(synth.weights(fmt, n, n, seed=70)), dtype=np.uint8))
    x, y, z = devbuf(synth.activations(1, n, 5)), devbuf(nbytes=4 * n), devbuf(nbytes=4 * n)
    w = ctx.store_create(fmt, n, n)
    w.write_rows_device(0, n, raw.ptr, raw.nbytes)
    ctx.sync()
    other = lib_b200.Context(0)

    def chain():
        w.write_rows_device(0, n, raw.ptr, raw.nbytes)
        other.matvec(w, x.ptr, 1, n, z.ptr, n)      # at once, on a stream of its own
        ctx.matvec(w, x.ptr, 1, n, y.ptr, n, flags)
        ctx.matvec(w, y.ptr, 1, n, z.ptr, n, flags)

    made = launches(ctx, chain)
    other.sync()
    assert made[0].name.startswith("qm_repack")
    products = [k for k in made if "gemv" in k.name or "fused" in k.name]
    assert len(products) == 2 and products[0].overlaps is None and products[1].overlaps is not None
    assert all("repack" not in (k.overlaps or "") for k in made)
    other.close()
    w.free()


# More experts than rows: most lists are empty, and the down launch keeps a pair per tile (its K is shared between
# pairs only where all tiles fit at once).
@pytest.mark.parametrize("experts,tokens,topk", [(64, 5, 1), (64, 43, 1), (16, 9, 2), (3, 1, 2)])
def test_moe_layer_with_few_rows(ctx, devbuf, experts, tokens, topk):
    from tests.test_gpu_moe import TOL, run_moe
    assert run_moe(ctx, devbuf, experts, 512, 768, tokens, topk, 23, list(range(tokens))) <= TOL


# Lists far longer than the mean, which the token tile is chosen for and which the host does not know: every token to one
# expert, K shared between pairs (four experts of hidden 512) and not (64 experts).
@pytest.mark.parametrize("experts,tokens", [(4, 40), (4, 333), (64, 200)])
def test_moe_layer_with_one_long_list(ctx, devbuf, experts, tokens):
    from tests.test_gpu_moe import TOL, moe_oracle, to_bf16_bits
    hidden, ffn, seed = 512, 768, 29
    gu_raw = [synth.weights(12, 2 * ffn, hidden, seed + e) for e in range(experts)]
    dn_raw = [synth.weights(12, hidden, ffn, seed + 100 + e) for e in range(experts)]
    gu = [ctx.store_upload(12, 2 * ffn, hidden, r) for r in gu_raw]
    dn = [ctx.store_upload(12, hidden, ffn, r) for r in dn_raw]
    x_bf = to_bf16_bits(synth.activations(tokens, hidden, seed + 200))
    ids, wts = np.full((tokens, 1), 2, np.int32), np.ones((tokens, 1), np.float32)
    out_d = devbuf(np.full((tokens, hidden), np.nan, np.float32))
    ctx.moe_grouped(gu, dn, devbuf(x_bf).ptr, tokens, hidden, devbuf(ids).ptr, devbuf(wts).ptr, 1, out_d.ptr, hidden)
    ctx.sync()
    assert ctx.last_status() == (0, 0)
    want = moe_oracle(gu_raw, dn_raw, hidden, ffn, x_bf, ids, wts, list(range(tokens)))
    got = out_d.get((tokens, hidden))
    assert np.isfinite(got).all() and float(np.linalg.norm(got - want)) <= TOL * float(np.linalg.norm(want))
    for w in gu + dn:
        w.free()
