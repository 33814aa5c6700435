"""GPU parity for the Q4_K and Q5_K decode products, through the C-ABI (zen_cuda_gemm_kquant, the device-pointer calls).

The reference computes both with fp32 activations (gemv_q4k_q5k_avx2, kernels/avx2.cpp:329-378); the checker is its C
restatement, pinned bit for bit to the compiled reference (tests/test_kquant_q4k_q5k_cpu.py), and the vectors the
unmodified reference produced.  Bar: 1e-3 under both gates of helpers.assert_parity.  The kernels keep the dot products in
integers with two int8 digits per activation (as for Q4_0 and Q6_K), so results land near 1e-5."""
import os

import numpy as np
import pytest

from helpers import assert_parity, seeded_acts, seeded_weights
from zeninfer_b200 import blocks

pytestmark = pytest.mark.gpu
FORMATS = [(blocks.Q4_K, "Q4_K", "q4_k"), (blocks.Q5_K, "Q5_K", "q5_k")]
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "kquant_vectors.npz")


@pytest.fixture(scope="module")
def be():
    from zeninfer_b200 import Backend
    return Backend()


@pytest.mark.parametrize("fmt,name,tag", FORMATS)
def test_against_the_reference_vectors(be, fmt, name, tag):
    with np.load(GOLDEN) as g:
        w, x, y = np.ascontiguousarray(g[tag + "_w"]), g[tag + "_x"], g[tag + "_y"]
    rel = assert_parity(be.gemv(name, w, x, w.shape[0], x.size), y, what=f"{name} gemv vs the reference's vector")
    assert rel < 1e-4
    be.release_weights(w)


@pytest.mark.parametrize("fmt,name,tag", FORMATS)
@pytest.mark.parametrize("rows,cols,tokens", [(1, 256, 1), (5, 512, 1), (67, 1280, 3), (130, 2048, 8), (1024, 4096, 1), (64, 14336, 2), (300, 768, 11),
                                              (2050, 4096, 8), (33, 4096, 40), (9, 4352, 5), (8, 8192, 7), (1027, 8192, 1), (4096, 14336, 1), (77, 12288, 2)])
def test_host_pointer_product_vs_oracle(be, zo, fmt, name, tag, rows, cols, tokens):
    w = blocks.random_k_blocks(fmt, rows, cols, 500 + rows)
    x = seeded_acts(tokens, cols, 510 + cols)
    got = be.gemm(name, w, x, tokens, rows, cols)       # more than 8 tokens: several launches
    ref = np.stack([zo.gemv(fmt, w, x[t], rows, cols) for t in range(tokens)])
    rel = assert_parity(got, ref, what=f"{name} {tokens}x{rows}x{cols}")
    assert rel < (3e-4 if tokens >= 9 else 1e-4)        # nine rows and more: the group-scale tensor-core kernel (~5e-5)
    be.release_weights(w)


@pytest.mark.parametrize("fmt,name,tag", FORMATS)
def test_device_pointer_calls(be, zo, fmt, name, tag):
    import torch
    from zeninfer_b200 import BackendError
    from zeninfer_b200.backend import ACT_FP32, ACT_INT8
    rows, cols, tokens = [96, 40], 1024, 3
    ws = [blocks.random_k_blocks(fmt, r, cols, 520 + r) for r in rows]
    hs = [be.dev_upload(name, w, r, cols) for w, r in zip(ws, rows)]
    part = be.dev_upload(name, ws[0], rows[0], cols, 32, 48)            # rows 32..79 of the first tensor
    x = seeded_acts(tokens, cols, 530)
    d_x = torch.from_numpy(x).cuda()
    outs = [torch.zeros((tokens, r), dtype=torch.float32, device="cuda") for r in rows + [48]]
    stream = torch.cuda.Stream()
    be.dev_gemv(hs, [o.data_ptr() for o in outs[:2]], d_x.data_ptr(), tokens, ACT_FP32, stream.cuda_stream)
    be.dev_gemv([part], [outs[2].data_ptr()], d_x.data_ptr(), tokens, ACT_FP32, stream.cuda_stream)
    stream.synchronize()
    be.dev_check(stream.cuda_stream)
    for w, r, o in zip(ws, rows, outs):
        ref = np.stack([zo.gemv(fmt, w, x[t], r, cols) for t in range(tokens)])
        assert_parity(o.cpu().numpy(), ref, what=f"{name} device-pointer product rows={r}")
    assert torch.equal(outs[2], outs[0][:, 32:80])
    with pytest.raises(BackendError):
        be.dev_gemv(hs[:1], [outs[0].data_ptr()], d_x.data_ptr(), tokens, ACT_INT8, stream.cuda_stream)   # fp32-equivalent activations only
    for h in hs + [part]:
        be.dev_free(h)


@pytest.mark.parametrize("fmt,name,tag", FORMATS)
@pytest.mark.parametrize("rows,cols,tokens", [(300, 4096, 40), (1027, 1280, 12), (64, 14336, 64), (130, 2048, 129), (19000, 256, 16)])
def test_tensor_core_product_vs_oracle(be, zo, fmt, name, tag, rows, cols, tokens):
    # many activation rows: codes widened to int8 in the workspace with the fp32 factors d * sc and dmin * m of every
    # sub-block, then the tcgen05 GEMM with two activation digits whose epilogue subtracts the minimum term.  Device entry
    # point with a caller workspace, then the host-pointer call (the same path from nine rows on).  19000 rows are 149
    # row tiles: the K range of one tile is shared between two CTAs.
    import torch
    w = blocks.random_k_blocks(fmt, rows, cols, 600 + rows)
    x = seeded_acts(tokens, cols, 610 + cols)
    ref = np.stack([zo.gemv(fmt, w, x[t], rows, cols) for t in range(tokens)])
    h = be.dev_upload(name, w, rows, cols)
    d_x = torch.from_numpy(x).cuda()
    y = torch.full((tokens, rows), float("nan"), device="cuda")
    ws_bytes = be.gemm_kquant_workspace_bytes(tokens, rows, cols)
    ws = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda")
    # the group-scale kernel over the tensor's cached two-digit planes (~5e-5); with it switched off, codes widened per call
    # and the per-block kernel with fp32 sub-block scales and the minimum term in its epilogue (~1e-5)
    outs = {}
    for groups in (False, True):
        before = be.set_gemm_groups(groups)
        try:
            y.fill_(float("nan"))
            be.dev_gemm_kquant(h, y.data_ptr(), d_x.data_ptr(), tokens, ws.data_ptr(), ws_bytes)
            be.dev_check()
        finally:
            be.set_gemm_groups(before)
        outs[groups] = y.cpu().numpy()
        if groups:
            # 16-bit fixed point per 256-weight group: the error scales with the LARGEST result (these random blocks give results
            # in the hundreds), so only the gate on max_abs / max_ref applies; the per-element gate is the other kernel's
            rel = float(np.abs(outs[groups].astype(np.float64) - ref).max() / np.abs(ref).max())
            assert np.all(np.isfinite(outs[groups])) and rel < 3e-4, rel
        else:
            rel = assert_parity(outs[groups], ref, what=f"{name} tensor product {tokens}x{rows}x{cols} groups={groups}")
            assert rel < 1e-4
    be.dev_free(h)
    host = be.gemm(name, w, x, tokens, rows, cols)
    assert np.array_equal(host, outs[True])       # the same kernels on the same bytes
    be.release_weights(w)


# ---- the matrix instructions' kernel (gemv_kq_mma.cuh), all formats ----
ALL = {"Q4_0": blocks.Q4_0, "Q6_K": blocks.Q6_K, "Q4_K": blocks.Q4_K, "Q5_K": blocks.Q5_K}


def _weights(fmt, rows, cols, seed):
    return blocks.random_k_blocks(fmt, rows, cols, seed) if fmt in (blocks.Q4_K, blocks.Q5_K) else seeded_weights(fmt, rows, cols, seed)


def _products(be, name, w, x, rows, cols):
    """dev_gemv of all rows of x in one launch."""
    import torch
    tokens = x.shape[0]
    h = be.dev_upload(name, w, rows, cols)
    d_x, y = torch.from_numpy(x).cuda(), torch.full((tokens, rows), float("nan"), device="cuda")
    be.dev_gemv([h], [y.data_ptr()], d_x.data_ptr(), tokens, 2)
    be.dev_check()
    be.dev_free(h)
    return y.cpu().numpy()


def _close_to_f64(got, fmt, w, x, some_rows, cols, repeat):
    """Within 2^-22 of an activation per product (two f16 digits) and the rounding of fp32 sums over a row, of the terms' magnitudes (a
    Q4_K / Q5_K weight is the difference of two terms, the smaller of at most 63 * 1.5e-4, random_k_blocks); and per product
    2^-14 of a block's step times its largest activation: what the matrix instruction keeps of a product beside the largest of its
    sixteen, 24 bits below the exponent of an f16 number of ten mantissa bits.  Q6_K from 4096 columns on (gemv_kq.cuh): an
    activation is off by half a step of its second digit at most, 1 / (127 * 512) of the largest of its 32."""
    decoded = blocks.dequantize(fmt, w[:some_rows], some_rows, cols).astype(np.float64)
    want, terms = x.astype(np.float64) @ decoded.T, np.abs(x).astype(np.float64) @ (np.abs(decoded) + (0.019 if fmt in (blocks.Q4_K, blocks.Q5_K) else 0.0)).T
    n = 16 if fmt == blocks.Q6_K else 32
    values = np.sort(decoded.reshape(some_rows, -1, n), axis=2)
    gaps = np.diff(values, axis=2)
    step = np.where(gaps > 1e-9 * np.abs(values).max(), gaps, np.inf).min(axis=2)          # [rows][blocks]
    largest = np.abs(x).astype(np.float64).reshape(x.shape[0], -1, n).max(axis=2)
    bound = terms * (2.0 ** -22 + 64 * 2.0 ** -24) + n * 2.0 ** -14 * largest @ np.where(np.isfinite(step), step, 0.0).T + 1e-30
    if fmt == blocks.Q6_K and cols >= 4096:
        largest, weight = np.abs(x).reshape(x.shape[0], -1, 32).max(axis=2).astype(np.float64), np.abs(decoded).reshape(some_rows, -1, 32).sum(axis=2)
        bound = terms * 64 * 2.0 ** -24 + largest @ weight.T / (127 * 512)
    for first in range(0, got.shape[1], some_rows):
        part = got[:, first:first + some_rows]
        assert np.all(np.abs(part - want[:, :part.shape[1]]) <= bound[:, :part.shape[1]])
        if not repeat:
            break


def _rows_of(be, name, parts, x, cols):
    """One launch of several tensors; their outputs."""
    import torch
    tokens = x.shape[0]
    hs = [be.dev_upload(name, w, w.shape[0], cols) for w in parts]
    d_x, ys = torch.from_numpy(x).cuda(), [torch.full((tokens, w.shape[0]), float("nan"), device="cuda") for w in parts]
    be.dev_gemv(hs, [y.data_ptr() for y in ys], d_x.data_ptr(), tokens, 2)
    be.dev_check()
    for h in hs:
        be.dev_free(h)
    return [y.cpu().numpy() for y in ys]


# A row's arithmetic is chosen by format and columns: neither a companion of 70 million weights nor other tokens of the launch may move it by
# more than the rounding of its sums, some 1e-6 (the two kernels of these formats are 2e-5 apart).
@pytest.mark.parametrize("name", list(ALL))
@pytest.mark.parametrize("cols", [1024, 3840, 4096, 4352])
def test_what_shares_a_launch_does_not_choose_a_rows_arithmetic(be, name, cols):
    fmt = ALL[name]
    w, x = _weights(fmt, 40, cols, cols), seeded_acts(8, cols, cols + 1)
    some = _weights(fmt, 64, cols, 5)
    large = np.ascontiguousarray(np.tile(some, ((70 << 20) // cols // 64 + 1, 1)))
    most = 8 if cols <= 4096 else 4                  # the limit of columns x tokens
    alone = np.concatenate([_rows_of(be, name, [w], x[t:t + 1], cols)[0] for t in range(most)])
    apart = lambda got: np.linalg.norm(got - alone[:got.shape[0]]) / np.linalg.norm(alone[:got.shape[0]])
    for tokens in (2, 3, most):
        assert apart(_rows_of(be, name, [w], x[:tokens], cols)[0]) < 5e-6
    for tokens in (1, 2, 3):
        assert apart(_rows_of(be, name, [large, w], x[:tokens], cols)[1]) < 5e-6


# A row's bits depend on its columns and tokens only: alone, in shards, beside other tensors, in slices that are taken in blocks and passes.
@pytest.mark.parametrize("name", list(ALL))
@pytest.mark.parametrize("cols,tokens", [(256, 1), (1024, 2), (2048, 5), (3840, 1), (3840, 4), (4096, 1), (4096, 4), (4096, 8), (11008, 2), (14336, 1)])
def test_a_rows_bits_are_the_same_in_any_launch(be, name, cols, tokens):
    fmt, rows = ALL[name], 300
    w, x = _weights(fmt, rows, cols, cols), seeded_acts(tokens, cols, cols + 1)
    whole, = _rows_of(be, name, [w], x, cols)
    for cut in (1, 100, 284):
        assert np.array_equal(np.concatenate([_rows_of(be, name, [part], x, cols)[0] for part in (w[:cut], w[cut:])], axis=1), whole)
    for more in (2_000, 24_000, 130_000):
        if more * cols > 140 << 20:
            break
        other = np.ascontiguousarray(np.tile(w[:100], (more // 100, 1)))
        first, got, last = _rows_of(be, name, [other, w, w[:77]], x, cols)
        assert np.array_equal(got, whole) and np.array_equal(last, whole[:, :77])
        assert np.array_equal(first, np.tile(whole[:, :100], (1, more // 100)))


@pytest.mark.parametrize("rows,cols,tokens", [(14336, 4096, 4), (28672, 2048, 4), (70000, 2048, 4), (70000, 1024, 8), (9000, 3840, 1)])
def test_q6_k_layouts_give_the_same_bits_for_many_rows(be, rows, cols, tokens):
    w, x = np.ascontiguousarray(np.tile(_weights(blocks.Q6_K, 40, cols, 1), (rows // 40 + 1, 1))[:rows]), seeded_acts(tokens, cols, 2)
    before, got = be.set_q6k_codes(True), []
    try:
        for codes in (True, False):
            be.set_q6k_codes(codes)
            got.append(_products(be, "Q6_K", w, x, rows, cols))
    finally:
        be.set_q6k_codes(before)
    assert np.array_equal(got[0], got[1])


# edges of tiles (16 rows), of units (256 columns; Q4_0 ends inside one), of warps' shares; one or more groups of four tokens;
# 16384 columns by three tokens and 14336 by two or three go over the row in several passes
@pytest.mark.parametrize("name", list(ALL))
@pytest.mark.parametrize("rows,cols,tokens", [(1, 256, 3), (15, 256, 4), (17, 512, 5), (33, 768, 8), (1200, 4096, 3), (2405, 1280, 4), (2405, 1280, 7), (300, 14336, 2), (300, 14336, 3),
                                              (140, 11008, 3), (5000, 256, 6), (1200, 3840, 3), (300, 3840, 8), (9000, 2048, 4)])
def test_several_rows_at_once(be, name, rows, cols, tokens):
    fmt = ALL[name]
    if name == "Q6_K" and cols * tokens > 32768:
        tokens = 2
    w, x = _weights(fmt, rows, cols, rows + tokens), seeded_acts(tokens, cols, cols)
    _close_to_f64(_products(be, name, w, x, rows, cols), fmt, w, x, rows, cols, False)


@pytest.mark.parametrize("rows,cols,tokens", [(37, 32, 3), (70, 96, 4), (129, 544, 8), (64, 4128, 2), (18, 16384, 3)])
def test_q4_0_rows_that_end_inside_a_unit(be, rows, cols, tokens):
    w, x = _weights(blocks.Q4_0, rows, cols, rows), seeded_acts(tokens, cols, cols)
    _close_to_f64(_products(be, "Q4_0", w, x, rows, cols), blocks.Q4_0, w, x, rows, cols, False)


# one activation row; the rows of a small matrix over and over
@pytest.mark.parametrize("name,rows,cols", [("Q4_0", 16500, 4096), ("Q4_0", 16400, 4128), ("Q4_0", 4700, 14336), ("Q4_0", 262200, 256), ("Q4_K", 8200, 4096), ("Q4_K", 3077, 11008),
                                            ("Q5_K", 8200, 4096), ("Q5_K", 32800, 1024)])
def test_one_row_of_a_large_matrix(be, name, rows, cols):
    fmt, some = ALL[name], min(rows, 50)
    part = _weights(fmt, some, cols, rows)
    w, x = np.ascontiguousarray(np.tile(part, (rows // some + 1, 1))[:rows]), seeded_acts(1, cols, cols)
    _close_to_f64(_products(be, name, w, x, rows, cols), fmt, w, x, some, cols, True)


@pytest.mark.parametrize("name,rows,cols", [(n, r, c) for n in ALL for r, c in ((1, 256), (17, 1024), (150, 3840), (9000, 2048), (2400, 512), (130, 14336))] + [("Q4_0", 37, 32), ("Q4_0", 70, 96)])
def test_one_row(be, name, rows, cols):
    test_one_row_of_a_large_matrix(be, name, rows, cols)


def test_more_rows_than_their_sums_fit(be):
    rows, some, tokens = 700_000, 64, 8
    part = _weights(blocks.Q4_0, some, 32, 3)
    w, x = np.ascontiguousarray(np.tile(part, (rows // some + 1, 1))[:rows]), seeded_acts(tokens, 32, 4)
    _close_to_f64(_products(be, "Q4_0", w, x, rows, 32), blocks.Q4_0, w, x, some, 32, True)


# Two blocks of one unit far apart: an activation is held to 2^-35 of the largest of its 256 columns (2^-39 in low nibbles), seen where
# the large ones meet weights that are zero.
@pytest.mark.parametrize("tokens", [1, 3, 8])
@pytest.mark.parametrize("log2", [8, 16, 30])
def test_small_activations_beside_large_ones(be, tokens, log2):
    rows, cols = 100, 1024
    w, x = _weights(blocks.Q4_0, rows, cols, 11), seeded_acts(tokens, cols, 12)
    w.reshape(rows, cols // 32, 18)[:, ::8, :2] = 0           # the scale of every unit's first block
    x.reshape(tokens, cols // 32, 32)[:, ::8] *= np.float32(2.0 ** log2)
    got = _products(be, "Q4_0", w, x, rows, cols)
    decoded = blocks.dequantize(blocks.Q4_0, w, rows, cols).astype(np.float64)
    small = np.abs(x).astype(np.float64) * (np.arange(cols) % 256 >= 32)
    largest = np.abs(x).reshape(tokens, -1, 256).max(axis=2).astype(np.float64)
    step = w.reshape(rows, cols // 32, 18)[:, :, :2].copy().view(np.float16).astype(np.float64)[..., 0]
    in_block = small.reshape(tokens, -1, 32).max(axis=2)
    bound = small @ np.abs(decoded).T * (2.0 ** -22 + 64 * 2.0 ** -24) + largest @ np.abs(decoded).reshape(rows, -1, 256).sum(axis=2).T * 2.0 ** -35 + 32 * 2.0 ** -14 * in_block @ np.abs(step).T
    bound += largest @ np.abs(step).reshape(rows, -1, 8).sum(axis=2).T * 256 * 2.0 ** -35      # nibbles are up to 8 steps from the weight they stand for
    assert np.all(np.abs(got - x.astype(np.float64) @ decoded.T) <= bound)


@pytest.mark.parametrize("name", list(ALL))
def test_activations_of_any_size(be, name):
    """The operands are scaled by a power of two per 256 columns: vectors of very large, very small and no values, and both in one."""
    fmt, rows, cols = ALL[name], 1100, 1024
    w, x = _weights(fmt, rows, cols, 9), seeded_acts(5, cols, 10)
    x[0] *= np.float32(2.0 ** 100)
    x[1] *= np.float32(2.0 ** -80)
    x[2] = 0
    x[3, :256] *= np.float32(2.0 ** 40)
    x[3, 256:512] *= np.float32(2.0 ** -40)
    x[4, 300] = np.float32(3e5)
    got = _products(be, name, w, x, rows, cols)
    assert not got[2].any()
    _close_to_f64(got, fmt, w, x, rows, cols, False)
    x[1, 17], x[4, 5] = np.nan, np.inf              # a row's own business
    bad = _products(be, name, w, x, rows, cols)
    assert np.array_equal(bad[[0, 2, 3]], got[[0, 2, 3]]) and not np.isfinite(bad[[1, 4]]).any()
