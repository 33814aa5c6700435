"""GPU parity for the Q8_0 prefill GEMM (tcgen05 kind::i8), through the C-ABI host-pointer call.

Oracle: the int8-activation arithmetic (per token, kernels/avx2.cpp:562-585).  At sizes the C oracle finishes in
seconds it is used directly; at the full prefill size the check is a float64 restatement: with exact codes and
scales, sum_b d_x d_w sum_k q_x q_w equals (q_x * d_x) @ (q_w * d_w)^T evaluated in float64.
"""
import numpy as np
import pytest

from helpers import assert_parity, ref_fp32_f64, seeded_acts, seeded_weights
from zeninfer_b200 import blocks
from zeninfer_b200.backend import ACT_FP32, ACT_INT8, BackendError

pytestmark = pytest.mark.gpu
Q8_0 = blocks.Q8_0


@pytest.fixture(scope="module")
def be():
    from zeninfer_b200 import Backend
    b = Backend()
    b.set_q8_act_mode(ACT_INT8)
    return b


def dequant_f64(packed, rows, cols):
    b = packed.reshape(rows, cols // 32, 34)
    d = b[..., :2].copy().view(np.float16).astype(np.float64)
    return (b[..., 2:].view(np.int8).astype(np.float64) * d).reshape(rows, cols)


def ref_f64(zo, packed, x, rows, cols):
    xq, xsc = zo.quantise_acts(x)
    xd = (xq.astype(np.float64).reshape(x.shape[0], -1, 32) * xsc.astype(np.float64)[..., None]).reshape(x.shape)
    return xd @ dequant_f64(packed, rows, cols).T


@pytest.mark.parametrize("tokens,rows,cols", [
    (9, 128, 128), (16, 100, 544), (17, 300, 96), (33, 67, 32), (64, 256, 4096), (65, 130, 2048),
    (128, 512, 1024), (129, 129, 4096), (171, 2048, 2048), (256, 1000, 14336), (300, 4096, 4096)])
def test_gemm_vs_int8_oracle(be, zo, tokens, rows, cols):
    w = seeded_weights(Q8_0, rows, cols, 200 + rows)
    x = seeded_acts(tokens, cols, 300 + tokens)
    got = be.gemm("Q8_0", w, x, tokens, rows, cols)
    if tokens * rows * cols <= 64 * 256 * 4096:
        assert_parity(got, zo.gemm(Q8_0, w, x, tokens, rows, cols, int8_acts=True), what=f"gemm {tokens}x{rows}x{cols} vs oracle")
    # whole 256-weight groups: the group-scale kernel, 16-bit fixed point per group on both sides; else exact block sums
    rel = assert_parity(got, ref_f64(zo, w, x, rows, cols), tol=1e-3 if cols % 256 == 0 else 1e-5, what=f"gemm {tokens}x{rows}x{cols} vs float64")
    if cols % 256 == 0:
        assert rel < 2e-4
        before = be.set_gemm_groups(False)
        try:
            exact = be.gemm("Q8_0", w, x, tokens, rows, cols)
        finally:
            be.set_gemm_groups(before)
        assert_parity(exact, ref_f64(zo, w, x, rows, cols), tol=1e-5, what=f"per-block gemm {tokens}x{rows}x{cols} vs float64")
        assert assert_parity(got, exact, what="group-scale kernel vs per-block kernel") < 2e-4
    be.release_weights(w)


def test_token_ladder_from_reference(be, zo):
    # tests/core_tests.cpp:345-372: rows = 100, cols = 544 (17 blocks), closed-form bytes and activations
    rows, cols = 100, 544
    r = np.arange(rows)[:, None, None]
    blk = np.arange(17)[None, :, None]
    j = np.arange(2, 34)[None, None, :]
    packed = np.zeros((rows, 17, 34), np.uint8)
    packed[..., 1] = 0x3C
    packed[..., 2:] = (r * 5 + blk * 11 + j * 3) & 255
    packed = np.ascontiguousarray(packed.reshape(rows, -1))
    for T in (9, 16, 32, 171):
        t = np.arange(T)[:, None]
        c = np.arange(cols)[None, :]
        xin = (((t * 7 + c) % 15 - 7).astype(np.float32) * np.float32(0.017)).astype(np.float32)
        got = be.gemm("Q8_0", packed, xin, T, rows, cols)
        assert_parity(got, zo.gemm(Q8_0, packed, xin, T, rows, cols, int8_acts=True), what=f"ladder T={T}")
    be.release_weights(packed)


def test_gemm_batch_shares_input(be, zo):
    cols, rows, tokens = 1024, [512, 128, 128], 40
    ws = [seeded_weights(Q8_0, r, cols, 400 + i) for i, r in enumerate(rows)]
    x = seeded_acts(tokens, cols, 410)
    outs = be.gemm_batch("Q8_0", ws, x, rows, tokens, cols)
    for w, r, o in zip(ws, rows, outs):
        assert_parity(o, zo.gemm(Q8_0, w, x, tokens, r, cols, int8_acts=True), what=f"batched gemm rows={r}")
        assert np.array_equal(o, be.gemm("Q8_0", w, x, tokens, r, cols))
        be.release_weights(w)


def test_gemm_batch_numbers_row_tiles_through_the_tensors(be, zo):
    # 100 + 25 + 25 = 150 row tiles in one launch on 148 SMs: the K tiles are shared evenly and the cuts fall inside tiles of
    # different tensors; the second tensor ends in a ragged tile; the fourth tensor goes into a second launch
    cols, rows, tokens = 1024, [12800, 3190, 3200, 130], 40
    ws = [seeded_weights(Q8_0, r, cols, 430 + i) for i, r in enumerate(rows)]
    x = seeded_acts(tokens, cols, 440)
    outs = be.gemm_batch("Q8_0", ws, x, rows, tokens, cols)
    for w, r, o in zip(ws, rows, outs):
        assert_parity(o, zo.gemm(Q8_0, w, x, tokens, r, cols, int8_acts=True), what=f"batched gemm rows={r}")
        be.release_weights(w)


def test_config1_full_size(be, zo):
    # activations 512 x 4096 N(0,1) seed 2, W 14336 x 4096 N(0,.02) seed 3 -> Q8_0
    tokens, rows, cols = 512, 14336, 4096
    w = seeded_weights(Q8_0, rows, cols, 3)
    x = seeded_acts(tokens, cols, 2)
    got = be.gemm("Q8_0", w, x, tokens, rows, cols)
    assert assert_parity(got, ref_f64(zo, w, x, rows, cols), what="config 1 vs float64 int8 restatement") < 2e-4
    # a sample of rows through the C oracle itself
    sel = np.arange(0, rows, 997)
    sub = np.ascontiguousarray(w[sel])
    ref = zo.gemm(Q8_0, sub, x[:32], 32, len(sel), cols, int8_acts=True)
    assert_parity(got[:32][:, sel], ref, what="config 1 sampled rows vs oracle")
    be.release_weights(w)


# ---- fp32-equivalent activations (two int8 digits per element) on the same tensor-core kernel: the counterpart of the
# reference's default prefill path, which takes fp32 activations (src/quant.cpp:1667-1680, kernels/avx2.cpp:878-1248)

@pytest.fixture()
def be_fp32(be):
    be.set_q8_act_mode(ACT_FP32)
    yield be
    be.set_q8_act_mode(ACT_INT8)


@pytest.mark.parametrize("tokens,rows,cols", [
    (9, 128, 128), (16, 100, 544), (17, 300, 96), (33, 67, 32), (64, 256, 4096), (65, 130, 2048),
    (129, 129, 4096), (171, 2048, 2048), (256, 1000, 14336), (300, 4096, 4096)])
def test_gemm_fp32_mode_vs_fp32_oracle(be_fp32, zo, tokens, rows, cols):
    w = seeded_weights(Q8_0, rows, cols, 500 + rows)
    x = seeded_acts(tokens, cols, 600 + tokens)
    x[0, :32] = 0.0                                   # an all-zero block: scale 0, both digits 0
    x[1 % tokens, 5] = 20.0                           # a 20-sigma outlier stretches its block's scale (the digits resolve amax / 65024)
    got = be_fp32.gemm("Q8_0", w, x, tokens, rows, cols)
    if tokens * rows * cols <= 64 * 256 * 4096:
        assert_parity(got, zo.gemm(Q8_0, w, x, tokens, rows, cols, int8_acts=False), what=f"fp32-mode gemm {tokens}x{rows}x{cols} vs oracle")
    rel = assert_parity(got, ref_fp32_f64(Q8_0, w, x, rows, cols), what=f"fp32-mode gemm {tokens}x{rows}x{cols} vs float64")
    assert rel < 3e-4                                 # 16-bit fixed point per 256-group (the outlier stretches its group's unit): inside the bar
    be_fp32.release_weights(w)


def test_gemm_fp32_mode_token_ladder_from_reference(be_fp32, zo):
    # tests/core_tests.cpp:345-372 again, now against the fp32-activation kernels the reference runs by default there.
    # Unit block scales and codes up to +-128 make this the hard case for two activation digits: an activation is
    # resolved to d_x / 512, so a result may be off by sum_k |w[r,k]| * d_x[t, block(k)] / 512.  The test holds the kernel
    # to that bound element by element (plus the gate on max_abs / max_ref); the reference's own absolute gate of 1e-3
    # on results near zero is missed here by a factor of about 1.4, which the two-digit scheme cannot close.
    rows, cols = 100, 544
    r = np.arange(rows)[:, None, None]
    blk = np.arange(17)[None, :, None]
    j = np.arange(2, 34)[None, None, :]
    packed = np.zeros((rows, 17, 34), np.uint8)
    packed[..., 1] = 0x3C
    packed[..., 2:] = (r * 5 + blk * 11 + j * 3) & 255
    packed = np.ascontiguousarray(packed.reshape(rows, -1))
    w_abs = np.abs(blocks.dequantize(Q8_0, packed, rows, cols).astype(np.float64)).reshape(rows, 17, 32).sum(axis=2)    # [rows, blocks]
    for T in (9, 16, 32, 171):
        t = np.arange(T)[:, None]
        c = np.arange(cols)[None, :]
        xin = (((t * 7 + c) % 15 - 7).astype(np.float32) * np.float32(0.017)).astype(np.float32)
        got = be_fp32.gemm("Q8_0", packed, xin, T, rows, cols).astype(np.float64)
        ref = ref_fp32_f64(Q8_0, packed, xin, rows, cols)
        assert np.abs(got - ref).max() / np.abs(ref).max() < 1e-4
        d_x = zo.quantise_acts(xin)[1].astype(np.float64)                       # [T, blocks]
        bound = d_x @ w_abs.T / 512.0 + 1e-5 * np.maximum(1.0, np.abs(ref))     # + fp32 accumulation slack
        assert np.all(np.abs(got - ref) <= bound), float((np.abs(got - ref) / bound).max())
        assert np.abs(got - ref).max() < 3e-3
    be_fp32.release_weights(packed)


def test_gemm_fp32_mode_batch_and_device_call(be_fp32, zo):
    import torch
    cols, rows, tokens = 1024, [12800, 3190, 3200, 130], 40      # 150 row tiles in one launch and a second launch
    ws = [seeded_weights(Q8_0, r, cols, 530 + i) for i, r in enumerate(rows)]
    x = seeded_acts(tokens, cols, 540)
    outs = be_fp32.gemm_batch("Q8_0", ws, x, rows, tokens, cols)
    for w, r, o in zip(ws, rows, outs):
        assert_parity(o, ref_fp32_f64(Q8_0, w, x, r, cols), what=f"fp32-mode batched gemm rows={r}")
    # device pointers: same kernel, caller's workspace
    handles = [be_fp32.dev_upload("Q8_0", w, r, cols) for w, r in zip(ws[:3], rows[:3])]
    d_x = torch.from_numpy(x).cuda()
    d_out = [torch.empty(tokens, r, device="cuda") for r in rows[:3]]
    nbytes = be_fp32.gemm_workspace_bytes(tokens, cols, ACT_FP32)
    assert nbytes > be_fp32.gemm_workspace_bytes(tokens, cols, ACT_INT8)
    ws_dev = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    be_fp32.dev_gemm_q8_0(handles, [o.data_ptr() for o in d_out], d_x.data_ptr(), tokens, ws_dev.data_ptr(), nbytes, act_mode=ACT_FP32)
    be_fp32.dev_check()
    for o, host in zip(d_out, outs):
        assert np.array_equal(o.cpu().numpy(), host)
    with pytest.raises(BackendError, match="workspace too small"):
        be_fp32.dev_gemm_q8_0(handles, [o.data_ptr() for o in d_out], d_x.data_ptr(), tokens, ws_dev.data_ptr(),
                              be_fp32.gemm_workspace_bytes(tokens, cols, ACT_INT8), act_mode=ACT_FP32)
    for h in handles:
        be_fp32.dev_free(h)
    for w in ws:
        be_fp32.release_weights(w)


def test_config1_full_size_fp32_mode(be_fp32, zo):
    tokens, rows, cols = 512, 14336, 4096
    w = seeded_weights(Q8_0, rows, cols, 3)
    x = seeded_acts(tokens, cols, 2)
    got = be_fp32.gemm("Q8_0", w, x, tokens, rows, cols)
    rel = assert_parity(got, ref_fp32_f64(Q8_0, w, x, rows, cols), what="config 1, fp32-equivalent activations, vs float64")
    assert rel < 3e-4
    sel = np.arange(0, rows, 997)
    sub = np.ascontiguousarray(w[sel])
    assert_parity(got[:32][:, sel], zo.gemm(Q8_0, sub, x[:32], 32, len(sel), cols, int8_acts=False), what="config 1 sampled rows vs the fp32 oracle")
    be_fp32.release_weights(w)


@pytest.mark.parametrize("int8", [False, True])
@pytest.mark.parametrize("tokens,rows,cols", [(9, 128, 256), (40, 300, 4096), (130, 257, 2048), (16, 64, 14336)])
def test_group_scale_kernel_equals_its_restatement(zo, tokens, rows, cols, int8):
    # the kernel against helpers.group_product: the same digits, the same integer sums, the same fp32 steps group by group.
    # Few enough tiles that no tile's K range is split between two CTAs (a split adds two partial sums in another order).
    import torch
    from helpers import group_product
    from zeninfer_b200 import Backend
    from zeninfer_b200.backend import ACT_FP32, ACT_INT8
    be = Backend()
    w = seeded_weights(Q8_0, rows, cols, 700 + rows)
    x = seeded_acts(tokens, cols, 710 + tokens)
    x[0, :256] = 0.0
    h = be.dev_upload("Q8_0", w, rows, cols)
    mode = ACT_INT8 if int8 else ACT_FP32
    ws_bytes = be.gemm_workspace_bytes(tokens, cols, mode)
    ws = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda")
    y = torch.full((tokens, rows), float("nan"), device="cuda")
    d_x = torch.from_numpy(x).cuda()
    be.dev_gemm_q8_0([h], [y.data_ptr()], d_x.data_ptr(), tokens, ws.data_ptr(), ws_bytes, act_mode=mode)
    be.dev_check()
    got = y.cpu().numpy()
    be.dev_free(h)
    xv = x
    if int8:
        xq, xsc = zo.quantise_acts(x)
        xv = (xq.astype(np.float32).reshape(tokens, -1, 32) * xsc.astype(np.float32)[..., None]).reshape(tokens, cols)
    want = group_product(blocks.dequantize(Q8_0, w, rows, cols), xv)
    # equal up to the last bit of a step here and there: the restatement rounds a fused multiply-add through float64
    assert np.abs(got.astype(np.float64) - want).max() <= 2e-6 * np.abs(want).max()
    assert np.mean(got == want) > 0.9


# A launch of many row tiles takes the narrowest of the four tile widths that holds its tokens: each width, full and one token into
# the next.
@pytest.mark.parametrize("tokens", [20, 32, 33, 64, 65, 96, 97])
def test_group_scale_tiles_of_every_width(zo, tokens):
    test_group_scale_kernel_equals_its_restatement(zo, tokens, 18944, 512, False)


@pytest.mark.parametrize("tokens", [8, 60, 77, 128])
def test_group_scale_tiles_split_between_two_ctas(tokens):
    # 149 row tiles: most are split, so a result is the sum of two partial sums and may differ from the restatement's by their roundings
    import torch
    from helpers import group_product
    from zeninfer_b200 import Backend
    be, rows, cols = Backend(), 19072, 512
    w, x = seeded_weights(Q8_0, rows, cols, 721), seeded_acts(tokens, cols, 722)
    h = be.dev_upload("Q8_0", w, rows, cols)
    ws_bytes = be.gemm_workspace_bytes(tokens, cols, ACT_FP32)
    ws, y, d_x = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda"), torch.full((tokens, rows), float("nan"), device="cuda"), torch.from_numpy(x).cuda()
    torch.cuda.synchronize()
    be.dev_gemm_q8_0([h], [y.data_ptr()], d_x.data_ptr(), tokens, ws.data_ptr(), ws_bytes, act_mode=ACT_FP32)
    be.dev_check()
    got = y.cpu().numpy()
    be.dev_free(h)
    want = group_product(blocks.dequantize(Q8_0, w, rows, cols), x)
    assert np.abs(got.astype(np.float64) - want).max() <= 2e-6 * np.abs(want).max()


# Split tiles of several token tiles: 96 columns (149 row tiles, 180 tokens) and 128 (40 row tiles, 500 tokens).
@pytest.mark.parametrize("tokens,rows,cols", [(180, 19072, 512), (500, 5120, 512)])
def test_group_scale_split_tiles_of_several_token_tiles(tokens, rows, cols):
    check_split_products(tokens, [rows], cols)


def test_group_scale_second_launch_with_split_tiles():
    # four tensors: the first three are one launch, whose split tiles are cleared beside the digits, the fourth another behind a
    # launch that clears its own
    check_split_products(30, [12800, 3190, 3200, 19072], 512)


def check_split_products(tokens, rows, cols):
    import torch
    from helpers import group_product
    from zeninfer_b200 import Backend
    be = Backend()
    ws, x = [seeded_weights(Q8_0, r, cols, 741 + i) for i, r in enumerate(rows)], seeded_acts(tokens, cols, 740)
    handles = [be.dev_upload("Q8_0", w, r, cols) for w, r in zip(ws, rows)]
    nbytes = be.gemm_workspace_bytes(tokens, cols, ACT_FP32)
    scratch, d_x = torch.zeros(nbytes, dtype=torch.uint8, device="cuda"), torch.from_numpy(x).cuda()
    outs = [torch.full((tokens, r), float("nan"), device="cuda") for r in rows]
    torch.cuda.synchronize()
    be.dev_gemm_q8_0(handles, [o.data_ptr() for o in outs], d_x.data_ptr(), tokens, scratch.data_ptr(), nbytes, act_mode=ACT_FP32)
    be.dev_check()
    for h, w, o, r in zip(handles, ws, outs, rows):
        be.dev_free(h)
        want = group_product(blocks.dequantize(Q8_0, w, r, cols), x)
        assert np.abs(o.cpu().numpy().astype(np.float64) - want).max() <= 2e-6 * np.abs(want).max()     # two partial sums: two roundings


def test_group_scale_product_in_place():
    # the output over the activations, 160 tiles (most of them split and cleared first): cleared only once the digits are formed, in a
    # launch of its own
    import torch
    from zeninfer_b200 import Backend
    be, n, tokens = Backend(), 2560, 1000
    w, x = seeded_weights(Q8_0, n, n, 731), seeded_acts(tokens, n, 732)
    h = be.dev_upload("Q8_0", w, n, n)
    ws_bytes = be.gemm_workspace_bytes(tokens, n, ACT_FP32)
    ws, y, d_x = torch.zeros(ws_bytes, dtype=torch.uint8, device="cuda"), torch.full((tokens, n), float("nan"), device="cuda"), torch.from_numpy(x).cuda()
    torch.cuda.synchronize()

    def product(out):
        before = be.stats()["dispatches"]
        be.dev_gemm_q8_0([h], [out.data_ptr()], d_x.data_ptr(), tokens, ws.data_ptr(), ws_bytes, act_mode=ACT_FP32)
        be.dev_check()
        return be.stats()["dispatches"] - before

    product(y)
    launches = product(y)
    want = y.cpu().numpy()
    assert product(d_x) == launches + 1
    be.dev_free(h)
    assert np.array_equal(d_x.cpu().numpy(), want)
