"""Parity of the CUDA kernels (called through the C ABI) with the oracle.

Tolerances are the ones the project states for this path: relative Frobenius
error <= 1e-4 on factors and inverses, <= 1e-3 on preconditioned gradients.
Pack/unpack is bit-exact.
"""

import numpy as np
import pytest
import torch

from oracle import kfac_oracle as orc
import bench_workloads as bw

pytestmark = pytest.mark.gpu

FACTOR_TOL = 1e-4
INVERSE_TOL = 1e-4
KFGRAD_TOL = 1e-3


@pytest.fixture(scope='module')
def ops():
    from chainerkfac_b200 import ops as _ops
    return _ops


@pytest.fixture(autouse=True, params=[1, 0], ids=['tcgen05', 'fp32'])
def engine(request):
    """Every test runs on both arithmetic engines: tcgen05 tensor cores with
    operands in terms (the default) and the fp32 FFMA tiles.  After a run the
    status word must be clean (no barrier wait ran out)."""
    import ctypes
    from chainerkfac_b200 import _lib
    lib = _lib.load()
    _lib.check(lib.kfac_set_engine(request.param), 'kfac_set_engine')
    yield request.param
    status = ctypes.c_int(-1)
    _lib.check(lib.kfac_tc_status(ctypes.byref(status)), 'kfac_tc_status')
    _lib.check(lib.kfac_set_engine(1), 'kfac_set_engine')
    assert status.value == 0


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def host(t):
    return t.detach().cpu().numpy()


def rel(a, b):
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


def check_symmetric(m):
    assert np.array_equal(m, m.T), 'factor is not bit-symmetric'


# ------------------------------------------------------------------ factors
@pytest.mark.parametrize('name', ['linear_bias', 'linear_nobias', 'linear_odd'])
def test_factor_linear_golden(ops, golden, name):
    g = golden(name)
    bias = 'b' in g
    x, gy = g['x0'], g['gy0']
    n = x.shape[0]
    A = host(ops.factor_dense(dev(x), bias, alpha=1.0 / n))
    G = host(ops.factor_dense(dev(gy), False, alpha=float(n)))
    assert rel(A, g['A0']) < FACTOR_TOL
    assert rel(G, g['G0']) < FACTOR_TOL
    check_symmetric(A)
    check_symmetric(G)


@pytest.mark.parametrize('name', ['conv3x3_bias', 'conv3x3_s2', 'conv1x1_s2',
                                  'conv7x7_s2'])
def test_factor_conv_golden(ops, golden, name):
    g = golden(name)
    bias = 'b' in g
    x, gy = g['x0'], g['gy0']
    n, _, ho, wo = gy.shape
    A = host(ops.factor_conv_input(dev(x), int(g['ksize']), int(g['stride']),
                                   int(g['pad']), bias, alpha=1.0 / n))
    G = host(ops.factor_conv_grad(dev(gy), alpha=n / float(ho * wo)))
    assert rel(A, g['A0']) < FACTOR_TOL
    assert rel(G, g['G0']) < FACTOR_TOL
    check_symmetric(A)


@pytest.mark.parametrize('rows,d,bias', [
    (32, 10, False), (128, 27, True), (128, 784, True), (128, 1000, True),
    (5000, 64, False), (40000, 147, True), (3000, 513, False), (1, 5, True),
    (17, 129, True), (2049, 300, False),
    # 256-row tile pairs: odd number of 128-row blocks with a bias column and
    # a cut contraction; six 256-row blocks, the last with 20 rows
    (70000, 600, True), (6272, 1300, False)])
def test_factor_dense_sweep(ops, rows, d, bias):
    rng = np.random.default_rng(rows * 131 + d)
    x = np.maximum(rng.standard_normal((rows, d)), 0).astype(np.float32)
    want = orc.linear_A(x.astype(np.float64), bias) * rows / 7.0
    got = host(ops.factor_dense(dev(x), bias, alpha=1.0 / 7.0))
    assert got.shape == want.shape
    assert rel(got, want) < FACTOR_TOL
    check_symmetric(got)


def test_factor_dense_strided_rows(ops):
    rng = np.random.default_rng(5)
    big = dev(rng.standard_normal((300, 96)).astype(np.float32))
    x = big[:, :50]                      # leading dimension 96
    from chainerkfac_b200 import _lib
    import ctypes
    lib = _lib.load()
    out = torch.empty((50, 50), device='cuda')
    ws = torch.empty(max(lib.kfac_factor_workspace_bytes(300, 50), 256),
                     dtype=torch.uint8, device='cuda')
    _lib.check(lib.kfac_factor_dense(
        ctypes.c_void_p(x.data_ptr()), 300, 50, 96, 0, 1.0, 0.0,
        ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(ws.data_ptr()),
        ws.numel(), None), 'strided')
    torch.cuda.synchronize()
    xs = host(big)[:, :50].astype(np.float64)
    assert rel(host(out), xs.T @ xs) < FACTOR_TOL


def test_factor_running_average_and_accumulation(ops):
    rng = np.random.default_rng(9)
    x1 = rng.random((64, 33)).astype(np.float32)
    x2 = rng.random((64, 33)).astype(np.float32)
    r = 0.9
    ema = ops.factor_dense(dev(x1), True, alpha=1.0 / 64)
    ops.factor_dense(dev(x2), True, alpha=r / 64, beta=1 - r, out=ema)
    want = orc.update_cov_ema(orc.linear_A(x2, True), orc.linear_A(x1, True), r)
    assert rel(host(ema), want) < FACTOR_TOL
    check_symmetric(host(ema))
    # long contraction (split across CTAs) with beta
    x3 = rng.random((9000, 33)).astype(np.float32)
    acc = ops.factor_dense(dev(x1), True, alpha=0.5 / 64)
    ops.factor_dense(dev(x3), True, alpha=0.5 / 9000, beta=1.0, out=acc)
    want = 0.5 * orc.linear_A(x1, True) + 0.5 * orc.linear_A(x3, True)
    assert rel(host(acc), want) < FACTOR_TOL


@pytest.mark.parametrize('n,c,h,k,s,p,bias', [
    (2, 3, 32, 7, 2, 3, True),      # stem-like
    (2, 64, 14, 3, 1, 1, False),    # 3x3, 576 columns
    (3, 16, 15, 3, 2, 1, False),    # strided 3x3, odd extent
    (2, 40, 9, 1, 1, 0, False),     # 1x1 (strided view path)
    (2, 24, 10, 1, 2, 0, True),     # 1x1 stride 2 (gather path)
    (1, 5, 6, 5, 1, 0, True),       # no padding
    (4, 512, 7, 3, 1, 1, False)])   # 4608 columns
def test_factor_conv_input_sweep(ops, n, c, h, k, s, p, bias):
    rng = np.random.default_rng(n * 7 + c + h + k)
    x = rng.standard_normal((n, c, h, h)).astype(np.float32)
    want = orc.conv_A(x.astype(np.float64), k, s, p, bias)
    got = host(ops.factor_conv_input(dev(x), k, s, p, bias, alpha=1.0 / n))
    assert got.shape == want.shape
    assert rel(got, want) < FACTOR_TOL
    check_symmetric(got)


@pytest.mark.parametrize('n,c,hw', [(2, 5, 3), (4, 64, 28), (3, 130, 7),
                                    (32, 256, 14), (2, 2048, 7)])
def test_factor_conv_grad_sweep(ops, n, c, hw):
    rng = np.random.default_rng(n + c + hw)
    gy = (rng.standard_normal((n, c, hw, hw)) / n).astype(np.float32)
    want = orc.conv_G(gy.astype(np.float64))
    got = host(ops.factor_conv_grad(dev(gy), alpha=n / float(hw * hw)))
    assert rel(got, want) < FACTOR_TOL
    check_symmetric(got)


def test_factor_group_matches_single_calls(ops):
    rng = np.random.default_rng(21)
    xd = dev(rng.random((300, 70)).astype(np.float32))
    xc = dev(rng.standard_normal((3, 16, 12, 12)).astype(np.float32))
    xs = dev(rng.standard_normal((2, 24, 10, 10)).astype(np.float32))
    gy = dev(rng.standard_normal((3, 40, 12, 12)).astype(np.float32))
    big = dev(rng.standard_normal((2, 8, 40, 40)).astype(np.float32))
    prev = dev(np.eye(71, dtype=np.float32))
    want = [
        ops.factor_dense(xd, True, alpha=0.5, beta=0.25, out=prev.clone()),
        ops.factor_conv_input(xc, 3, 1, 1, False, alpha=1 / 3.),
        ops.factor_conv_input(xs, 1, 2, 0, True, alpha=0.5),
        ops.factor_conv_grad(gy, alpha=2.0),
        ops.factor_conv_input(big, 3, 1, 1, True, alpha=1.0),
    ]
    outs = [prev.clone()] + [torch.empty_like(w) for w in want[1:]]
    items = [
        ops.dense_item(xd, True, 0.5, 0.25, outs[0]),
        ops.conv_input_item(xc, 3, 1, 1, False, 1 / 3., 0.0, outs[1]),
        ops.conv_input_item(xs, 1, 2, 0, True, 0.5, 0.0, outs[2]),
        ops.conv_grad_item(gy, 2.0, 0.0, outs[3]),
        ops.conv_input_item(big, 3, 1, 1, True, 1.0, 0.0, outs[4]),
    ]
    ops.factor_group(items, xd.device)
    for w, o in zip(want, outs):
        assert rel(host(o), host(w)) < 1e-5
        check_symmetric(host(o))
    assert rel(host(outs[1]), orc.conv_A(host(xc).astype(np.float64), 3, 1, 1,
                                         False)) < FACTOR_TOL


def test_scratch_buffers_are_per_stream(ops):
    """Factor builds issued on different CUDA streams may run at the same
    time (the exchange stream builds a low-rank block's matrix while the main
    stream builds the next size class): their partial-tile scratch must not
    be the same memory."""
    ws = ops.Workspace()
    dev0 = torch.device('cuda', torch.cuda.current_device())
    a = ws.get(1 << 20, dev0)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        b = ws.get(1 << 20, dev0)
        assert ws.get(1 << 10, dev0) is b          # grow-only, reused
    assert a.data_ptr() != b.data_ptr()
    assert ws.get(1 << 20, dev0) is a
    # and a grouped build on a side stream beside one on the main stream
    rng = np.random.default_rng(5)
    x1 = dev(rng.standard_normal((90000, 200)).astype(np.float32))
    x2 = dev(rng.standard_normal((80000, 150)).astype(np.float32))
    o1 = torch.empty((200, 200), device='cuda')
    o2 = torch.empty((150, 150), device='cuda')
    torch.cuda.synchronize()
    for _ in range(3):
        ops.factor_group([ops.dense_item(x1, False, 1.0 / 90000, 0.0, o1)],
                         dev0)
        with torch.cuda.stream(side):
            ops.factor_group([ops.dense_item(x2, False, 1.0 / 80000, 0.0, o2)],
                             dev0)
    torch.cuda.synchronize()
    w1 = host(x1).astype(np.float64)
    w2 = host(x2).astype(np.float64)
    assert rel(host(o1), w1.T @ w1 / 90000) < FACTOR_TOL
    assert rel(host(o2), w2.T @ w2 / 80000) < FACTOR_TOL


@pytest.mark.parametrize('channels_last', [False, True])
@pytest.mark.parametrize('n,c,h,w,stride', [
    (2, 32, 8, 8, 1), (3, 33, 5, 9, 1), (1, 64, 1, 1, 1), (2, 64, 14, 1, 1),
    (5, 70, 7, 7, 1), (4, 128, 9, 6, 1), (2, 257, 4, 4, 1), (33, 512, 7, 7, 1),
    (2, 130, 41, 40, 2), (6, 32, 8, 8, 1), (43, 33, 3, 3, 1),
    (32, 70, 7, 2, 1), (28, 129, 2, 7, 1), (8, 128, 9, 6, 1),
    (28, 257, 4, 4, 1), (200, 64, 2, 2, 1)])
def test_factor_of_3x3_convolutions(ops, engine, n, c, h, w, stride,
                                    channels_last):
    """Patch factors as shifted products (one granule of channels, ragged
    granules, several tiles, the smallest images and pixel counts that go there)
    and from staged patches (images of one or two rows or columns, few pixels,
    stride 2), on top of an existing average, against fp64."""
    if engine == 0 and channels_last:
        pytest.skip('channels-last inputs belong to the tensor-core engine')
    torch.manual_seed(2)
    x = torch.randn(n, c, h, w, device='cuda').clamp_(min=0)
    u = torch.nn.functional.unfold(x.double(), 3, padding=1, stride=stride)
    u = u.transpose(1, 2).reshape(-1, 9 * c)
    if channels_last:
        x = x.contiguous(memory_format=torch.channels_last)
    out = torch.full((9 * c, 9 * c), 3.0, device='cuda')
    ops.factor_group([ops.conv_input_item(x, 3, stride, 1, False, 1.0 / n, 0.5,
                                          out)], x.device)
    ref = u.t() @ u / n + 1.5
    assert rel(host(out), host(ref)) < FACTOR_TOL
    check_symmetric(host(out))


@pytest.mark.parametrize('n,c,h,w', [
    (32, 64, 1, 1), (128, 70, 1, 1), (32, 256, 2, 2), (40, 32, 1, 9)])
def test_taps_outside_small_images_stay_zero(ops, n, c, h, w):
    """Entries between taps that never see the image at the same position are
    sums of zeros; nothing is left there by larger sums."""
    torch.manual_seed(7)
    x = torch.rand(n, c, h, w, device='cuda') + 1.0
    out = torch.full((9 * c, 9 * c), 3.0, device='cuda')
    ops.factor_group([ops.conv_input_item(x, 3, 1, 1, False, 1.0 / n, 0.0,
                                          out)], x.device)
    u = torch.nn.functional.unfold(x.double(), 3, padding=1)
    u = u.transpose(1, 2).reshape(-1, 9 * c)
    ref = u.t() @ u / n
    assert rel(host(out), host(ref)) < FACTOR_TOL
    assert bool((ref == 0).any())
    assert float(out[ref == 0].abs().max()) == 0.0


@pytest.mark.parametrize('b2', [0.0, 0.75])
def test_factor_group_second_output(ops, engine, b2):
    """Running averages kept up to date by the build: factors that are
    assembled from shifted products (432 pixels), reduced from wide and narrow
    pieces, built by the gather kernel, and one without a second array."""
    torch.manual_seed(5)
    xc = torch.randn(6, 40, 9, 8, device='cuda')
    xs = [torch.randn(r, d, device='cuda')
          for r, d in ((2100, 1028), (40000, 60), (70, 33), (50, 20))]
    u = torch.nn.functional.unfold(xc.double(), 3, padding=1)
    mats = [u.transpose(1, 2).reshape(-1, 360)] + [x.double() for x in xs]
    outs = [torch.empty(m.shape[1], m.shape[1], device='cuda') for m in mats]
    second = [torch.full_like(o, 3.0) for o in outs[:4]] + [None]
    items = [ops.conv_input_item(xc, 3, 1, 1, False, 0.5, 0.0, outs[0])] + [
        ops.dense_item(x, False, 0.5, 0.0, o) for x, o in zip(xs, outs[1:])]
    ops.factor_group(items, xc.device, second, 0.25, b2)
    for m, o, s in zip(mats, outs, second):
        ref = 0.5 * (m.t() @ m)
        assert rel(host(o), host(ref)) < FACTOR_TOL
        if s is not None:
            assert rel(host(s), host(0.25 * ref + b2 * 3.0)) < FACTOR_TOL
            check_symmetric(host(s))


@pytest.mark.parametrize('rows,d,ones', [
    (2000, 1024, False), (1999, 1025, False), (1500, 1411, True)])
def test_wide_factor_from_staged_planes(ops, rows, d, ones):
    """Tiles, strips and granules that the last column cuts."""
    torch.manual_seed(3)
    x = torch.randn(rows, d - int(ones), device='cuda')
    out = torch.full((d, d), 3.0, device='cuda')
    ops.factor_group([ops.dense_item(x, ones, 0.5, 0.5, out)], x.device)
    xd = x.double()
    if ones:
        xd = torch.cat([xd, xd.new_ones(rows, 1)], 1)
    assert rel(host(out), host(0.5 * (xd.t() @ xd) + 1.5)) < FACTOR_TOL
    check_symmetric(host(out))
    xt = x.t().contiguous()
    if not ones:
        ops.factor_group([ops.dense_t_item(xt, 1.0, 0.0, out)], x.device)
        assert rel(host(out), host(xd.t() @ xd)) < FACTOR_TOL


@pytest.mark.parametrize('n,c,h,w', [
    (300, 60, 8, 8), (32, 64, 28, 28), (257, 100, 8, 5), (65, 128, 13, 12),
    (1000, 256, 2, 2), (40, 200, 12, 12), (31, 260, 12, 12), (9, 1028, 11, 12)])
@pytest.mark.parametrize('channels_last', [False, True])
def test_factor_of_plain_operands_read_by_tma(ops, n, c, h, w, channels_last):
    """Gradient factors of a million elements and more: one tile of 64, 128
    and 256 columns and several, cut last rows and columns, images that are no
    multiple of a k-block, on top of an existing average, against fp64."""
    torch.manual_seed(4)
    g = torch.randn(n, c, h, w, device='cuda')
    m = g.permute(0, 2, 3, 1).reshape(-1, c).double()
    if channels_last:
        g = g.contiguous(memory_format=torch.channels_last)
    out = torch.full((c, c), 3.0, device='cuda')
    ops.factor_group([ops.conv_grad_item(g, 2.0, 0.5, out)], g.device)
    assert rel(host(out), host(2.0 * (m.t() @ m) + 1.5)) < FACTOR_TOL
    check_symmetric(host(out))


@pytest.mark.parametrize('kblocks,d,ones', [
    (129, 64, False), (196, 256, False), (255, 512, False), (230, 1028, False),
    (255, 130, True), (380, 250, True)])
def test_long_contractions_are_cut_in_groups(ops, engine, kblocks, d, ones):
    """Beside work that fills the chip many times over, a contraction a little
    longer than one CTA may accumulate is cut all the same.  Non-negative values:
    the truncating accumulator drifts by up to 2^-25 per MMA, six per 32 rows, of
    at most 128 (gather kernel, for appended columns: 256) 32-row blocks; what the
    two-term split leaves out (2^-17 of a value, of either sign) averages out."""
    if engine == 0:
        pytest.skip('the limit belongs to the tensor-core engine')
    torch.manual_seed(8)
    big = torch.rand(65536, 1024, device='cuda')
    x = torch.rand(32 * kblocks, d - int(ones), device='cuda')
    out = torch.empty(d, d, device='cuda')
    outs = [torch.empty(1024, 1024, device='cuda') for _ in range(6)]
    bigs = [torch.empty(250, 250, device='cuda') for _ in range(12)]
    ops.factor_group(
        [ops.dense_item(x, ones, 1.0, 0.0, out)] +
        [ops.dense_item(big, False, 1.0, 0.0, o) for o in outs] +
        [ops.dense_item(big.view(-1, 256)[:, :249].contiguous(), True, 1.0,
                        0.0, o) for o in bigs], x.device)
    xd = x.double()
    if ones:
        xd = torch.cat([xd, xd.new_ones(32 * kblocks, 1)], 1)
    limit = 256 if ones else 128
    assert rel(host(out), host(xd.t() @ xd)) < 6 * limit * 2.0 ** -25
    bd = big.double()
    assert rel(host(outs[3]), host(bd.t() @ bd)) < 6 * 128 * 2.0 ** -25


@pytest.mark.parametrize('build', ['dense', 'ones', 'conv_grad', 'conv_1x1',
                                   'group_of_one'])
def test_lone_factor_in_a_captured_graph(ops, engine, build):
    """A factor built on its own can be recorded into a graph: replayed after
    other builds, it reads its operand anew and nothing else that is gone."""
    torch.manual_seed(12)
    shape = (64, 256, 12, 12) if build.startswith('conv') else (9000, 256)
    x = torch.randn(shape, device='cuda')
    d = 257 if build == 'ones' else 256
    out = torch.empty(d, d, device='cuda')

    def call():
        if build in ('dense', 'ones'):
            ops.factor_dense(x, build == 'ones', alpha=0.5, out=out)
        elif build == 'conv_grad':
            ops.factor_conv_grad(x, alpha=0.5, out=out)
        elif build == 'conv_1x1':
            ops.factor_conv_input(x, 1, 1, 0, alpha=0.5, out=out)
        else:
            ops.factor_group([ops.dense_item(x, False, 0.5, 0.0, out)],
                             x.device)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        call()
    x.normal_()
    other = torch.randn(20000, 256, device='cuda')
    for _ in range(20):
        ops.factor_dense(other, False)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    m = x.double()
    m = m.permute(0, 2, 3, 1).reshape(-1, 256) if m.dim() == 4 else m
    if build == 'ones':
        m = torch.cat([m, m.new_ones(m.shape[0], 1)], 1)
    assert rel(host(out), host(0.5 * (m.t() @ m))) < FACTOR_TOL
    check_symmetric(host(out))


def test_group_of_several_batches(ops, engine):
    """Factors whose partial tiles do not fit the workspace of one batch
    (285 MB each), and kinds that come behind them, against fp64."""
    if engine == 0:
        pytest.skip('batches belong to the tensor-core engine')
    torch.manual_seed(9)
    x = torch.randn(32768, 4096, device='cuda')
    xc = torch.randn(3, 40, 9, 8, device='cuda')
    xs = torch.randn(1999, 1025, device='cuda')
    out = [torch.empty(4096, 4096, device='cuda') for _ in range(9)]
    oc = [torch.empty(360, 360, device='cuda') for _ in range(2)]
    os = torch.empty(1025, 1025, device='cuda')
    items = [ops.conv_input_item(xc, 3, 1, 1, False, 1.0, 0.0, oc[0])] + [
        ops.dense_item(x, False, 2.0 ** -i, 0.0, o)
        for i, o in enumerate(out)] + [
        ops.conv_input_item(xc, 3, 1, 1, False, 1.0, 0.0, oc[1]),
        ops.dense_item(xs, False, 1.0, 0.0, os)]
    ops.factor_group(items, x.device)
    ref = x.double().t() @ x.double()
    for i, o in enumerate(out):
        assert float((o.double() * 2.0 ** i - ref).norm() / ref.norm()) < \
            FACTOR_TOL
    u = torch.nn.functional.unfold(xc.double(), 3, padding=1)
    u = u.transpose(1, 2).reshape(-1, 360)
    assert all(rel(host(o), host(u.t() @ u)) < FACTOR_TOL for o in oc)
    xd = xs.double()
    assert rel(host(os), host(xd.t() @ xd)) < FACTOR_TOL


def test_factor_builds_from_staged_operands(ops, engine):
    """The optional operand feed of the factor builds (staging pass that
    writes X^T as two bf16 planes, TMA boxes into the tile kernel) against the
    oracle and against the default feed: every operand kind and layout,
    ragged sizes, a cut contraction, the appended ones column."""
    from chainerkfac_b200 import _lib
    if engine == 0:
        pytest.skip('the staged feed belongs to the tensor-core engine')
    lib = _lib.load()
    rng = np.random.default_rng(77)

    def arr(*shape):
        return dev(rng.standard_normal(shape).astype(np.float32))

    xd, xs = arr(5000, 300), arr(70, 33)
    xl = arr(70000, 130)                      # several splits
    xc, x2, x7 = arr(4, 16, 14, 14), arr(2, 8, 15, 15), arr(2, 3, 30, 30)
    xn = arr(4, 32, 8, 8).contiguous(memory_format=torch.channels_last)
    x1 = arr(3, 24, 6, 6).contiguous(memory_format=torch.channels_last)
    gy = arr(3, 40, 12, 12)
    gn = arr(3, 40, 5, 5).contiguous(memory_format=torch.channels_last)
    xt = arr(48, 1000)
    cases = [
        lambda o: ops.dense_item(xd, True, 1 / 5000., 0.0, o),
        lambda o: ops.dense_item(xs, False, 1.0, 0.0, o),
        lambda o: ops.dense_item(xl, True, 1 / 70000., 0.0, o),
        lambda o: ops.conv_input_item(xc, 3, 1, 1, True, 0.25, 0.0, o),
        lambda o: ops.conv_input_item(x2, 3, 2, 1, False, 0.5, 0.0, o),
        lambda o: ops.conv_input_item(x7, 7, 2, 3, True, 0.5, 0.0, o),
        lambda o: ops.conv_input_item(xn, 3, 1, 1, True, 0.25, 0.0, o),
        lambda o: ops.conv_input_item(x1, 1, 1, 0, False, 1.0, 0.0, o),
        lambda o: ops.conv_grad_item(gy, 2.0, 0.0, o),
        lambda o: ops.conv_grad_item(gn, 2.0, 0.0, o),
        lambda o: ops.dense_t_item(xt, 1.0, 0.0, o),
    ]
    sides = [301, 33, 131, 145, 72, 148, 289, 24, 40, 40, 48]
    results = {}
    for staged in (0, 1):
        lib.kfac_set_factor_staging(staged)
        try:
            outs = [torch.full((d, d), 7.0, device='cuda') for d in sides]
            ops.factor_group([c(o) for c, o in zip(cases, outs)], xd.device)
            # a lone factor takes the by-value descriptor path
            lone = ops.factor_conv_input(xc, 3, 1, 1, True, alpha=0.25)
            torch.cuda.synchronize()
            results[staged] = [host(o) for o in outs] + [host(lone)]
        finally:
            lib.kfac_set_factor_staging(0)
    for k, (a, b) in enumerate(zip(results[1], results[0])):
        assert rel(a, b) < 2e-6, (k, rel(a, b))
        check_symmetric(a)
    want = orc.conv_A(host(xc).astype(np.float64), 3, 1, 1, True)
    assert rel(results[1][3], want) < FACTOR_TOL
    want = orc.conv_A(host(xn).astype(np.float64), 3, 1, 1, True)
    assert rel(results[1][6], want) < FACTOR_TOL
    want = host(xl).astype(np.float64)
    want = np.concatenate([want, np.ones((70000, 1))], 1)
    assert rel(results[1][2], want.T @ want / 70000.) < FACTOR_TOL
    assert rel(results[1][10],
               host(xt).astype(np.float64) @ host(xt).astype(np.float64).T) \
        < FACTOR_TOL


@pytest.mark.parametrize('name', ['bn_4d', 'bn_2d'])
def test_bn_factor_golden(ops, golden, name):
    g = golden(name)
    x, gy = g['x'], g['gy']
    n = x.shape[0]
    grads = ops.bn_sample_grads(dev(x), dev(gy), float(g['eps']), float(n))
    want = orc.bn_sample_grads(x, gy, float(g['eps']))
    assert rel(host(grads), want) < FACTOR_TOL
    F = host(ops.factor_dense(grads, False, alpha=1.0 / n))
    assert rel(F, g['F']) < FACTOR_TOL


def test_bounded_wait_expires_and_reports(ops):
    """A barrier wait that can never be satisfied gives up after its poll
    limit, raises its status word and lets the kernel return (the mechanism
    every tile kernel's waits use); the context stays usable."""
    import ctypes
    from chainerkfac_b200 import _lib
    lib = _lib.load()
    status, returned = ctypes.c_int(-1), ctypes.c_int(-1)
    _lib.check(lib.kfac_selftest_wait_expiry(ctypes.byref(status),
                                             ctypes.byref(returned)),
               'kfac_selftest_wait_expiry')
    assert status.value == 1 and returned.value == 2
    x = torch.ones(4, 3, device='cuda')
    assert float(ops.factor_dense(x, False, alpha=1.0).sum()) == 36.0


# ------------------------------------------------------------------ inverse
def spd(rng, d, m=None):
    m = m or max(2 * d, 64)
    X = rng.standard_normal((m, d)).astype(np.float32)
    return (X.T @ X / m + 1e-3 * np.eye(d)).astype(np.float32)


def run_pairs(ops, dimsA, dimsG, damping, use_pi=True, seed=0):
    rng = np.random.default_rng(seed)
    mats, partner, role = [], [], []
    for i, (da, dg) in enumerate(zip(dimsA, dimsG)):
        mats += [spd(rng, da), spd(rng, dg)]
        partner += [2 * i + 1, 2 * i]
        role += [0, 1]
    F = [dev(m) for m in mats]
    inv = [torch.empty_like(f) for f in F]
    plan = ops.InversePlan(F, inv, partner, role)
    plan.run(damping, use_pi)
    torch.cuda.synchronize()
    assert host(plan.info).tolist() == [0] * len(mats)
    diag = host(plan.diag)
    for i in range(len(dimsA)):
        A, G = mats[2 * i], mats[2 * i + 1]
        pi, dA, dG = orc.connection_damping(
            A, G, damping, 0.0, 'tracenorm' if use_pi else 'none')
        assert abs(diag[2 * i] - dA) <= 1e-5 * dA
        assert abs(diag[2 * i + 1] - dG) <= 1e-5 * dG
        for m, add, got in ((A, dA, inv[2 * i]), (G, dG, inv[2 * i + 1])):
            want = orc.damped_inverse(m, np.float32(add))
            truth = np.linalg.inv(m.astype(np.float64) +
                                  float(add) * np.eye(m.shape[0]))
            got = host(got)
            assert rel(got, want) < INVERSE_TOL, (m.shape, rel(got, want))
            assert rel(got, truth) < INVERSE_TOL
            assert np.array_equal(got, got.T)
        # the factors themselves stay undamped
        assert np.array_equal(host(F[2 * i]), A)
    plan.close()


def test_inverse_small_batch(ops):
    run_pairs(ops, [10, 27, 65, 148, 300], [7, 64, 128, 129, 257], 1e-3)


def test_inverse_no_pi(ops):
    run_pairs(ops, [33, 200], [16, 130], 2.5e-4, use_pi=False, seed=3)


def test_inverse_mlp_shapes(ops):
    run_pairs(ops, [785, 1001], [1000, 10], 1e-3, seed=1)


def test_inverse_large(ops):
    run_pairs(ops, [1152, 2304], [128, 513], 2.5e-4, seed=2)


@pytest.mark.parametrize('d', [10, 65])
def test_inverse_golden(ops, golden, d):
    g = golden('inverse_%d' % d)
    F = [dev(g['a'])]
    inv = [torch.empty_like(F[0])]
    plan = ops.InversePlan(F, inv, [-1], [2], l2_coef=[0.0], scale=[0.0])
    plan.run(0.0)
    assert rel(host(inv[0]), g['inv']) < INVERSE_TOL
    plan.close()


def test_inverse_bn_role_and_repeat(ops, golden):
    g = golden('bn_4d')
    F = [dev(g['F'])]
    inv = [torch.empty_like(F[0])]
    plan = ops.InversePlan(F, inv, [-1], [2], scale=[float(g['stab_coeff'])])
    for _ in range(2):          # a plan is reusable
        plan.run(float(g['damping']))
        assert abs(host(plan.diag)[0] - g['diag']) < 1e-6 * g['diag']
        assert rel(host(inv[0]), g['F_inv']) < INVERSE_TOL
    plan.close()


def test_inverse_bn_block_floors_each_half_separately(ops):
    """gamma and beta carry their own l2_coef floors
    (batch_normalization.py:141-157): the first half of the diagonal gets
    max(l2_gamma, damping) * stab_coeff, the second max(l2_beta, damping) *
    stab_coeff."""
    rng = np.random.default_rng(21)
    c, damping, stab = 9, 1e-2, 4.0
    F = spd(rng, 2 * c)
    Fd = [dev(F)]
    inv = [torch.empty_like(Fd[0])]
    plan = ops.InversePlan(Fd, inv, [-1], [2], l2_coef=[0.05], scale=[stab],
                           l2_coef_second=[0.002])
    plan.run(damping)
    add = np.concatenate([np.full(c, max(0.05, damping) * stab),
                          np.full(c, max(0.002, damping) * stab)])
    want = np.linalg.inv(F.astype(np.float64) + np.diag(add))
    assert rel(host(inv[0]), want) < INVERSE_TOL
    assert abs(host(plan.diag)[0] - 0.05 * stab) < 1e-6
    plan.close()


def test_pivots_over_the_exponent_range(ops):
    """1 / sqrt(q) and p / sqrt(q) of the diagonal kernel against fp64, four
    values in every binade of the normal numbers and their neighbours: 2^-24 for
    the last rounding, half of that for q r, which enters the correction by half
    (and 2^-24 for p r), and 2^-45 of the approximation's squared 2^-22.9."""
    from chainerkfac_b200 import _lib
    rng = np.random.default_rng(21)
    e = np.repeat(np.arange(-126, 128), 64)
    q = np.ldexp(1.0 + rng.random(e.size), e).astype(np.float32)
    q = q[(q >= np.float32(2.0 ** -126)) & np.isfinite(q)]
    edge = np.float32([2.0 ** -126, 1.0, 2.0, 4.0,
                       np.finfo(np.float32).max])
    q = np.concatenate([q, edge, np.nextafter(edge[1:], np.float32(0))])
    p = (np.sqrt(q) * rng.uniform(-1.0, 1.0, q.size)).astype(np.float32)
    bad = np.float32([0.0, -0.0, -1.0, -np.inf, np.nan, 1e-39, -1e-39])
    n = q.size
    args = [dev(np.concatenate([q, bad])),
            dev(np.concatenate([p, np.ones_like(bad)]))]
    outs = [torch.empty_like(args[0]) for _ in range(3)]
    lib = _lib.load()
    _lib.check(lib.kfac_selftest_pivots(
        n + bad.size, *[t.data_ptr() for t in args + outs], ops._stream()),
        'kfac_selftest_pivots')
    r, quot, checked = [host(t).astype(np.float64) for t in outs]
    want = 1.0 / np.sqrt(q.astype(np.float64))
    ulp = 2.0 ** -24
    assert np.max(np.abs(r[:n] / want - 1.0)) < 1.5 * ulp + 2.0 ** -44
    assert np.array_equal(checked[:n], r[:n])
    tail = np.abs(quot[:n] - p * want) / np.abs(p * want)
    assert np.max(tail) < 2.5 * ulp + 2.0 ** -44
    # a failed pivot: NaN from then on, or one where the caller asks for it
    assert np.all(~np.isfinite(r[n:])) and np.array_equal(
        checked[n:], np.ones(bad.size))


def test_inverse_reports_non_spd(ops):
    a = np.eye(40, dtype=np.float32)
    a[17, 17] = -1.0
    F = [dev(a), dev(np.eye(6, dtype=np.float32))]
    inv = [torch.empty_like(f) for f in F]
    plan = ops.InversePlan(F, inv, [-1, -1], [2, 2], scale=[0.0, 0.0])
    plan.run(0.0)
    assert host(plan.info).tolist() == [18, 0]
    assert rel(host(inv[1]), np.eye(6)) < 1e-6
    plan.close()


@pytest.mark.parametrize('count', [255, 256, 257, 900])
def test_refined_factors_are_all_counted(ops, count):
    """Plans of more factors than a block has threads: the count is whole, and of
    the factors whose estimate exceeds the threshold."""
    rng = np.random.default_rng(count)
    F = [dev(spd(rng, 3 + i % 7)) for i in range(count)]
    inv = [torch.empty_like(f) for f in F]
    plan = ops.InversePlan(F, inv, [-1] * count, [2] * count)
    plan.run(1e-3)
    est = np.sort(plan.error_estimates())
    assert est[0] >= 0
    above = list(est[1:]) + [2 * est[-1] + 1e-6]
    for at in (0, count // 2, count - 1):
        line = float(np.float32(0.5 * (est[at] + above[at])))
        plan.set_refine(1024, line)
        for _ in range(5):
            plan.run(1e-3)
            assert plan.refined() == int((est > line).sum())
    plan.set_refine(0)
    plan.run(1e-3)
    assert plan.refined() == 0
    plan.close()


@pytest.mark.parametrize('d', [97, 130, 640, 1100, 2200])
def test_inverse_of_badly_scaled_factors(ops, d):
    """Columns whose scales span six orders of magnitude: the error of entry
    (i, j) against sqrt(inv_ii inv_jj), the bound a Cholesky factorisation has
    whatever the scales (condition of the scaled factor about 30, fp32 sums of
    at most d terms: d 2^-24 30 at worst, 4e-3 at 2200; 1e-4 as everywhere)."""
    rng = np.random.default_rng(d)
    x = rng.standard_normal((2 * d, d))
    x *= np.logspace(-3, 3, d)[rng.permutation(d)]
    f = (x.T @ x / (2 * d)).astype(np.float32)
    f = (f + f.T) / 2
    F = [dev(f)]
    inv = [torch.empty_like(F[0])]
    plan = ops.InversePlan(F, inv, [-1], [2], scale=[1.0])
    plan.run(1e-6)
    torch.cuda.synchronize()
    assert host(plan.info).tolist() == [0]
    truth = np.linalg.inv(f.astype(np.float64) + 1e-6 * np.eye(d))
    s = np.sqrt(np.diag(truth))
    got = host(inv[0])
    assert np.array_equal(got, got.T)
    assert (np.abs(got - truth) / s[:, None] / s[None, :]).max() < 1e-4
    plan.close()


@pytest.mark.parametrize('d,row,col', [(40, 30, 5), (400, 390, 5),
                                       (700, 600, 130), (1300, 1290, 700)])
def test_inverse_reports_the_first_failing_pivot(ops, d, row, col):
    """A large entry left of row `row` makes that pivot negative, wherever the
    entry takes part in a product, and no pivot before it."""
    a = np.eye(d, dtype=np.float32)
    a[row, col] = a[col, row] = 1e6
    F = [dev(a)]
    inv = [torch.empty_like(F[0])]
    plan = ops.InversePlan(F, inv, [-1], [2], scale=[0.0])
    plan.run(0.0)
    assert host(plan.info).tolist() == [row + 1]
    plan.close()


@pytest.mark.parametrize('value', [float('inf'), float('nan')])
@pytest.mark.parametrize('d,row,col', [(300, 200, 5), (1100, 1000, 20)])
def test_inverse_of_a_non_finite_factor_is_not_finite(ops, value, d, row, col):
    a = np.eye(d, dtype=np.float32)
    a[row, col] = a[col, row] = value
    F = [dev(a)]
    inv = [torch.empty_like(F[0])]
    plan = ops.InversePlan(F, inv, [-1], [2], scale=[0.0])
    plan.run(0.0)
    assert host(plan.info).tolist() == [row + 1]
    assert not np.isfinite(host(inv[0])).all()
    plan.close()


def _inverse_in(ops, F, offset):
    """Inverses by a plan whose workspace begins `offset` bytes behind a multiple
    of 256."""
    import ctypes
    from chainerkfac_b200 import _lib
    lib = _lib.load()
    n, inv = len(F), [torch.zeros_like(f) for f in F]
    dims = _lib.int_array([f.shape[0] for f in F])
    need = lib.kfac_inverse_workspace_bytes(n, dims)
    ws = torch.empty(need + 512, dtype=torch.uint8, device='cuda')
    ptr = (ws.data_ptr() + 255) // 256 * 256 + offset
    info = torch.zeros(n, dtype=torch.int32, device='cuda')
    diag = torch.zeros(n, dtype=torch.float32, device='cuda')
    plan = ctypes.c_void_p()
    _lib.check(lib.kfac_inverse_plan_create(
        n, dims, _lib.ptr_array([f.data_ptr() for f in F]),
        _lib.ptr_array([f.data_ptr() for f in inv]), _lib.int_array([-1] * n),
        _lib.int_array([2] * n), _lib.float_array([0.0] * n),
        _lib.float_array([1.0] * n), ctypes.c_void_p(ptr), need,
        ctypes.byref(plan)), 'kfac_inverse_plan_create')
    try:
        _lib.check(lib.kfac_inverse_plan_run(
            plan, 1e-2, 0, ctypes.c_void_p(info.data_ptr()),
            ctypes.c_void_p(diag.data_ptr()), ops._stream()), 'run')
        torch.cuda.synchronize()
    finally:
        lib.kfac_inverse_plan_destroy(plan)
    assert not info.any()
    return inv


def test_inverse_does_not_depend_on_where_its_workspace_begins(ops):
    rng = np.random.default_rng(8)
    F = [dev(spd(rng, d)) for d in (40, 130, 700, 1500)]
    want = _inverse_in(ops, F, 0)
    for offset in (4, 16, 252):
        for a, b in zip(_inverse_in(ops, F, offset), want):
            assert torch.equal(a, b)


def test_inverse_without_look_ahead(ops, monkeypatch):
    """The chain as one stream of launches, each waiting for the one before."""
    monkeypatch.setenv('KFAC_INVERSE_LOOKAHEAD', '0')
    rng = np.random.default_rng(9)
    host_f = [spd(rng, d) for d in (40, 130, 700, 1500)]
    for f, inv in zip(host_f, _inverse_in(ops, [dev(f) for f in host_f], 0)):
        want = np.linalg.inv(f.astype(np.float64) + 1e-2 * np.eye(len(f)))
        assert rel(host(inv), want) < INVERSE_TOL


# ------------------------------------------------------------- precondition
def precond_case(rng, dG, dW, bias):
    dA = dW + int(bias)
    Gi = spd(rng, dG)
    Ai = spd(rng, dA)
    gW = rng.standard_normal((dG, dW)).astype(np.float32)
    gb = rng.standard_normal(dG).astype(np.float32) if bias else None
    return Gi, Ai, gW, gb


@pytest.mark.parametrize('shapes', [
    [(128, 256, False), (64, 60, False)],            # 16-byte rows, few tiles
    [(33, 31, True), (129, 257, False), (5, 3, True)],   # none of them
    [(1024, 1152, False), (512, 1000, True), (260, 2048, False),
     (301, 785, True)],          # both: long layers, in chunks
])
def test_precondition_tile_variants(ops, shapes):
    """Narrow tiles and chunks, operands read as 16-byte words and float by
    float, cut rows, columns and contractions, the appended bias column."""
    rng = np.random.default_rng(31)
    cases = [precond_case(rng, *s) for s in shapes]
    Gi, Ai, gW = ([dev(c[k]) for c in cases] for k in range(3))
    gb = [None if c[3] is None else dev(c[3]) for c in cases]
    kW = [torch.empty_like(t) for t in gW]
    kb = [None if t is None else torch.empty_like(t) for t in gb]
    ops.precondition(Gi, Ai, gW, gb, kW, kb)
    for c, w, b in zip(cases, kW, kb):
        g = c[2].astype(np.float64)
        if c[3] is not None:
            g = np.concatenate([g, c[3].astype(np.float64)[:, None]], 1)
        ref = c[0].astype(np.float64) @ g @ c[1].astype(np.float64)
        got = host(w) if b is None else np.concatenate(
            [host(w), host(b)[:, None]], 1)
        assert rel(got, ref) < 2e-5     # TF32 pairs and fp32 sums: < 1e-5


@pytest.mark.parametrize('fused', [False, True])
def test_precondition_of_many_short_layers(ops, fused):
    """Layers that are all short, of whole 16-byte words and not, with more tiles
    than SMs: 256 columns a tile and a launch for each kind; kf alone and with the
    momentum update (to the roundings of its three operations)."""
    rng = np.random.default_rng(37)
    shapes = [(384, 384, False), (384, 380, False), (256, 512, False)] * 6 + \
        [(255, 255, False), (129, 96, True), (253, 257, False)] * 6
    cases = [precond_case(rng, *s) for s in shapes]
    Gi, Ai, gW = ([dev(c[k]) for c in cases] for k in range(3))
    gb = [None if c[3] is None else dev(c[3]) for c in cases]
    kW = [torch.empty_like(t) for t in gW]
    kb = [None if t is None else torch.empty_like(t) for t in gb]
    update = []
    if fused:
        pW, vW = ([dev(rng.standard_normal(c[2].shape).astype(np.float32))
                   for c in cases] for _ in range(2))
        pb, vb = ([None if t is None else torch.full_like(t, x) for t in gb]
                  for x in (1.0, 2.0))
        old = [(host(p), host(v)) for p, v in zip(pW, vW)]
        update = [pW, pb, vW, vb, 0.5, 0.9]
    ops.precondition(Gi, Ai, gW, gb, kW, kb, *update)
    for i, (c, w, b) in enumerate(zip(cases, kW, kb)):
        g, got = c[2].astype(np.float64), host(w)
        if b is not None:
            g = np.concatenate([g, c[3].astype(np.float64)[:, None]], 1)
            got = np.concatenate([got, host(b)[:, None]], 1)
        ref = c[0].astype(np.float64) @ g @ c[1].astype(np.float64)
        assert rel(got, ref) < 2e-5     # as above
        if not fused:
            continue
        parts = [(got[:, :c[2].shape[1]], *old[i], pW[i], vW[i])]
        if b is not None:
            parts.append((got[:, -1], 1.0, 2.0, pb[i], vb[i]))
        for kf, p, v, p_new, v_new in parts:
            v = 0.9 * v - 0.5 * kf.astype(np.float64)
            scale = np.abs(v).max()
            assert np.abs(host(v_new) - v).max() < 2.0 ** -22 * (scale + 4.0)
            assert np.abs(host(p_new) - p - v).max() < 2.0 ** -22 * (scale + 8.0)


@pytest.mark.parametrize('dG,dW,bias,offset,magnitude', [
    (512, 512, False, 0, 1.0), (33, 640, True, 0, 1e-18),
    (1, 1024, False, 0, 1e12), (640, 5, True, 1, 1.0),
    (300, 1023, True, 0, 1e12), (129, 897, False, 1, 1e-18),
    (257, 1000, False, 2, 1.0), (1025, 255, True, 3, 1e-18),
    (1, 2048, False, 0, 1e12)])
def test_precondition_of_long_layers(ops, dG, dW, bias, offset, magnitude):
    """Long enough for operands in chunks: cut tiles and k-blocks, the bias as an
    appended column, parameters at odd addresses, gradient rows of different
    sizes (dead units), with and without a copy of kf.  22-bit terms: 2^-21 per
    operand and sums of up to 1025 + 256 terms, 1e-5 in all."""
    rng = np.random.default_rng(dG * 7 + dW)
    Gi, Ai, gW, gb = precond_case(rng, dG, dW, bias)
    rows = (magnitude * 10.0 ** rng.integers(-4, 1, dG)).astype(np.float32)
    gW = gW * rows[:, None]
    gW[dG // 2] *= dG == 1
    gb = None if gb is None else gb * rows

    def place(a):      # `offset` floats behind a 16-byte boundary
        buf = torch.zeros(a.size + 4, device='cuda')
        t = buf[offset:offset + a.size].view(a.shape)
        t.copy_(dev(a))
        return t
    pW = rng.standard_normal(gW.shape).astype(np.float32)
    vW = (magnitude * rng.standard_normal(gW.shape)).astype(np.float32)
    bias_t = [None] * 3 if gb is None else [
        place(a) for a in (gb, np.ones_like(gb), np.zeros_like(gb))]
    g = gW.astype(np.float64)
    if gb is not None:
        g = np.concatenate([g, gb.astype(np.float64)[:, None]], 1)
    ref = Gi.astype(np.float64) @ g @ Ai.astype(np.float64)
    for kf in (place(np.zeros_like(gW)), None):
        kb = None if gb is None or kf is None else torch.empty_like(bias_t[0])
        w2, v2 = place(pW), place(vW)
        b2 = None if gb is None else bias_t[1].clone()
        vb2 = None if gb is None else bias_t[2].clone()
        ops.precondition([dev(Gi)], [dev(Ai)], [place(gW)], [bias_t[0]],
                         [kf], [kb], [w2], [b2], [v2], [vb2], lr=0.5,
                         momentum=0.9)
        if kf is not None:
            got = host(kf) if kb is None else np.concatenate(
                [host(kf), host(kb)[:, None]], 1)
            assert rel(got, ref) < 1e-5
        want = 0.9 * vW.astype(np.float64) - 0.5 * ref[:, :dW]
        assert rel(host(v2), want) < 1e-5
        assert rel(host(w2), pW + want) < 1e-5
        if gb is not None:
            assert rel(host(vb2), -0.5 * ref[:, dW]) < 1e-5
            assert rel(host(b2), 1.0 - 0.5 * ref[:, dW]) < 1e-5


def _precondition(ops, Gi, Ai, g, bias=False):
    """kf of one layer, and what fp64 gives for the same fp32 inputs; with
    `bias` the last column of `g` is the bias gradient."""
    Gi, Ai, g = (a.astype(np.float32) for a in (Gi, Ai, g))
    cols = g.shape[1] - int(bias)
    kW = torch.empty((g.shape[0], cols), device='cuda')
    kb = torch.empty(g.shape[0], device='cuda') if bias else None
    ops.precondition([dev(Gi)], [dev(Ai)], [dev(np.ascontiguousarray(
        g[:, :cols]))], [dev(np.ascontiguousarray(g[:, cols])) if bias else None],
        [kW], [kb])
    got = host(kW)
    if bias:
        got = np.concatenate([got, host(kb)[:, None]], 1)
    return got, Gi.astype(np.float64) @ g.astype(np.float64) @ \
        Ai.astype(np.float64).T


def _worst(got, ref, axis, terms=0.0):
    """Largest error of a row (axis 1) or column (axis 0), relative to it;
    with `terms`, the sums of the products' sizes, to a sixteenth of those at
    least (what cancels in a sum is not lost by its error)."""
    norm = np.linalg.norm(np.maximum(np.abs(ref), terms / 16), axis=axis)
    err = np.linalg.norm(got - ref, axis=axis)
    assert not err[norm == 0].any()
    return (err[norm > 0] / norm[norm > 0]).max()


def _inverse_of(rng, d, scale, damping):
    x = rng.standard_normal((2 * d, d)) * scale
    return np.linalg.inv(x.T @ x / (2 * d) + damping * np.eye(d))


@pytest.mark.parametrize('dG,dW,bias', [(64, 1600, False), (300, 785, True),
                                        (513, 511, False)])
@pytest.mark.parametrize('small', [1e-4, 1e-8, 1e-12, 1e-30])
def test_precondition_of_rows_of_any_scale(ops, dG, dW, bias, small):
    """Every row of kf to 1e-5 of itself, however small its gradient is beside
    the other rows': half of the rows, all but one, rows spread evenly; G_inv
    nearly diagonal, so that a row of kf is as small as its gradient, and as the
    damped factor of such rows.  22-bit terms (2^-21 per operand) and sums of up
    to 1600 + 64 terms, cut off towards zero: 1e-5."""
    rng = np.random.default_rng(dG + dW)
    dA = dW + int(bias)
    Ai = _inverse_of(rng, dA, 1.0, 1e-2)
    near = np.diag(rng.random(dG) + 0.5) + \
        small * 0.1 * rng.standard_normal((dG, dG))
    base = rng.standard_normal((dG, dA))
    half = np.where(np.arange(dG) % 2, small, 1.0)
    for rows in (half, np.where(np.arange(dG) == 7, 1.0, small),
                 small ** rng.random(dG)):
        got, ref = _precondition(ops, near, Ai, base * rows[:, None], bias)
        assert _worst(got, ref, 1) < 1e-5
    got, ref = _precondition(ops, _inverse_of(rng, dG, half, small ** 2), Ai,
                             base * half[:, None], bias) \
        if small > 1e-10 else (ref, ref)
    assert _worst(got, ref, 1) < 1e-5


@pytest.mark.parametrize('dG,dW,bias', [(64, 1600, False), (300, 785, True),
                                        (513, 511, False)])
@pytest.mark.parametrize('small', [1e-4, 1e-8, 1e-12])
def test_precondition_of_features_of_any_scale(ops, dG, dW, bias, small):
    """Every row and column of kf to 1e-5 of itself with input features of
    different scales, A_inv that of such features with a damping below the
    smallest or between the two kinds (features that are nearly always zero), some
    features exactly zero, and with rows of different scales besides.  A single
    large entry takes nothing from the other rows.  Bound: as for rows."""
    rng = np.random.default_rng(dG + dW + 1)
    dA = dW + int(bias)
    Gi = _inverse_of(rng, dG, 1.0, 1e-2)
    base = rng.standard_normal((dG, dA))
    half = np.where(np.arange(dA) % 2, small, 1.0)
    half[dA // 3] = 0.0
    spread = small ** rng.random(dA)
    rows = small ** rng.random(dG)
    near = np.diag(rng.random(dG) + 0.5) + \
        small * 0.1 * rng.standard_normal((dG, dG))
    for f, damping in ((half, 1e-3), (spread, 1e-3), (spread, small ** 2)):
        Ai = _inverse_of(rng, dA, f, damping)
        for G, g in ((Gi, base * f), (near, base * f * rows[:, None])):
            got, ref = _precondition(ops, G, Ai, g, bias)
            terms = np.abs(G) @ np.abs(g) @ np.abs(Ai)
            assert _worst(got, ref, 1, terms) < 1e-5
            assert _worst(got, ref, 0, terms) < 1e-5
    g = base.copy()
    g[5, 3] = 1 / small
    got, ref = _precondition(ops, near, _inverse_of(rng, dA, 1.0, 1e-2), g, bias)
    assert _worst(got, ref, 1) < 1e-5


def test_precondition_of_long_layers_under_capture(ops, engine):
    """The launches of a preconditioning in chunks begin before the one in front
    has ended; captured and replayed on other gradients, call after call on one
    workspace, they give what calls by themselves do."""
    if engine == 0:
        pytest.skip('chunks belong to the tensor-core engine')
    rng = np.random.default_rng(41)
    cases = [precond_case(rng, 512, 512, False), precond_case(rng, 300, 785, True)]
    Gi, Ai, gW = ([dev(c[k]) for c in cases] for k in range(3))
    gb = [None if c[3] is None else dev(c[3]) for c in cases]
    kW = [torch.empty_like(t) for t in gW]
    kb = [None if t is None else torch.empty_like(t) for t in gb]

    def call():
        ops.precondition(Gi, Ai, gW, gb, kW, kb)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        call()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            for _ in range(3):
                call()
        for scale in (1.0, 1e-6, 1e6):
            for t in gW:
                t.mul_(scale)
            call()
            want = [t.clone() for t in kW + kb if t is not None]
            for t in kW:
                t.zero_()
            graph.replay()
            for a, b in zip([t for t in kW + kb if t is not None], want):
                assert torch.equal(a, b)
    torch.cuda.synchronize()


@pytest.mark.parametrize('value', [float('inf'), float('nan')])
def test_precondition_of_a_non_finite_gradient_is_not_finite(ops, value):
    rng = np.random.default_rng(3)
    Gi, Ai, gW, _ = precond_case(rng, 130, 1030, False)
    gW[17, 1000] = value
    kf = torch.zeros(gW.shape, device='cuda')
    ops.precondition([dev(Gi)], [dev(Ai)], [dev(gW)], [None], [kf], [None])
    assert not np.isfinite(host(kf)).any()


@pytest.mark.parametrize('d', [1, 31, 127, 129, 257, 385, 513, 770, 1025])
def test_inverse_around_block_sizes(ops, d):
    """Sides around the diagonal block, the panel and the row pitch."""
    run_pairs(ops, [d], [max(1, d // 3)], 1e-3, seed=d)


@pytest.mark.parametrize('dims', [[129], [300, 10, 257], [640, 1100, 96],
                                  [520] * 20])
def test_inverse_by_graph_and_by_plain_launches(ops, engine, monkeypatch, dims):
    """The same launches in the same order: bit for bit, three runs over inputs
    that change (the graph's kernels begin before the ones in front have ended)."""
    rng = np.random.default_rng(len(dims))
    F = [torch.empty((d, d), device='cuda') for d in dims]
    plans, outs = [], []
    for graph in ('1', '0'):
        monkeypatch.setenv('KFAC_INVERSE_GRAPH', graph)
        outs.append([torch.empty_like(f) for f in F])
        plans.append(ops.InversePlan(F, outs[-1], [-1] * len(dims),
                                     [2] * len(dims), scale=[1.0] * len(dims)))
    for _ in range(3):
        for f in F:
            x = dev(rng.standard_normal((f.shape[0] + 50, f.shape[0])))
            f.copy_(x.t() @ x / len(x))
            f.copy_((f + f.t()) / 2)
        for plan in plans:
            plan.run(1e-2)
        # (what they were: a diagonal kernel and a solve per block but the first;
        # nothing begins early on the other engine)
        assert plans[0].early_launches() >= 2 * ((max(dims) - 1) // 128) * engine
        assert plans[1].early_launches() == -1
        torch.cuda.synchronize()
        for a, b in zip(*outs):
            assert torch.isfinite(a).all() and torch.equal(a, b)
    for plan in plans:
        plan.close()


@pytest.mark.parametrize('dims', [[513, 512, 30], [641, 640, 513], [1153, 700, 300],
                                  [1537, 1025, 512], [2305, 1664, 129]])
def test_inverse_windows_behind_a_panel(ops, dims):
    """The updates of the columns behind a panel of 512, in two parts: windows of
    one row and more, and matrices that end before, at and behind the panel."""
    run_pairs(ops, dims, [max(1, d // 5) for d in dims], 1e-3, seed=dims[0])


def test_inverses_repeat_bit_for_bit_beside_each_other(ops, engine):
    """Sums are in a fixed order, so nothing changes from run to run, also where
    three plans fill the SMs and warps of a block wait for each other longer (a
    warp's columns of a diagonal sub-block were touched by another one too soon in
    one of ten runs of such a set)."""
    from bench_workloads import layer_dims, resnet50_layers
    dims = [d for l in resnet50_layers() for d in layer_dims(l)[:2]]
    g = torch.Generator(device='cuda')
    g.manual_seed(5)
    F = []
    for d in dims:
        x = torch.randn((2 * d, d), device='cuda', generator=g)
        f = x.t() @ x / (2 * d)
        F.append((f + f.t()) / 2)
    inv = [torch.empty_like(f) for f in F]
    plan = ops.InversePlanSet(F, inv, [i ^ 1 for i in range(len(F))],
                              [0, 1] * (len(F) // 2))
    plan.run(1e-3)
    first = [v.clone() for v in inv]
    for _ in range(100):
        plan.run(1e-3)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(first, inv))
        for p in plan.plans:
            assert p.early_launches() > 0 if engine else p.early_launches() == 0


@pytest.mark.parametrize('blocks', [0, 1, 4])
@pytest.mark.parametrize('rows', [1, 31, 32, 33, 64, 65, 95, 96, 97, 127, 128])
def test_inverse_sub_blocks_of_the_diagonal_kernel(ops, blocks, rows):
    """A last diagonal block of `rows` rows, on its own and behind others: its
    sub-blocks of 32 columns and their remainders, with and without the update of
    the block before it.  Error of entry (i, j) against sqrt(inv_ii inv_jj), which
    a Cholesky factorisation bounds by the condition of the scaled factor (here at
    most 35) times the rounding of sums of at most d terms, d 2^-24."""
    d = 128 * blocks + rows
    rng = np.random.default_rng(d)
    x = rng.standard_normal((2 * d + 64, d)) * np.exp(rng.uniform(-3, 3, d))
    f = (x.T @ x / len(x)).astype(np.float32)
    f = (f + f.T) / 2
    F = [dev(f)] * 3
    inv = [torch.empty_like(F[0]) for _ in F]
    plan = ops.InversePlan(F, inv, [-1] * 3, [2] * 3, scale=[1.0] * 3)
    plan.set_refine(0)
    plan.run(1e-7)
    torch.cuda.synchronize()
    assert host(plan.info).tolist() == [0] * 3
    truth = np.linalg.inv(f.astype(np.float64) + 1e-7 * np.eye(d))
    s = np.sqrt(np.diag(truth))
    for i in inv:
        got = host(i)
        assert np.array_equal(got, got.T)
        assert (np.abs(got - truth) / s[:, None] / s[None, :]).max() < \
            35 * d * 2.0 ** -24
    assert torch.equal(inv[0], inv[2])
    plan.close()


def _multiply_adds(W):
    """X = L^-1 of a Cholesky factor, a column of [W; I] at a time in fp32, every
    product added with one rounding."""
    f32, n = np.float32, len(W)
    M = np.tril(W)
    for j in range(n):
        r = f32(1) / np.sqrt(M[j, j])
        col = M[:, j] * r
        col[j] = r
        # (a product of two fp32 numbers is exact in fp64)
        to = (M - np.outer(col.astype(np.float64), col)).astype(f32)
        for i in range(n):
            end = n if i <= j else i + 1
            M[i, j + 1:end] = to[i, j + 1:end]
        M[:j + 1, j] = col[:j + 1]
    return np.triu(M).T


@pytest.mark.parametrize('d', [1, 2, 31, 33, 100, 128])
def test_yardstick_engine_eliminates_in_fp32(ops, engine, d):
    """Engine 0 is what the tensor-core engine is measured against: its diagonal
    blocks are multiply-adds in fp32 to the bit, none of the other's terms."""
    if engine == 1:
        pytest.skip('the tensor-core engine eliminates in bf16 terms')
    rng = np.random.default_rng(d)
    f = spd(rng, d)
    F = dev(f)
    plan = ops.InversePlan([F], [torch.empty_like(F)], [-1], [2])
    plan.run(1e-3)
    W = f.copy()
    W[np.arange(d), np.arange(d)] += host(plan.diag)[0]
    # the workspace: W, V and X, rows of a multiple of 32, from 256 bytes on
    pitch = (d + 31) // 32 * 32
    each = (4 * d * pitch + 255) // 256 * 256
    at = -plan.workspace.data_ptr() % 256 + 2 * each
    X = host(plan.workspace)[at:at + 4 * d * pitch].view(np.float32)
    assert np.array_equal(X.reshape(d, pitch)[:, :d], _multiply_adds(W))
    plan.close()


def test_precondition_matches_oracle(ops):
    rng = np.random.default_rng(11)
    shapes = [(10, 1000, True), (64, 147, True), (300, 129, False),
              (1000, 784, True), (7, 5, False), (256, 2304, False)]
    cases = [precond_case(rng, *s) for s in shapes]
    Gi = [dev(c[0]) for c in cases]
    Ai = [dev(c[1]) for c in cases]
    gW = [dev(c[2]) for c in cases]
    gb = [None if c[3] is None else dev(c[3]) for c in cases]
    kW = [torch.empty_like(t) for t in gW]
    kb = [None if t is None else torch.empty_like(t) for t in gb]
    ops.precondition(Gi, Ai, gW, gb, kW, kb)
    for c, w, b in zip(cases, kW, kb):
        wantW, wantb = orc.connection_kfgrads(c[1], c[0], c[2], c[3])
        assert rel(host(w), wantW) < KFGRAD_TOL
        if b is not None:
            assert rel(host(b), wantb) < KFGRAD_TOL


def test_precondition_conv_shape_and_fused_update(ops):
    rng = np.random.default_rng(12)
    Gi, Ai, gW2, gb = precond_case(rng, 20, 3 * 3 * 6, True)
    gW = gW2.reshape(20, 6, 3, 3)
    W = rng.standard_normal(gW.shape).astype(np.float32)
    b = rng.standard_normal(20).astype(np.float32)
    vW = rng.standard_normal(gW.shape).astype(np.float32)
    vb = rng.standard_normal(20).astype(np.float32)
    dW_, db_, dvW, dvb = dev(W), dev(b), dev(vW), dev(vb)
    kW, kb = torch.empty_like(dW_), torch.empty_like(db_)
    ops.precondition([dev(Gi)], [dev(Ai)], [dev(gW)], [dev(gb)], [kW], [kb],
                     [dW_], [db_], [dvW], [dvb], lr=0.05, momentum=0.9)
    wantW, wantb = orc.connection_kfgrads(Ai, Gi, gW, gb)
    assert rel(host(kW), wantW) < KFGRAD_TOL
    assert rel(host(kb), wantb) < KFGRAD_TOL
    orc.momentum_update(W, vW, wantW, 0.05, 0.9)
    orc.momentum_update(b, vb, wantb, 0.05, 0.9)
    assert rel(host(dW_), W) < 1e-5
    assert rel(host(db_), b) < 1e-5
    assert rel(host(dvW), vW) < KFGRAD_TOL


def test_momentum_update_and_axpby(ops):
    rng = np.random.default_rng(13)
    p = rng.standard_normal(100003).astype(np.float32)
    v = rng.standard_normal(100003).astype(np.float32)
    g = rng.standard_normal(100003).astype(np.float32)
    dp, dv = dev(p), dev(v)
    ops.momentum_update(dev(g), dp, dv, 0.01, 0.9)
    orc.momentum_update(p, v, g, 0.01, 0.9)
    assert rel(host(dp), p) < 1e-6 and rel(host(dv), v) < 1e-6
    y = dev(g)
    ops.axpby(0.25, dev(p), 0.75, y, y)
    assert rel(host(y), 0.25 * p + 0.75 * g) < 1e-6


@pytest.mark.parametrize('shape', [
    (4, 5), (33, 10), (7, 3, 1, 1), (3, 5, 7, 7), (8, 64, 8, 8),
    (5, 33, 9, 11), (2, 129, 3, 2), (3, 8, 66, 63), (3, 20, 66, 63),
    (2, 6, 112, 112), (1, 4, 64, 65)])
@pytest.mark.parametrize('channels_last', [False, True])
@pytest.mark.parametrize('mean', [0.0, 30.0])
def test_bn_sample_grads_layouts(ops, shape, channels_last, mean):
    """Planes read by a part of a warp, a warp or a block, channels-last rows
    with and without 16-byte words, partial channel groups, against fp64; the
    mean of x may be many times its spread."""
    torch.manual_seed(1)
    x = torch.randn(shape, device='cuda') + mean
    gy = torch.randn(shape, device='cuda')
    if channels_last and len(shape) == 4:
        x = x.contiguous(memory_format=torch.channels_last)
        gy = gy.contiguous(memory_format=torch.channels_last)
    out = ops.bn_sample_grads(x, gy, 1e-5, 2.0)
    xd, gd = x.double(), gy.double() * 2.0
    batch = [0] + list(range(2, xd.dim()))
    xh = (xd - xd.mean(batch, keepdim=True)) / torch.sqrt(
        xd.var(batch, unbiased=False, keepdim=True) + 1e-5)
    ref = torch.cat([(gd * xh).flatten(2).sum(2) if xd.dim() > 2 else gd * xh,
                     gd.flatten(2).sum(2) if xd.dim() > 2 else gd], 1)
    # as for fp32 sums of up to hw terms, each rounded: sqrt(hw) 2^-24 relative
    # to the terms, of the order of the sums themselves for random signs, times
    # the distance of a shift from the mean in units of the spread (< 5); what
    # the double sums leave is bounded in test_bn_sample_grads_with_outliers
    hw = 1
    for v in shape[2:]:
        hw *= v
    assert rel(host(out), host(ref)) < 5 * 6e-8 * max(4.0, hw ** 0.5)


def test_bn_sample_grads_of_mixed_layouts_in_one_group(ops):
    """Layers of both layouts, in any order, in one grouped call give what each
    gives alone, bit for bit."""
    torch.manual_seed(11)
    pairs = []
    for k, shape in enumerate([(4, 16, 9, 9), (4, 5), (3, 7, 5, 6), (4, 32, 8, 8),
                               (2, 70, 66, 63), (4, 64, 1, 1), (6, 12, 7, 7)]):
        x, gy = torch.randn(shape, device='cuda'), torch.randn(shape,
                                                               device='cuda')
        if len(shape) == 4 and k % 3 == 0:
            x = x.contiguous(memory_format=torch.channels_last)
            gy = gy.contiguous(memory_format=torch.channels_last)
        pairs.append((x, gy))
    alone = [ops.bn_sample_grads(x, gy, 1e-5, 2.0) for x, gy in pairs]
    for order in (range(7), range(6, -1, -1), (0, 3, 6), (1, 2)):
        items = [ops.bn_item(*pairs[i], 1e-5, 2.0) for i in order]
        ops.bn_sample_grads_group(items)
        for i, it in zip(order, items):
            assert torch.equal(it.result, alone[i])


@pytest.mark.parametrize('shape', [
    (33, 10), (8, 64, 8, 8), (5, 33, 9, 11), (32, 8, 56, 56)])
@pytest.mark.parametrize('channels_last', [False, True])
@pytest.mark.parametrize('where', ['first', 'corners', 'sample'])
def test_bn_sample_grads_with_outliers(ops, shape, channels_last, where):
    """The first value of every channel, the corner of every image or a whole
    sample far outside the rest: no digits are lost to it."""
    torch.manual_seed(6)
    x = 3.0 + 1e-3 * torch.randn(shape, device='cuda')
    gy = torch.randn(shape, device='cuda')
    at = {'first': (slice(0, 1), slice(None), 0, 0),
          'corners': (slice(None), slice(None), 0, 0),
          'sample': (slice(0, 1),)}[where]
    x[at[:x.dim()]] += 5.0
    if channels_last and len(shape) == 4:
        x = x.contiguous(memory_format=torch.channels_last)
        gy = gy.contiguous(memory_format=torch.channels_last)
    out = ops.bn_sample_grads(x, gy, 1e-5, 2.0)
    xd, gd = x.double(), gy.double() * 2.0
    batch = [0] + list(range(2, xd.dim()))
    xh = (xd - xd.mean(batch, keepdim=True)) / torch.sqrt(
        xd.var(batch, unbiased=False, keepdim=True) + 1e-5)
    ref = torch.cat([(gd * xh).flatten(2).sum(2) if xd.dim() > 2 else gd * xh,
                     gd.flatten(2).sum(2) if xd.dim() > 2 else gd], 1)
    # every rounding is 2^-24 of a term: of the two terms of sum g xhat (the
    # sample's own part and its mean's distance from the batch's, at most
    # sqrt(n) spreads, times sum g), of their sum and of the factors
    n, c = shape[0], shape[1]
    assert rel(host(out[:, c:]), host(ref[:, c:])) < 4 * 2.0 ** -24
    off = (xh.flatten(2).mean(2) if xd.dim() > 2 else xh) * ref[:, c:]
    size = (off.norm() + (ref[:, :c] - off).norm() + ref[:, :c].norm()).item()
    err = (out[:, :c].double() - ref[:, :c]).norm().item()
    assert err < 4 * 2.0 ** -24 * size


def test_bn_kfgrad(ops, golden):
    g = golden('bn_4d')
    c = g['g_gamma'].shape[0]
    y0 = torch.empty(c, device='cuda')
    y1 = torch.empty(c, device='cuda')
    flag = torch.zeros(2, dtype=torch.int32, device='cuda')
    ops.symv_split(dev(g['F_inv']), dev(g['g_gamma']), dev(g['g_beta']), y0, y1,
                   flag)
    assert rel(host(y0), g['kf_gamma']) < KFGRAD_TOL
    assert rel(host(y1), g['kf_beta']) < KFGRAD_TOL
    assert flag.tolist() == [0, 0]
    # a NaN anywhere in the product: the raw gradients come back instead
    # (the reference's _check_nan fallback), the counter goes up, and the
    # next clean call is unaffected
    bad = g['F_inv'].copy()
    bad[2, 3] = np.nan
    ops.symv_split(dev(bad), dev(g['g_gamma']), dev(g['g_beta']), y0, y1, flag)
    assert flag.tolist() == [0, 1]
    assert np.array_equal(host(y0), g['g_gamma'])
    assert np.array_equal(host(y1), g['g_beta'])
    ops.symv_split(dev(g['F_inv']), dev(g['g_gamma']), dev(g['g_beta']), y0, y1,
                   flag)
    assert flag.tolist() == [0, 1]
    assert rel(host(y0), g['kf_gamma']) < KFGRAD_TOL


def test_bn_lowrank_form_matches_dense_oracle(ops):
    """The low-rank form of a BatchNormalization block -- (D + sum_s w_s
    U_s^T U_s)^-1 g through the m x m matrix I + Hs Hs^T -- against the dense
    path of the oracle: running average of three steps' factors (decay 0.9),
    separate damping of the gamma and beta halves, damped inverse, product
    with the gradient."""
    rng = np.random.default_rng(31)
    n, c, steps, r = 8, 20, 3, 0.9
    d_gamma, d_beta = 16.0 * 1e-3, 16.0 * 5e-3
    Us = [(rng.standard_normal((n, 2 * c)) * 0.3).astype(np.float32)
          for _ in range(steps)]
    # oracle: F_t = r U^T U / n + (1 - r) F_{t-1}, first step plain
    F = None
    for U in Us:
        cov = (U.T @ U / n).astype(np.float32)
        F = cov if F is None else orc.update_cov_ema(cov, F, r)
    add = np.concatenate([np.full(c, d_gamma), np.full(c, d_beta)])
    Finv = np.linalg.inv(F.astype(np.float64) + np.diag(add))
    gg = rng.standard_normal(c).astype(np.float32)
    gb = rng.standard_normal(c).astype(np.float32)
    want = Finv @ np.concatenate([gg, gb])
    # weights of the slots, oldest first: (1-r)^2, r(1-r), r; each over n
    w = [(1 - r) ** 2 / n, r * (1 - r) / n, r / n, 0.0]    # one unused slot
    hist = dev(np.concatenate(Us + [np.full((n, 2 * c), 7.0, np.float32)]))
    m = 4 * n
    Hs = torch.empty_like(hist)
    M0 = torch.empty((m, m), device='cuda')
    Minv = torch.empty_like(M0)
    kg, kb = torch.empty(c, device='cuda'), torch.empty(c, device='cuda')
    flag = torch.zeros(2, dtype=torch.int32, device='cuda')
    item = ops.bn_lowrank_item(hist, Hs, c, n, w, d_gamma, d_beta, Minv,
                               dev(gg), dev(gb), kg, kb, flag)
    ops.bn_lowrank_scale([item])
    ops.factor_group([ops.dense_t_item(Hs, 1.0, 0.0, M0)], M0.device)
    plan = ops.InversePlan([M0], [Minv], [-1], [2], scale=[1.0])
    plan.run(1.0, use_pi=False)
    ops.bn_lowrank_apply([item])
    got = np.concatenate([host(kg), host(kb)])
    assert rel(got, want) < KFGRAD_TOL
    assert rel(got, want) < 1e-4        # and in fact far inside it
    assert flag.tolist() == [0, 0]
    # the unused slot contributes nothing: its rows are zero in Hs
    assert float(Hs[3 * n:].abs().max()) == 0.0
    plan.close()


# -------------------------------------------------------------- wire format
@pytest.mark.parametrize('n,c,h,k,s,p,bias', [
    (2, 40, 9, 1, 1, 0, True),      # its own patch matrix: read in place
    (2, 64, 14, 3, 1, 1, False),    # staged as zero-bordered NCHW planes
    (2, 24, 10, 1, 2, 0, False),    # staged without a border
    (2, 3, 32, 7, 2, 3, True),      # few channels, bias column
    (3, 40, 9, 3, 1, 1, True)])     # sizes that are no multiples of 32
def test_factor_conv_channels_last(ops, n, c, h, k, s, p, bias):
    """Channels-last activations and gradients give the factors of the same
    logical NCHW tensors."""
    rng = np.random.default_rng(7 * n + c + h + k)
    x = np.maximum(rng.standard_normal((n, c, h, h)), 0).astype(np.float32)
    want = orc.conv_A(x.astype(np.float64), k, s, p, bias)
    xd = dev(x).contiguous(memory_format=torch.channels_last)
    got = host(ops.factor_conv_input(xd, k, s, p, bias, alpha=1.0 / n))
    assert rel(got, want) < FACTOR_TOL
    out = torch.empty_like(dev(got))
    ops.factor_group([ops.conv_input_item(xd, k, s, p, bias, 1.0 / n, 0.0,
                                          out)], out.device)
    assert rel(host(out), want) < FACTOR_TOL
    gy = (rng.standard_normal((n, c, h, h)) / n).astype(np.float32)
    wantg = orc.conv_G(gy.astype(np.float64))
    gd = dev(gy).contiguous(memory_format=torch.channels_last)
    gotg = host(ops.factor_conv_grad(gd, alpha=n / float(h * h)))
    assert rel(gotg, wantg) < FACTOR_TOL
    outg = torch.empty_like(dev(gotg))
    ops.factor_group([ops.conv_grad_item(gd, n / float(h * h), 0.0, outg)],
                     outg.device)
    assert rel(host(outg), wantg) < FACTOR_TOL


def test_axpby_group_matches_single_calls(ops):
    rng = np.random.default_rng(77)
    shapes = [(3, 3), (8192,), (100, 130), (1,), (8193, 2)]
    xs = [dev(rng.standard_normal(s).astype(np.float32)) for s in shapes]
    ys = [dev(rng.standard_normal(s).astype(np.float32)) for s in shapes]
    want = [ops.axpby(0.9, x, 0.1, y, torch.empty_like(y))
            for x, y in zip(xs, ys)]
    outs = [y.clone() for y in ys]
    ops.axpby_group(0.9, xs, 0.1, outs, outs)        # in place on y
    for o, w in zip(outs, want):
        assert torch.equal(o, w)
    outs = [torch.full_like(y, 7.0) for y in ys]
    ops.axpby_group(1.0, xs, 0.0, ys, outs)          # plain copy
    for o, x in zip(outs, xs):
        assert torch.equal(o, x)


def test_wire_pack_unpack_bit_exact(ops):
    rng = np.random.default_rng(14)
    shapes = [((37, 37), True), ((11,), False), ((1, 1), True),
              ((300, 300), True), ((4, 9), False)]
    arrs = []
    for shp, tri in shapes:
        a = rng.standard_normal(shp).astype(np.float32)
        if tri:
            a = (a + a.T).astype(np.float32)
        arrs.append(a)
    tri = [t for _, t in shapes]
    d_arrs = [dev(a) for a in arrs]
    n = ops.wire_nelems(d_arrs, tri)
    nested = [[(a, t) for a, t in zip(arrs, tri)]]
    assert n == orc.wire_nelems(nested)
    wire = torch.full((n,), 7.0, device='cuda')
    ops.wire_pack(d_arrs, tri, wire)
    assert np.array_equal(host(wire), orc.pack_arrays(nested))
    # selective pack with zero fill (all-gather send side)
    sel = [1, 0, 1, 0, 1]
    ops.wire_pack(d_arrs, tri, wire, select=sel, zero_skipped=True)
    want = orc.pack_arrays(nested)
    off = 0
    for a, t, s in zip(arrs, tri, sel):
        m = a.shape[0] * (a.shape[0] + 1) // 2 if t else a.size
        if not s:
            want[off:off + m] = 0
        off += m
    assert np.array_equal(host(wire), want)
    # unpack with mean scaling mirrors the triangles
    ops.wire_pack(d_arrs, tri, wire)
    outs = [torch.zeros_like(t) for t in d_arrs]
    ops.wire_unpack(outs, tri, wire, scale=0.25)
    for a, o in zip(arrs, outs):
        assert np.array_equal(host(o), a * np.float32(0.25))
    # fused running average on unpack
    prev = [dev(np.ones_like(a)) for a in arrs]
    ops.wire_unpack(prev, tri, wire, scale=1.0, ema_r=0.5)
    for a, o in zip(arrs, prev):
        assert rel(host(o), 0.5 * a + 0.5) < 1e-6


@pytest.mark.parametrize('skew', [0, 1, 3])
@pytest.mark.parametrize('wdt', [torch.float32, torch.float16,
                                 torch.bfloat16])
def test_wire_pack_runs(ops, wdt, skew):
    """Runs of 8192 wire elements written by whole lines: triangles and
    plain arrays shorter than a line, one run long give or take an element,
    and several runs long, from wires that start inside a line.  Exact."""
    sizes = [(127, True), (1, True), (128, True), (2, True), (3, True),
             (130, True), (8191, False), (8192, False), (8193, False),
             (5, False), (257, True), (20001, False)]
    g = torch.Generator(device='cuda').manual_seed(3)
    arrs = [torch.randn((n, n) if t else (n,), generator=g, device='cuda')
            for n, t in sizes]
    tri = [t for _, t in sizes]
    select = [i % 5 != 4 for i in range(len(sizes))]
    n = ops.wire_nelems(arrs, tri)
    parts = []
    for a, t, s in zip(arrs, tri, select):
        m = a.shape[0]
        w = a[tuple(torch.tril_indices(m, m, device='cuda'))] if t else a
        parts.append(w if s else torch.zeros_like(w))
    buf = torch.full((n + skew + 1,), 7.0, device='cuda', dtype=wdt)
    ops.wire_pack(arrs, tri, buf[skew:skew + n], select=select,
                  zero_skipped=True)
    assert torch.equal(buf[skew:skew + n], torch.cat(parts).to(wdt))
    assert (buf[:skew] == 7).all() and (buf[skew + n:] == 7).all()


@pytest.mark.parametrize('wdt', [torch.float16, torch.bfloat16])
def test_wire_reduced_precision(ops, wdt):
    """A 16-bit wire buffer holds each value rounded to the wire type (the
    cast of pure_nccl_communicator.py:354-375); the sum over several wire
    buffers is formed in fp32 from the widened values (:438-461)."""
    rng = np.random.default_rng(15)
    shapes = [((70, 70), True), ((1000,), False), ((129, 129), True)]
    arrs = []
    for shp, tri in shapes:
        a = rng.standard_normal(shp).astype(np.float32)
        arrs.append((a + a.T).astype(np.float32) if tri else a)
    tri = [t for _, t in shapes]
    nested = [[(a, t) for a, t in zip(arrs, tri)]]
    n = orc.wire_nelems(nested)
    ranks = 3
    wires, want = [], np.zeros(n, np.float32)
    for r in range(ranks):
        scaled = [dev(a * np.float32(r + 1)) for a in arrs]
        w = torch.zeros(n, dtype=wdt, device='cuda')
        ops.wire_pack(scaled, tri, w)
        exp = torch.from_numpy(orc.pack_arrays(
            [[(a * np.float32(r + 1), t) for a, t in zip(arrs, tri)]])).to(wdt)
        assert torch.equal(w.cpu(), exp)          # rounded to nearest
        want += exp.float().numpy()
        wires.append(w)
    outs = [torch.zeros_like(dev(a)) for a in arrs]
    ops.wire_unpack_sum(outs, tri, [w.data_ptr() for w in wires],
                        scale=1.0 / ranks, wire_dtype=wdt)
    ref = [np.zeros_like(a) for a in arrs]
    orc.unpack_arrays([[(a, t) for a, t in zip(ref, tri)]], want,
                      divisor=float(ranks))
    for o, a in zip(outs, ref):
        assert rel(host(o), a) < 1e-6
        if a.ndim == 2:
            assert np.array_equal(host(o), host(o).T)


def test_wire_unpack_sum_of_rank_buffers(ops):
    """The owner's side of the peer-memory reduce-scatter: the same slot of
    several wire buffers (one per rank; here all on this GPU) summed in rank
    order, scaled to the mean and mirrored.  Sizes straddle the 64-wide tiles
    and the 8192-element runs; unselected arrays must stay untouched and must
    not shift the offsets of the others."""
    rng = np.random.default_rng(41)
    shapes = [((130, 130), True), ((8192 + 77,), False), ((64, 64), True),
              ((5, 7), False), ((513, 513), True), ((0,), False),
              ((65, 65), True)]
    tri = [t for _, t in shapes]
    ranks = 5
    per_rank, wires = [], []
    for q in range(ranks):
        arrs = []
        for shp, t in shapes:
            a = rng.standard_normal(shp).astype(np.float32)
            if t:
                a = (a + a.T).astype(np.float32)
            arrs.append(a)
        per_rank.append(arrs)
        d = [dev(a) for a in arrs]
        w = torch.empty(ops.wire_nelems(d, tri), device='cuda')
        ops.wire_pack(d, tri, w)
        assert np.array_equal(
            host(w), orc.pack_arrays([[(a, t) for a, t in zip(arrs, tri)]]))
        wires.append(w)
    sel = [1, 1, 0, 1, 1, 1, 1]
    outs = [torch.full(shp, 3.0, device='cuda') for shp, _ in shapes]
    ops.wire_unpack_sum(outs, tri, [w.data_ptr() for w in wires], select=sel,
                        scale=1.0 / ranks)
    for i, (o, s) in enumerate(zip(outs, sel)):
        if not s:
            assert np.array_equal(host(o), np.full(shapes[i][0], 3.0, np.float32))
            continue
        acc = np.zeros(shapes[i][0], np.float32)
        for q in range(ranks):         # rank order, fp32, as the kernel sums
            acc = acc + per_rank[q][i]
        want = acc * np.float32(1.0 / ranks)
        assert np.array_equal(host(o), want), i
        if tri[i]:
            assert np.array_equal(host(o), host(o).T)
    with pytest.raises(Exception):
        ops.wire_unpack_sum(outs, tri, [wires[0].data_ptr()] * 17)


# ------------------------------------------- full-size, size-independent checks
def test_config4_full_size_inverse_property(ops, engine):
    """The isolated curvature microbench at its full sizes: factors with the
    dimensions of every ResNet-50 layer, each X^T X / m + 1e-3 I with m = 8192
    rows of N(0,1), built by the factor kernel, inverted in one batch (three
    streams by size class).  Checked through inv * F ~ I, which needs no CPU
    inverse of a 4608 x 4608 matrix."""
    if engine == 0:
        pytest.skip('full-size sweep runs on the tensor-core engine only')
    dims = sorted({d for l in bw.resnet50_layers()
                   for d in bw.layer_dims(l)[:2]})
    g = torch.Generator(device='cuda')
    g.manual_seed(4)
    m = 8192
    F = []
    for d in dims:
        X = torch.randn((m, d), device='cuda', generator=g)
        eye = torch.eye(d, device='cuda') * 1e-3
        F.append(ops.factor_dense(X, False, alpha=1.0 / m, beta=1.0, out=eye))
        del X
    inv = [torch.empty_like(f) for f in F]
    plan = ops.InversePlanSet(F, inv, [-1] * len(F), [2] * len(F),
                              scale=[0.0] * len(F))
    plan.run(0.0)
    torch.cuda.synchronize()
    assert int(plan.info.abs().sum()) == 0
    for d, f, i in zip(dims, F, inv):
        resid = (i.double() @ f.double() -
                 torch.eye(d, device='cuda', dtype=torch.float64))
        err = float(resid.norm() / d ** 0.5)
        assert err < INVERSE_TOL, (d, err)
        assert torch.equal(i, i.T)
    plan.close()


def test_config1_mlp_shapes_step(ops):
    """One K-FAC pass at the MNIST-MLP shapes (784-1000-1000-10, batch 128,
    damping 1e-3) against the oracle, all three layers in grouped calls."""
    rng = np.random.default_rng(1)
    dims = [(784, 1000), (1000, 1000), (1000, 10)]
    xs = [rng.random((128, di)).astype(np.float32) for di, _ in dims]
    gys = [(rng.standard_normal((128, do)) / 128).astype(np.float32)
           for _, do in dims]
    gWs = [rng.standard_normal((do, di)).astype(np.float32) for di, do in dims]
    gbs = [rng.standard_normal(do).astype(np.float32) for _, do in dims]
    F, items = [], []
    for (di, do), x, gy in zip(dims, xs, gys):
        A = torch.empty((di + 1, di + 1), device='cuda')
        G = torch.empty((do, do), device='cuda')
        F += [A, G]
        items.append(ops.dense_item(dev(x), True, 1.0 / 128, 0.0, A))
        items.append(ops.dense_item(dev(gy), False, 128.0, 0.0, G))
    ops.factor_group(items, F[0].device)
    inv = [torch.empty_like(f) for f in F]
    plan = ops.InversePlan(F, inv, [1, 0, 3, 2, 5, 4], [0, 1] * 3)
    plan.run(1e-3)
    assert plan.refined() >= 2      # at least the two large A factors
    kW = [torch.empty(w.shape, device='cuda') for w in gWs]
    kb = [torch.empty(b.shape, device='cuda') for b in gbs]
    ops.precondition([inv[1], inv[3], inv[5]], [inv[0], inv[2], inv[4]],
                     [dev(w) for w in gWs], [dev(b) for b in gbs], kW, kb)
    for i in range(3):
        want = orc.connection_step(orc.linear_A(xs[i], True),
                                   orc.linear_G(gys[i]), gWs[i], gbs[i], 1e-3)
        assert rel(host(F[2 * i]), want['ema_A']) < FACTOR_TOL
        # These factors are ill-conditioned (uniform[0,1) inputs: cond ~ 6e3
        # to 1.4e4 with damping 1e-3); the plan's probe sees that and runs
        # the fp64-residual refinement step on them.  The inverse stage is
        # compared on identical inputs: the oracle inverts the factor this
        # stage was given (a factor that differs by 2e-6 moves the inverse
        # by up to cond * 2e-6, whoever computes it), with the damping the
        # oracle derives from it.
        for j, key in ((0, 'A_inv'), (1, 'G_inv')):
            f = host(F[2 * i + j])
            _, dA, dG = orc.connection_damping(host(F[2 * i]),
                                               host(F[2 * i + 1]), 1e-3)
            add = np.float32(dA if j == 0 else dG)
            oracle_inv = orc.damped_inverse(f, add)
            truth = np.linalg.inv(f.astype(np.float64) +
                                  float(add) * np.eye(len(f)))
            got = host(inv[2 * i + j])
            assert rel(got, oracle_inv) < INVERSE_TOL, (i, key)
            assert rel(got, truth) < INVERSE_TOL, (i, key)
        assert rel(host(kW[i]), want['kfgrad_W']) < KFGRAD_TOL
        assert rel(host(kb[i]), want['kfgrad_b']) < KFGRAD_TOL
    plan.close()
