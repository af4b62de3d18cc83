"""Fused bias + ReLU (+ pooling) kernels of the convolution blocks (`csrc/kernels/model_ops.cu`,
`bagua_core_b200/ops/fused_conv.py`): the CUDA kernels against their host restatement and against
plain fp32 PyTorch math, the modules under autocast, and the fused VGG-16 against the unfused one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def bb_launches():
    import bagua_core_b200 as bb

    return bb._C.op_stats()["launches"]


def _stream():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("rows,C", [(1, 8), (37, 64), (1000, 128), (4099, 256), (32 * 14 * 14, 512), (3, 2048)])
def test_bias_relu_forward_and_backward_match_fp32_math(rows, C):
    import bagua_core_b200 as bb

    g = torch.Generator().manual_seed(rows + C)
    z = torch.randn(rows, C, generator=g).to(torch.bfloat16).cuda()
    bias = torch.randn(C, generator=g).to(torch.bfloat16).cuda()
    ref = torch.relu(z.float() + bias.float())
    y = z.clone()
    bb._C.k_bias_relu_(y, bias, _stream())
    assert torch.allclose(y.float(), ref, rtol=8e-3, atol=8e-3)
    assert torch.equal(y > 0, ref.to(torch.bfloat16) > 0)

    dy = torch.randn(rows, C, generator=g).to(torch.bfloat16).cuda()
    dz = torch.empty_like(dy)
    db = torch.empty(C, device="cuda")
    bb._C.k_bias_relu_backward(dy, y, dz, db, _stream())
    dz_ref = torch.where(y > 0, dy, torch.zeros_like(dy))
    assert torch.equal(dz, dz_ref)
    db_ref = dz_ref.double().sum(0)
    assert torch.allclose(db.double(), db_ref, rtol=1e-4, atol=1e-3 * max(1.0, rows ** 0.5))
    # bit-reproducible
    db2 = torch.empty_like(db)
    bb._C.k_bias_relu_backward(dy, y, torch.empty_like(dy), db2, _stream())
    assert torch.equal(db, db2)


def test_channels_last_activation_is_accepted_and_nchw_rejected():
    import bagua_core_b200 as bb

    z = torch.randn(4, 64, 6, 5).to(torch.bfloat16).cuda().contiguous(memory_format=torch.channels_last)
    bias = torch.randn(64).to(torch.bfloat16).cuda()
    ref = torch.relu(z.float() + bias.float().view(1, -1, 1, 1))
    bb._C.k_bias_relu_(z, bias, _stream())
    assert torch.allclose(z.float(), ref, rtol=8e-3, atol=8e-3)
    with pytest.raises(RuntimeError, match="channels-last"):
        bb._C.k_bias_relu_(torch.zeros(4, 64, 6, 5, dtype=torch.bfloat16, device="cuda"), bias, _stream())


@pytest.mark.parametrize("shape", [(1, 8, 2, 2), (2, 64, 6, 10), (3, 128, 56, 56), (32, 512, 14, 14)])
def test_maxpool2x2_matches_torch_bit_for_bit(shape):
    from bagua_core_b200.ops.fused_conv import MaxPool2x2

    g = torch.Generator().manual_seed(sum(shape))
    # values on a coarse grid so that windows contain ties; half of them clamped to zero like a ReLU output
    x = torch.relu((torch.randn(*shape, generator=g) * 4).round() / 4).to(torch.bfloat16).cuda()
    x = x.contiguous(memory_format=torch.channels_last)
    xa, xb = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
    ya = MaxPool2x2()(xa)
    yb = torch.nn.functional.max_pool2d(xb, 2, 2)
    assert ya.is_contiguous(memory_format=torch.channels_last)
    assert torch.equal(ya, yb)
    go = torch.randn(ya.shape, generator=g).to(torch.bfloat16).cuda().contiguous(memory_format=torch.channels_last)
    ya.backward(go)
    yb.backward(go)
    assert torch.equal(xa.grad, xb.grad)


def test_maxpool2x2_falls_back_for_odd_sizes_and_fp32():
    from bagua_core_b200.ops.fused_conv import MaxPool2x2

    for x in (torch.randn(2, 8, 5, 7, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last),
              torch.randn(2, 8, 4, 4, device="cuda")):
        assert torch.equal(MaxPool2x2()(x), torch.nn.functional.max_pool2d(x, 2, 2))


def test_conv_bias_relu_module_matches_conv_plus_relu_under_autocast():
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU

    torch.manual_seed(0)
    fused = ConvBiasReLU(16, 64, 3, padding=1).cuda().to(memory_format=torch.channels_last)
    plain = torch.nn.Conv2d(16, 64, 3, padding=1).cuda().to(memory_format=torch.channels_last)
    plain.load_state_dict(fused.state_dict())
    x = torch.randn(8, 16, 20, 20, device="cuda").contiguous(memory_format=torch.channels_last)
    xa = x.clone().requires_grad_(True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        ya = fused(xa)
        yb = torch.relu(plain(x))
    assert ya.dtype == torch.bfloat16 and torch.allclose(ya.float(), yb.float(), rtol=2e-2, atol=2e-2)
    # Backward against fp32 math on the forward's own ReLU mask and on the bf16-rounded operands
    # (a few masks differ between two bf16 forwards, so another bf16 backward is not a sharp reference).
    go = torch.randn_like(ya)
    ya.backward(go)
    dz = torch.where(ya > 0, go, torch.zeros_like(go)).float()
    w16, x16 = fused.weight.detach().to(torch.bfloat16).float(), x.to(torch.bfloat16).float()
    refs = [torch.nn.grad.conv2d_input(x.shape, w16, dz, padding=1), torch.nn.grad.conv2d_weight(x16, w16.shape, dz, padding=1),
            dz.sum((0, 2, 3))]
    for got, ref in zip([xa.grad, fused.weight.grad, fused.bias.grad], refs):
        assert got.dtype == torch.float32 and got.shape == ref.shape
        scale = ref.abs().max().item() + 1e-6
        assert (got - ref).abs().max().item() <= 1.5e-2 * scale


def test_fused_vgg16_step_matches_unfused():
    from bagua_core_b200.models import VGG16

    torch.manual_seed(1)
    a = VGG16(num_classes=10, dropout=0.0, fused_ops=True).cuda().to(memory_format=torch.channels_last)
    b = VGG16(num_classes=10, dropout=0.0).cuda().to(memory_format=torch.channels_last)
    for pa, pb in zip(a.parameters(), b.parameters()):
        pb.data.copy_(pa.data)
    x = torch.randn(4, 3, 64, 64, device="cuda").contiguous(memory_format=torch.channels_last)
    t = torch.randint(0, 10, (4,), device="cuda")
    losses = []
    for m in (a, b):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = torch.nn.functional.cross_entropy(m(x).float(), t)
        loss.backward()
        losses.append(loss.item())
    assert abs(losses[0] - losses[1]) <= 2e-2 * max(1.0, abs(losses[1]))
    for pa, pb in zip(a.parameters(), b.parameters()):
        scale = pb.grad.abs().max().item() + 1e-6
        assert (pa.grad - pb.grad).abs().max().item() <= 0.2 * scale  # ReLU masks flip here and there between two bf16 runs


@pytest.mark.parametrize("shape", [(1, 8, 2, 2), (2, 64, 6, 10), (4, 128, 28, 28), (32, 512, 14, 14), (8, 64, 56, 56)])
def test_cuda_kernels_match_the_host_restatement_exactly(shape):
    """Every model kernel on the GPU against the same binding on CPU tensors (plain loops)."""
    import bagua_core_b200 as bb

    C = bb._C
    n, c, h, w = shape
    g = torch.Generator().manual_seed(sum(shape))

    def rnd(*s, relu=False):
        t = (torch.randn(*s, generator=g) * 4).round() / 4
        t = torch.relu(t) if relu else t
        t = t.to(torch.bfloat16)
        return t.contiguous(memory_format=torch.channels_last) if t.dim() == 4 else t

    s = _stream()
    # bias + ReLU
    z, bias = rnd(n, c, h, w), rnd(c)
    z_h, z_d = z.clone(), z.cuda()
    C.k_bias_relu_(z_h, bias, 0)
    C.k_bias_relu_(z_d, bias.cuda(), s)
    assert torch.equal(z_d.cpu(), z_h)
    dy = rnd(n, c, h, w)
    dz_h, db_h = torch.empty_like(dy), torch.empty(c)
    dz_d, db_d = torch.empty_like(dy).cuda(), torch.empty(c, device="cuda")
    C.k_bias_relu_backward(dy, z_h, dz_h, db_h, 0)
    C.k_bias_relu_backward(dy.cuda(), z_d, dz_d, db_d, s)
    assert torch.equal(dz_d.cpu(), dz_h)
    assert torch.allclose(db_d.cpu(), db_h, rtol=1e-4, atol=1e-2)
    # max pooling
    x = rnd(n, c, h, w, relu=True)
    y_h = torch.empty((n, c, h // 2, w // 2), dtype=torch.bfloat16).contiguous(memory_format=torch.channels_last)
    y_d = y_h.cuda()
    C.k_maxpool2x2_forward(x, y_h, 0)
    C.k_maxpool2x2_forward(x.cuda(), y_d, s)
    assert torch.equal(y_d.cpu(), y_h)
    gy = rnd(n, c, h // 2, w // 2)
    dx_h, dx_d = torch.empty_like(x), torch.empty_like(x).cuda()
    C.k_maxpool2x2_backward(x, gy, dx_h, 0)
    C.k_maxpool2x2_backward(x.cuda(), gy.cuda(), dx_d, s)
    assert torch.equal(dx_d.cpu(), dx_h)
    # bias + ReLU + pooling in one pass
    a_h, a_d = z.clone(), z.cuda()
    p_h, p_d = torch.empty_like(y_h), torch.empty_like(y_h).cuda()
    C.k_bias_relu_pool_(a_h, p_h, bias, 0)
    C.k_bias_relu_pool_(a_d, p_d, bias.cuda(), s)
    assert torch.equal(a_d.cpu(), a_h) and torch.equal(p_d.cpu(), p_h)
    dzp_h, dbp_h = torch.empty_like(z), torch.empty(c)
    dzp_d, dbp_d = torch.empty_like(z).cuda(), torch.empty(c, device="cuda")
    C.k_bias_relu_pool_backward(gy, a_h, dzp_h, dbp_h, 0)
    C.k_bias_relu_pool_backward(gy.cuda(), a_d, dzp_d, dbp_d, s)
    assert torch.equal(dzp_d.cpu(), dzp_h)
    assert torch.allclose(dbp_d.cpu(), dbp_h, rtol=1e-4, atol=1e-2)


def test_conv_bias_relu_pool_module_matches_the_composition_under_autocast():
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU, ConvBiasReLUPool

    torch.manual_seed(0)
    pooled = ConvBiasReLUPool(16, 64, 3, padding=1).cuda().to(memory_format=torch.channels_last)
    single = ConvBiasReLU(16, 64, 3, padding=1).cuda().to(memory_format=torch.channels_last)
    single.load_state_dict(pooled.state_dict())
    x = torch.randn(8, 16, 20, 24, device="cuda").contiguous(memory_format=torch.channels_last)
    xa, xb = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        pa = pooled(xa)
        pb = torch.nn.functional.max_pool2d(single(xb), 2, 2)
    assert torch.allclose(pa.float(), pb.float(), rtol=2e-2, atol=2e-2)  # same math; the library may pick another conv algorithm
    go = torch.randn_like(pa)
    pa.backward(go)
    pb.backward(go)
    for a, b in [(xa.grad, xb.grad), (pooled.weight.grad, single.weight.grad), (pooled.bias.grad, single.bias.grad)]:
        scale = b.abs().max().item() + 1e-6
        assert (a - b).abs().max().item() <= 6e-2 * scale  # masks agree except where two conv algorithms round apart




@pytest.mark.parametrize("n", [1, 7, 4096, (1 << 20) + 3])
def test_sgd_step_with_bf16_copy_equals_the_plain_step(n):
    import bagua_core_b200 as bb

    C = bb._C
    g = torch.Generator().manual_seed(n)
    p, grad = torch.randn(n, generator=g).cuda(), torch.randn(n, generator=g).cuda()
    m = torch.zeros(n, device="cuda")
    p2, m2, h = p.clone(), m.clone(), torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    for step in range(3):
        C.k_sgd_momentum_flat(p, grad, m, 0.1, 0.9, 0.0, 1e-4, True, step == 0, s)
        C.k_sgd_momentum_flat_shadow(p2, grad, m2, h, 0.1, 0.9, 0.0, 1e-4, True, step == 0, s)
        torch.cuda.synchronize()
        assert torch.equal(p, p2) and torch.equal(m, m2) and torch.equal(h, p2.to(torch.bfloat16))
    # an unaligned view takes the scalar path
    if n > 8:
        q = torch.randn(n + 1, generator=g).cuda()[1:]  # 4 bytes past a 16-byte boundary
        q2 = torch.empty(n + 1, device="cuda")[1:].copy_(q)
        hq = torch.zeros(n + 1, dtype=torch.bfloat16, device="cuda")[1:]
        C.k_sgd_momentum_flat(q, grad, m, 0.1, 0.9, 0.0, 0.0, False, False, s)
        C.k_sgd_momentum_flat_shadow(q2, grad, m2, hq, 0.1, 0.9, 0.0, 0.0, False, False, s)
        torch.cuda.synchronize()
        assert torch.equal(q, q2) and torch.equal(hq, q2.to(torch.bfloat16))


def test_vgg_training_with_bf16_weight_copies_is_bit_identical_to_casting():
    """Same model, same data: lookups switched off (the blocks cast the fp32 weights in every forward pass) against
    lookups on (they read the optimizer's copies)."""
    import os

    import bagua_core_b200.parallel as P
    from bagua_core_b200.models import VGG16
    from bagua_core_b200.ops import shadow as S

    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    os.environ.setdefault("MASTER_PORT", "29541")
    dev = torch.device("cuda", 0)
    results = []
    for use_copies in (False, True):
        S.enabled = use_copies
        torch.manual_seed(0)
        model = VGG16(num_classes=10, dropout=0.0, fused_ops=True).to(dev).to(memory_format=torch.channels_last)
        P.init_process_group(dev)
        opt = P.FlatSGD(model.parameters(), lr=0.01, momentum=0.9, bf16_shadow=True)
        bm = P.with_bagua(model, [opt], P.GradientAllReduceAlgorithm(), bucket_bytes=10 << 20)
        g = torch.Generator().manual_seed(5)
        hits0, losses = S.hits, []
        for _ in range(4):
            x = torch.randn(4, 3, 64, 64, generator=g).to(dev).contiguous(memory_format=torch.channels_last)
            y = torch.randint(0, 10, (4,), generator=g).to(dev)
            opt.zero_grad()
            with torch.autocast("cuda", dtype=torch.bfloat16):
                loss = torch.nn.functional.cross_entropy(bm(x).float(), y)
            loss.backward()
            opt.step()
            losses.append(loss.item())
        torch.cuda.synchronize()
        results.append((losses, torch.cat([p.detach().reshape(-1) for p in model.parameters()]).clone(), S.hits - hits0))
        P.destroy_process_group()
    S.enabled = True
    assert results[0][2] == 0 and results[1][2] == 3 * 16  # 13 convolutions + 3 linear layers, from the second step on
    assert results[0][0] == results[1][0]
    assert torch.equal(results[0][1], results[1][1])




@pytest.mark.parametrize("rows,n_in,n_out", [(32, 25088, 4096), (32, 4096, 1000), (5, 72, 24)])
def test_linear_weight_gradient_accumulated_in_place_is_the_fp32_product(rows, n_in, n_out):
    """The library GEMM adds dyᵀ x (bf16 operands) into the fp32 gradient; compared with the same
    operands multiplied in fp32 by plain PyTorch, twice in a row (the second call adds)."""
    from bagua_core_b200.ops import wgrad as W
    from bagua_core_b200.ops.fused_linear import ShadowLinear

    saved, W.enabled = W.enabled, True
    try:
        torch.manual_seed(rows + n_in)
        m = ShadowLinear(n_in, n_out).cuda()
        for p in m.parameters():
            p.grad = torch.zeros_like(p)
        fired = []
        m.weight.register_post_accumulate_grad_hook(lambda p: fired.append(1))
        x = torch.randn(rows, n_in, device="cuda")
        a0 = W.accumulated
        for k in (1, 2):
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = m(x)
            dy = torch.randn_like(y)
            y.backward(dy)
            torch.cuda.synchronize()
            assert W.accumulated == a0 + k and len(fired) == k, (W.accumulated, W.declined, W.cuda_mode)
            want = k * (dy.to(torch.bfloat16).float().t() @ x.to(torch.bfloat16).float()) if k == 1 else want + \
                dy.to(torch.bfloat16).float().t() @ x.to(torch.bfloat16).float()
            scale = want.abs().max().item()
            assert (m.weight.grad - want).abs().max().item() <= 2e-3 * scale + 1e-5
        assert W.cuda_mode in ("addmm", "mm_add")
    finally:
        W.enabled = saved


def test_vgg_training_with_in_place_weight_gradients_agrees_with_the_ordinary_path():
    import os

    import bagua_core_b200.parallel as P
    from bagua_core_b200.models import VGG16
    from bagua_core_b200.ops import wgrad as W

    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    os.environ.setdefault("MASTER_PORT", "29543")
    dev = torch.device("cuda", 0)
    saved, results = W.enabled, []
    try:
        for inplace in (False, True):
            W.enabled = inplace
            torch.manual_seed(0)
            model = VGG16(num_classes=10, dropout=0.0, fused_ops=True).to(dev).to(memory_format=torch.channels_last)
            P.init_process_group(dev)
            opt = P.FlatSGD(model.parameters(), lr=0.01, momentum=0.9)
            bm = P.with_bagua(model, [opt], P.GradientAllReduceAlgorithm(), bucket_bytes=10 << 20)
            g = torch.Generator().manual_seed(5)
            a0, losses = W.accumulated, []
            for _ in range(4):
                x = torch.randn(4, 3, 64, 64, generator=g).to(dev).contiguous(memory_format=torch.channels_last)
                y = torch.randint(0, 10, (4,), generator=g).to(dev)
                opt.zero_grad()
                with torch.autocast("cuda", dtype=torch.bfloat16):
                    loss = torch.nn.functional.cross_entropy(bm(x).float(), y)
                loss.backward()
                opt.step()
                losses.append(loss.item())
            torch.cuda.synchronize()
            results.append((losses, torch.cat([p.detach().reshape(-1) for p in model.parameters()]).clone(),
                            W.accumulated - a0))
            P.destroy_process_group()
    finally:
        W.enabled = saved
    assert results[0][2] == 0 and results[1][2] == 4 * 3  # three linear layers, four steps
    assert all(abs(a - b) < 5e-2 for a, b in zip(results[0][0], results[1][0])), (results[0][0], results[1][0])
    assert (results[0][1] - results[1][1]).abs().max().item() < 2e-2


@pytest.mark.parametrize("shape", [(1, 8, 2, 2), (3, 2048, 4, 6), (2, 64, 6, 10), (5, 16, 14, 2), (8, 64, 56, 56)])
def test_pooling_without_the_activation_equals_the_in_place_pair(shape):
    """Values on a coarse grid (ties in most windows), negative biases (windows without a positive value), -0."""
    import bagua_core_b200 as bb

    n, c, h, w = shape
    g = torch.Generator().manual_seed(sum(shape))

    def rnd(*s):
        t = ((torch.randn(*s, generator=g) * 4).round() / 4).to(torch.bfloat16).cuda()
        return t.contiguous(memory_format=torch.channels_last) if len(s) == 4 else t

    z, bias, dp = rnd(*shape), rnd(c) - 0.25, rnd(n, c, h // 2, w // 2)
    z[:, :, 0, 0] = -0.0
    bias[0] = -0.0
    y, z0 = z.clone(), z.clone()
    p, dz, db = torch.empty_like(dp), torch.empty_like(z), torch.empty(c, device="cuda")
    bb._C.k_bias_relu_pool_(y, p, bias, _stream())
    bb._C.k_bias_relu_pool_backward(dp, y, dz, db, _stream())
    p2, dz2, db2 = torch.full_like(p, 9), torch.full_like(z, 9), torch.empty_like(db)
    bb._C.k_bias_relu_pool(z, p2, bias, _stream())
    bb._C.k_bias_relu_pool_backward(dp, z, dz2, db2, _stream(), bias)
    assert torch.equal(z, z0) and torch.equal(p, p2) and torch.equal(dz, dz2) and torch.equal(db, db2)


@pytest.mark.parametrize("rows,n_in,n_out", [(1, 8, 8), (31, 16, 264), (3072, 64, 1024), (33, 40, 1000), (5, 72, 10), (70, 8, 4096)])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_linear_gradients_land_in_an_fp32_bucket_at_any_alignment(rows, n_in, n_out, offset):
    """Weight and bias gradients are views of one buffer, back to back from element `offset` on: added in place,
    twice, and equal to the same bf16 operands multiplied and summed in fp32."""
    from bagua_core_b200.ops import wgrad as W
    from bagua_core_b200.ops.fused_linear import ShadowLinear

    saved, W.enabled = W.enabled, True
    try:
        torch.manual_seed(rows + n_out)
        m = ShadowLinear(n_in, n_out).cuda()
        flat = torch.zeros(offset + n_out + n_out * n_in + 8, device="cuda")
        m.bias.grad = flat[offset:offset + n_out]
        m.weight.grad = flat[offset + n_out:offset + n_out + n_out * n_in].view(n_out, n_in)
        x = torch.randn(rows, n_in, device="cuda", requires_grad=True)
        want_w, want_b = torch.zeros_like(m.weight), torch.zeros_like(m.bias)
        for _ in range(2):
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = m(x)
            dy = torch.randn_like(y)
            y.backward(dy)
            want_w += dy.float().t() @ x.detach().bfloat16().float()
            want_b += dy.float().sum(0)
        assert m.weight.grad.data_ptr() == flat[offset + n_out:].data_ptr()
        assert (m.weight.grad - want_w).abs().max() <= 2e-3 * want_w.abs().max() + 1e-5
        assert torch.allclose(m.bias.grad, want_b, rtol=1e-4, atol=1e-3 * rows ** 0.5)
        assert bool((flat[:offset] == 0).all() and (flat[-8:] == 0).all())
    finally:
        W.enabled = saved


def test_block_gradients_added_in_place_have_the_bits_of_the_ordinary_path():
    from bagua_core_b200.ops import wgrad as W
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU, ConvBiasReLUPool

    saved, grads = W.enabled, []
    try:
        for W.enabled in (False, True):
            torch.manual_seed(5)
            net = torch.nn.Sequential(ConvBiasReLU(3, 24, 3, padding=1), ConvBiasReLUPool(24, 64, 3, padding=1)).cuda()
            net = net.to(memory_format=torch.channels_last)
            for p in net.parameters():
                p.grad = torch.zeros_like(p, memory_format=torch.preserve_format)
            x = torch.randn(3, 3, 12, 20, device="cuda").contiguous(memory_format=torch.channels_last)
            for _ in range(2):
                with torch.autocast("cuda", dtype=torch.bfloat16):
                    net(x).float().square().sum().backward()
            grads.append([p.grad.clone() for p in net.parameters()])
    finally:
        W.enabled = saved
    for a, b in zip(*grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("N,H,W,Ci,C", [(1, 1, 1, 3, 64), (1, 1, 63, 1, 64), (2, 13, 5, 2, 128), (1, 8, 8, 3, 64), (3, 65, 1, 3, 256),
                                        (2, 61, 67, 3, 64), (8, 112, 112, 3, 64)])
@pytest.mark.parametrize("in_place", [False, True])
def test_first_layer_gradients_match_fp32_math(N, H, W, Ci, C, in_place):
    """No gradient for the input: the block's weight and bias gradients come from one kernel."""
    from bagua_core_b200.ops import wgrad as Wg
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU

    torch.manual_seed(N * H + W)
    m = ConvBiasReLU(Ci, C, 3, padding=1).cuda().to(memory_format=torch.channels_last if in_place or N > 1 else torch.contiguous_format)
    torch.nn.init.normal_(m.bias, 0.0, 0.1)
    for p in m.parameters():
        p.grad = torch.ones_like(p)
    x = torch.randn(N, Ci, H, W, device="cuda").to(memory_format=torch.channels_last)
    saved = Wg.enabled
    Wg.enabled = in_place
    try:
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = m(x)
        dy = torch.randn(y.shape, device="cuda").to(torch.bfloat16).to(memory_format=torch.channels_last)
        mid = bb_launches()
        y.backward(dy)
    finally:
        Wg.enabled = saved
    assert bb_launches() - mid == 2
    dz = torch.where(y > 0, dy, torch.zeros_like(dy)).detach().double()
    patches = torch.nn.functional.unfold(x.bfloat16().double(), 3, padding=1)  # [N, Ci * 9, H * W]
    dw = torch.einsum("ncp,nkp->ck", dz.reshape(N, C, H * W), patches).view(C, Ci, 3, 3)
    db = dz.sum((0, 2, 3))
    assert (m.bias.grad.double() - (1 + db)).abs().max() <= 1e-5 * db.abs().max()
    # rounded to bf16, and the patches' order of summation moves a few values to their neighbours
    got, want = m.weight.grad.double() - 1, dw
    assert ((got - want).abs() <= 4.1e-3 * want.abs() + 1e-5 * want.abs().max()).all()


@pytest.mark.parametrize("image_grad,c_in,kept", [(False, 3, False), (True, 3, True), (False, 64, True)])
def test_a_block_whose_backward_reads_the_activation_keeps_no_signs(image_grad, c_in, kept):
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU

    torch.manual_seed(c_in)
    m = ConvBiasReLU(c_in, 64, 3, padding=1).cuda().to(memory_format=torch.channels_last)
    x = torch.randn(2, c_in, 14, 10, device="cuda").to(memory_format=torch.channels_last).requires_grad_(image_grad)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t) or t, lambda t: t), torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(x)
    assert [t.numel() for t in seen if t.dtype == torch.uint8] == ([y.numel() // 8] if kept else [])
    dy = torch.randn(y.shape, device="cuda").to(torch.bfloat16).to(memory_format=torch.channels_last)
    # the bias gradient alone takes the general path, with or without them
    db, = torch.autograd.grad(y, [m.bias], dy)
    want = torch.where(y > 0, dy, torch.zeros_like(dy)).double().sum((0, 2, 3))
    assert (db.double() - want).abs().max() <= 1e-5 * want.abs().max()


@pytest.mark.parametrize("N,C,H,W", [(1, 8, 2, 2), (2, 64, 6, 10), (1, 2048, 4, 2), (3, 16, 1, 7), (5, 32, 34, 38), (2, 128, 3, 5), (8, 64, 112, 96)])
@pytest.mark.parametrize("pool", [False, True])
def test_blocks_keep_the_signs_and_places_that_their_backward_needs(N, C, H, W, pool):
    """An identity as convolution, and few values, so that windows are full of ties, zeros and negative zeros."""
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU, ConvBiasReLUPool

    if pool and (H % 2 or W % 2):
        pytest.skip("windows do not tile the image: the framework's path")
    g = torch.Generator(device="cuda").manual_seed(C + H)

    def draw(*shape):
        return (torch.randint(-2, 3, shape, device="cuda", generator=g) / 2).to(torch.bfloat16)

    m = (ConvBiasReLUPool if pool else ConvBiasReLU)(C, C, 1).cuda().to(dtype=torch.bfloat16)
    with torch.no_grad():
        m.weight.copy_(torch.eye(C).view(C, C, 1, 1))
        m.bias.copy_(torch.where(torch.rand(C, device="cuda", generator=g) < 0.5, -0.0, -0.5))
    x = draw(N, H, W, C).permute(0, 3, 1, 2).requires_grad_()
    ref = x.detach().clone(memory_format=torch.preserve_format).requires_grad_()
    z = ref + m.bias.detach().view(1, -1, 1, 1)
    z.retain_grad()
    want = torch.relu(z)
    want = torch.nn.functional.max_pool2d(want, 2, 2) if pool else want
    y = m(x)
    assert torch.equal(y, want)
    dy = draw(*y.permute(0, 2, 3, 1).shape).permute(0, 3, 1, 2)
    y.backward(dy)
    want.backward(dy)
    assert torch.equal(x.grad, ref.grad)
    # sums of halves are exact in fp32
    assert torch.equal(m.bias.grad, z.grad.float().sum((0, 2, 3)).to(torch.bfloat16))


# rectangles that end with the image and that reach over it, one and several strips, rows in pairs, one block and many splits
@pytest.mark.parametrize("N,H,W,Ci,Co", [(1, 1, 1, 64, 64), (2, 3, 7, 64, 128), (1, 14, 14, 128, 64), (3, 17, 23, 192, 64), (1, 5, 57, 64, 64),
                                         (2, 65, 129, 64, 64), (1, 1, 3, 128, 128), (2, 9, 11, 128, 256), (5, 28, 28, 256, 128),
                                         (1, 5, 300, 128, 128), (2, 56, 56, 128, 384), (2, 14, 14, 512, 512), (4, 112, 112, 128, 128)])
def test_convolution_weight_gradient_is_the_rounded_sum(N, H, W, Ci, Co):
    """Multiples of 1/4 up to 1/2: every sum is exact in fp32 in any order, so the bits are those of the rounded result."""
    import bagua_core_b200 as bb

    g = torch.Generator(device="cuda").manual_seed(H * W + Ci)

    def draw(c):
        t = torch.randint(-2, 3, (N, H, W, c), device="cuda", generator=g).to(torch.bfloat16) / 4
        return t.permute(0, 3, 1, 2)

    dz, x = draw(Co), draw(Ci)
    xp = torch.nn.functional.pad(x.permute(0, 2, 3, 1).double(), (0, 0, 1, 1, 1, 1))
    d = dz.permute(0, 2, 3, 1).double().reshape(-1, Co)
    want = torch.stack([torch.stack([d.t() @ xp[:, r:r + H, s:s + W].reshape(-1, Ci) for s in range(3)], -1) for r in range(3)], -2)
    want = want.to(torch.bfloat16)
    for layout in (torch.channels_last, torch.contiguous_format):
        low = torch.full((Co, Ci, 3, 3), 7.0, device="cuda", dtype=torch.bfloat16).to(memory_format=layout)
        bb._C.k_conv_weight_gradient(dz, x, low, _stream())
        assert torch.equal(low, want)


@pytest.mark.parametrize("N,H,W,Ci,C,own", [(2, 56, 56, 64, 64, True), (1, 56, 56, 64, 64, False), (8, 56, 56, 256, 512, True),
                                            (7, 56, 56, 256, 512, False), (2, 56, 56, 64, 32, False), (256, 7, 7, 64, 64, False)])
@pytest.mark.parametrize("kind", [torch.bfloat16, torch.float32])
def test_conv_blocks_on_both_sides_of_the_rule_for_their_weight_gradient(N, H, W, Ci, C, own, kind):
    import bagua_core_b200 as bb
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU

    assert bb._C.k_conv_weight_gradient_preferred(N, H, W, C, Ci) == own
    torch.manual_seed(C)
    m = ConvBiasReLU(Ci, C, 3, padding=1).cuda().to(dtype=kind, memory_format=torch.channels_last)
    x = torch.randn(N, Ci, H, W, device="cuda", dtype=kind).to(memory_format=torch.channels_last).requires_grad_()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(x)
    dy = torch.randn(y.shape, device="cuda").to(torch.bfloat16).to(memory_format=torch.channels_last)
    before = bb_launches()
    y.backward(dy)
    assert bb_launches() - before == (4 if own and kind is torch.bfloat16 else 2)
    dz = torch.where(y > 0, dy, torch.zeros_like(dy)).detach()
    ref = torch.ops.aten.convolution_backward(dz, x.detach().bfloat16(), m.weight.detach().bfloat16(), None, [1, 1], [1, 1], [1, 1], False,
                                              [0, 0], 1, [False, True, False])[1].float()
    got = m.weight.grad.float()
    # two roundings to bf16 (2^-9 each) of sums in fp32 whose order differs
    assert (got - ref).norm() <= 2 ** -8 * ref.norm()
    assert ((got - ref).abs() <= 2 ** -7 * ref.abs() + 2e-5 * ref.abs().max()).all()


@pytest.mark.parametrize("rows,H", [(1, 8), (5, 264), (37, 768), (3072, 1024)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_add_layer_norm_has_the_bits_of_the_plain_composition(rows, H, accumulate):
    import bagua_core_b200 as bb

    g = torch.Generator().manual_seed(rows + H)
    x, r, dy = (torch.randn(rows, H, generator=g).bfloat16().cuda().requires_grad_() for _ in range(3))
    gamma, beta = (torch.randn(H, generator=g).cuda().requires_grad_() for _ in range(2))
    for res in (r, None):
        y = bb._C.add_layer_norm(x, res, gamma, beta, 1e-5, accumulate)
        ref = torch.nn.functional.layer_norm(x if res is None else x + res, (H,), gamma.bfloat16(), beta.bfloat16(), 1e-5)
        assert torch.equal(y, ref)
        leaves, out = [t for t in (x, res, gamma, beta) if t is not None], []
        for v in (y, ref):
            for t in leaves:
                t.grad = torch.zeros_like(t)
            v.backward(dy.detach())
            out.append([t.grad.clone() for t in leaves])
        for a, b in zip(*out):
            assert torch.equal(a, b)


@pytest.mark.parametrize("batch,seq,V,same", [(1, 1, 5, 0), (3, 7, 11, 0), (8, 384, 30522, 0), (2, 300, 9, 500), (8, 512, 1000, 3000)])
def test_embedding_sum_and_norm_match_the_plain_composition(batch, seq, V, same):
    """`same`: that many tokens are one id (padding): above 256 its rows are added by several blocks."""
    import bagua_core_b200 as bb

    g = torch.Generator().manual_seed(seq)
    H = 72
    ids = torch.randint(0, V, (batch, seq), generator=g)
    ids.view(-1)[torch.randperm(batch * seq, generator=g)[:same]] = V - 1
    ids = ids.cuda()
    tabs = [torch.randn(n, H, generator=g).cuda() for n in (V, 512, 2)] + [torch.randn(H, generator=g).cuda() for _ in range(2)]
    a, b = ([t.clone().requires_grad_() for t in tabs] for _ in range(2))
    y = bb._C.embed_layer_norm(ids, *a, 1e-12, False)
    s = torch.nn.functional.embedding(ids, b[0]) + b[1][:seq][None] + b[2][0][None, None]
    ref = torch.nn.functional.layer_norm(s, (H,), b[3], b[4], 1e-12)
    dy = torch.randn(ref.shape, generator=g).bfloat16().cuda()
    assert torch.allclose(y.float(), ref, rtol=1e-2, atol=1e-2)
    y.backward(dy)
    ref.backward(dy.float())
    for p, q in zip(a, b):
        assert torch.allclose(p.grad, q.grad, rtol=1e-3, atol=1e-4 * max(1.0, q.grad.abs().max().item())), p.shape


@pytest.mark.parametrize("rows,n_out", [(1, 8), (9, 264), (64, 128), (65, 128), (300, 4096)])
@pytest.mark.parametrize("accumulate", [False, True])
@pytest.mark.parametrize("activation", [1, 2])
def test_linear_with_activation_matches_the_plain_composition(rows, n_out, accumulate, activation):
    import bagua_core_b200 as bb

    act = {1: torch.nn.functional.gelu, 2: torch.nn.functional.relu}[activation]
    torch.manual_seed(rows)
    x = torch.randn(rows, 32, device="cuda").bfloat16().requires_grad_()
    w, b = torch.randn(n_out, 32, device="cuda", requires_grad=True), torch.randn(n_out, device="cuda", requires_grad=True)
    for p in (w, b):
        p.grad = torch.ones_like(p)
    y = bb._C.linear(x, w, b, None, accumulate, activation)
    z = bb._C.linear(x.detach(), w.detach(), b.detach(), None, False).requires_grad_()
    assert torch.equal(y, act(z))
    dy = torch.randn_like(y)
    y.backward(dy)
    (dz,) = torch.autograd.grad(act(z), z, dy)
    xf, wf, df = x.detach().float(), w.detach().bfloat16().float(), dz.float()
    for got, want in ((x.grad, df @ wf), (w.grad, 1 + df.t() @ xf), (b.grad, 1 + df.sum(0))):
        assert (got.float() - want).abs().max() <= 1e-2 * want.abs().max()


@pytest.mark.parametrize("rows", [1, 256, 257])
@pytest.mark.parametrize("n_out,n_in", [(10, 72), (136, 64)])
def test_weight_gradient_of_any_alignment_is_accumulated(rows, n_out, n_in):
    import bagua_core_b200 as bb

    torch.manual_seed(rows)
    x = torch.randn(rows, n_in, device="cuda").bfloat16()
    w = torch.randn(n_out, n_in, device="cuda", requires_grad=True)
    for offset in (0, 1, 2):
        flat = torch.ones(n_out * n_in + 8, device="cuda")
        w.grad = flat[offset:offset + n_out * n_in].view(n_out, n_in)
        y = bb._C.linear(x, w, None, None, True)
        dy = torch.randn_like(y)
        y.backward(dy)
        want = 1 + dy.float().t() @ x.float()
        assert w.grad.data_ptr() == flat.data_ptr() + 4 * offset
        assert (w.grad - want).abs().max() <= 1e-4 * want.abs().max()
        assert (flat[:offset] == 1).all() and (flat[offset + n_out * n_in:] == 1).all()


@pytest.mark.parametrize("batch,seq", [(1, 1), (3, 7), (8, 384), (40, 33)])
def test_span_loss_matches_two_cross_entropies(batch, seq):
    import bagua_core_b200 as bb

    F = torch.nn.functional
    g = torch.Generator().manual_seed(batch)
    x = (3 * torch.randn(batch, seq, 2, generator=g)).bfloat16().cuda().requires_grad_()
    span = torch.randint(0, seq, (2, batch), generator=g).cuda()
    if batch > 1:
        span[0, 1] = -100
    loss = bb._C.span_loss(x, span[0], span[1])
    ref = (F.cross_entropy(x.float()[..., 0], span[0]) + F.cross_entropy(x.float()[..., 1], span[1])) / 2
    assert torch.allclose(loss, ref, rtol=1e-5)
    (a,), (b,) = torch.autograd.grad(3 * loss, x), torch.autograd.grad(3 * ref, x)
    assert torch.allclose(a.float(), b.float(), rtol=1e-2, atol=1e-6)


def test_bert_layers_through_the_fused_kernels_agree_with_the_plain_composition():
    from bagua_core_b200.models import BertConfig, BertForQuestionAnswering
    from bagua_core_b200.ops import wgrad as W

    saved, out = W.enabled, []
    try:
        for mode in ("plain", "fused", "fused, in place"):
            torch.manual_seed(4)
            net = BertForQuestionAnswering(BertConfig(vocab_size=500, hidden=128, layers=2, heads=4, ffn=256, dropout=0.0,
                                                      fp32_layernorm_io=mode == "plain")).cuda()
            W.enabled = mode.endswith("in place")
            for p in net.parameters():
                p.grad = torch.zeros_like(p)
            g = torch.Generator().manual_seed(1)
            ids = torch.randint(0, 500, (3, 40), generator=g).cuda()
            span = torch.randint(0, 40, (3, 2), generator=g).cuda()
            with torch.autocast("cuda", dtype=torch.bfloat16):
                loss = net(ids, span[:, 0], span[:, 1])
            loss.backward()
            out.append((loss.item(), torch.cat([p.grad.reshape(-1) for p in net.parameters()])))
    finally:
        W.enabled = saved
    for loss, grad in out[1:]:
        assert abs(loss - out[0][0]) < 2e-2
        assert (grad - out[0][1]).norm() <= 4e-2 * out[0][1].norm()


@pytest.mark.parametrize("width", [32, 128, 0])
@pytest.mark.parametrize("activation", ["", "relu", "gelu"])
def test_a_linear_layer_refuses_an_input_of_another_width(width, activation):
    """The products behind the layer are given addresses and sizes only: a wrong width must be refused before them."""
    from bagua_core_b200.ops import wgrad as W
    from bagua_core_b200.ops.fused_linear import ShadowLinear

    m, saved = ShadowLinear(64, 24).cuda(), W.enabled
    W.enabled = True
    try:
        for shape in ((5, width), (2, 5, width)):
            with torch.autocast("cuda", dtype=torch.bfloat16), pytest.raises(RuntimeError):
                m(torch.ones(shape, device="cuda", requires_grad=True), activation)
            with torch.autocast("cuda", dtype=torch.bfloat16), pytest.raises(RuntimeError):
                m(torch.ones(shape[:-1] + (64,)), activation)  # on the host
    finally:
        W.enabled = saved


def test_a_bias_that_is_not_one_value_per_column_takes_the_general_path():
    import bagua_core_b200 as bb
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU

    x, w = torch.randn(6, 16, device="cuda").bfloat16(), torch.randn(24, 16, device="cuda")
    for n in (23, 25):
        with pytest.raises(RuntimeError):
            bb._C.linear(x, w, torch.zeros(n, device="cuda"), None, False)
    flat = torch.zeros(64, device="cuda")  # one value for all columns, its gradient in front of others
    b = torch.ones(1, device="cuda", requires_grad=True)
    b.grad = flat[:1]
    w.requires_grad_().grad = torch.zeros_like(w)
    for activation in (0, 2):
        y = bb._C.linear(x, w, b, None, True, activation)
        y.sum().backward()
    assert bool((flat[1:] == 0).all()) and flat[0] == 6 * 24 + (y > 0).sum()
    m = ConvBiasReLU(16, 64, 3, padding=1).cuda().to(memory_format=torch.channels_last)
    m.bias = torch.nn.Parameter(torch.zeros(32, device="cuda"))
    with torch.autocast("cuda", dtype=torch.bfloat16), pytest.raises(RuntimeError, match="bias"):
        m(torch.zeros(1, 16, 8, 8, device="cuda"))


@pytest.mark.parametrize("offset", [1, 4, 8])
def test_gradients_that_start_anywhere_give_those_of_an_aligned_copy(offset):
    import bagua_core_b200 as bb
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU, ConvBiasReLUPool

    def shifted(t):  # the same values in the same strides, `offset` elements behind an aligned address
        buf = torch.empty(t.numel() + offset, dtype=t.dtype, device=t.device)
        return torch.as_strided(buf, t.shape, t.stride(), offset).copy_(t)

    torch.manual_seed(offset)
    layers = []
    w = torch.randn(40, 16, device="cuda")
    for activation in (0, 1, 2):
        layers.append((lambda x, a=activation: bb._C.linear(x, w, None, None, False, a), torch.randn(70, 16, device="cuda").bfloat16()))
    layers.append((lambda x: bb._C.attention(x, 2, 0.0), torch.randn(2, 16, 96, device="cuda").bfloat16()))
    for cls in (ConvBiasReLU, ConvBiasReLUPool):
        m = cls(16, 64, 3, padding=1).cuda().to(dtype=torch.bfloat16, memory_format=torch.channels_last)
        layers.append((m, torch.randn(2, 16, 8, 8, device="cuda").bfloat16().contiguous(memory_format=torch.channels_last)))
    for f, x in layers:
        x.requires_grad_()
        y = f(x)
        dy = torch.randn(y.shape, device="cuda").bfloat16().as_strided(y.shape, y.stride())
        a, b = (torch.autograd.grad(f(x), x, g)[0] for g in (dy, shifted(dy)))
        # (the library's attention adds parts of its gradients in any order)
        assert torch.equal(a, b) or (x.dim() == 3 and torch.allclose(a.float(), b.float(), rtol=1e-2, atol=1e-3))


@pytest.mark.parametrize("frozen", [(0,), (1,), (2,), (3,), (4,), (0, 1, 2), (0, 2, 3, 4), (3, 4)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_a_frozen_parameter_of_the_embedding_keeps_its_gradient(frozen, accumulate):
    """It may be frozen after its bucket was laid out: `.grad` is there, and must not be added to."""
    import bagua_core_b200 as bb

    g = torch.Generator().manual_seed(1)
    ids = torch.randint(0, 50, (3, 70), generator=g).cuda()
    grads = []
    for off in ((), frozen):
        torch.manual_seed(0)
        ps = [torch.randn(*s, device="cuda", requires_grad=True) for s in ((50, 72), (80, 72), (2, 72), (72,), (72,))]
        for k, p in enumerate(ps):
            p.grad = torch.ones_like(p)
            p.requires_grad_(k not in off)
        y = bb._C.embed_layer_norm(ids, *ps, 1e-12, accumulate)
        torch.manual_seed(2)
        y.backward(torch.randn(y.shape, device="cuda").bfloat16())
        grads.append([p.grad for p in ps])
    for k, (a, b) in enumerate(zip(*grads)):
        assert not torch.equal(a, torch.ones_like(a))
        assert torch.equal(b, torch.ones_like(a) if k in frozen else a), k


def test_parameters_used_twice_in_a_graph_get_the_gradients_of_the_ordinary_path():
    """Autograd adds the uses' gradients first and accumulates once: with a `.grad` far above them in size, adding each by
    itself would round differently."""
    import bagua_core_b200 as bb

    g = torch.Generator().manual_seed(3)
    ids = torch.randint(0, 40, (2, 30), generator=g).cuda()
    x = torch.randn(60, 64, generator=g).bfloat16().cuda()
    grads = []
    for accumulate in (False, True):
        torch.manual_seed(0)
        ps = [torch.randn(*s, device="cuda", requires_grad=True) for s in ((40, 64), (30, 64), (1, 64), (64,), (64,), (64, 64), (64, 64))]
        tok, pos, typ, gamma, beta, w1, w2 = ps
        for p in ps:
            p.grad = torch.full_like(p, 1e5) + torch.rand_like(p)
        ys = [bb._C.embed_layer_norm(i, tok, pos, typ, gamma, beta, 1e-5, accumulate) for i in (ids, ids.flip(0))]
        ys += [bb._C.add_layer_norm(x, None, gamma, beta, 1e-5, accumulate), bb._C.add_layer_norm(x * 2, None, gamma, beta, 1e-5, accumulate)]
        ys += [bb._C.linear(x, w, beta, None, accumulate, a) for w, a in ((w1, 0), (w2, 2))]  # one bias for two layers
        sum((k + 1) * y.float().square().sum() for k, y in enumerate(ys)).backward()
        grads.append([p.grad for p in (tok, pos, typ, gamma, beta)])
    for a, b in zip(*grads):
        assert torch.equal(a, b)


def _second_order(f, inputs, seed):
    """Gradients of a sum of squared gradients, with respect to the inputs and to the first gradient's own input."""
    y = f(*inputs)
    g = torch.Generator().manual_seed(seed)
    dy = torch.randn(y.shape, generator=g).to(y).requires_grad_()
    first = torch.autograd.grad(y, inputs, dy, create_graph=True)
    penalty = sum(t.float().square().sum() for t in first)
    return list(first) + list(torch.autograd.grad(penalty, list(inputs) + [dy], allow_unused=True))


def test_gradients_of_gradients_are_those_of_the_plain_composition():
    import bagua_core_b200 as bb

    C, F = bb._C, torch.nn.functional
    torch.manual_seed(0)

    def rnd(*s, bf16=False):
        t = torch.randn(*s, device="cuda")
        return (t.bfloat16() if bf16 else t).requires_grad_()

    ids, span = torch.randint(0, 30, (2, 12)).cuda(), torch.randint(0, 12, (2, 3)).cuda()
    b16 = lambda t: t.bfloat16()  # noqa: E731
    acts = {0: lambda t: t, 1: F.gelu, 2: F.relu}
    cases = []
    for act in (0, 1, 2):
        for bf16 in (False, True):
            cases.append((lambda x, w, b, a=act: C.linear(x, w, b, None, True, a),
                          lambda x, w, b, a=act: acts[a](F.linear(b16(x), b16(w), b16(b))), [rnd(2, 9, 16, bf16=bf16), rnd(24, 16), rnd(24)]))
    for pool in (False, True):
        cases.append((lambda x, w, b, p=pool: C.conv_bias_relu(x, w, b, [1, 1], [1, 1], [1, 1], 1, p, None, True),
                      lambda x, w, b, p=pool: (lambda y: F.max_pool2d(y, 2, 2) if p else y)(F.relu(F.conv2d(x, w, b, padding=1))),
                      [rnd(2, 8, 6, 6, bf16=True), rnd(16, 8, 3, 3, bf16=True), rnd(16, bf16=True)]))
    cases.append((lambda x, r, g, b: C.add_layer_norm(x, r, g, b, 1e-5, True),
                  lambda x, r, g, b: F.layer_norm(x + r, (64,), b16(g), b16(b), 1e-5),
                  [rnd(5, 64, bf16=True), rnd(5, 64, bf16=True), rnd(64), rnd(64)]))
    cases.append((lambda *t: C.embed_layer_norm(ids, *t, 1e-5, True),
                  lambda t, p, y, g, b: b16(F.layer_norm(F.embedding(ids, t) + p[:12][None] + y[0][None, None], (64,), g, b, 1e-5)),
                  [rnd(30, 64), rnd(20, 64), rnd(2, 64), rnd(64), rnd(64)]))
    cases.append((lambda x: C.span_loss(x, span[0], span[1]),
                  lambda x: (F.cross_entropy(x.float()[..., 0], span[0]) + F.cross_entropy(x.float()[..., 1], span[1])) / 2,
                  [rnd(3, 12, 2, bf16=True)]))

    def heads(x):
        q, k, v = x.view(2, 16, 3, 2, 16).permute(2, 0, 3, 1, 4)
        return F.scaled_dot_product_attention(q, k, v).transpose(1, 2).reshape(2, 16, 32)

    cases.append((lambda x: C.attention(x, 2, 0.0), heads, [rnd(2, 16, 96, bf16=True)]))
    with torch.nn.attention.sdpa_kernel(torch.nn.attention.SDPBackend.MATH):  # the one whose backward is differentiable
        for n, (f, ref, inputs) in enumerate(cases):
            for p in inputs:
                p.grad = torch.zeros_like(p)
            for k, (a, b) in enumerate(zip(_second_order(f, inputs, n), _second_order(ref, inputs, n))):
                assert (a is None) == (b is None), (n, k)
                if a is not None:  # bf16 in each of a few steps
                    assert (a.double() - b.double()).norm() <= 3e-2 * b.double().norm() + 1e-6, (n, k)
            assert all(bool((p.grad == 0).all()) for p in inputs)


def test_gradients_that_are_asked_for_are_returned_and_not_added():
    import bagua_core_b200 as bb

    g = torch.Generator().manual_seed(3)
    ids = torch.randint(0, 40, (2, 30), generator=g).cuda()
    x = torch.randn(60, 64, generator=g).bfloat16().cuda()
    image = torch.randn(2, 3, 8, 8, generator=g).bfloat16().cuda().contiguous(memory_format=torch.channels_last)
    cases = [(lambda *p: bb._C.embed_layer_norm(ids, *p, 1e-5, True), [(40, 64), (30, 64), (1, 64), (64,), (64,)]),
             (lambda *p: bb._C.add_layer_norm(x, None, *p, 1e-5, True), [(64,), (64,)]),
             (lambda *p: bb._C.linear(x, *p, None, True), [(24, 64), (24,)]),
             (lambda *p: bb._C.linear(x, *p, None, True, 1), [(24, 64), (24,)]),
             (lambda *p: bb._C.conv_bias_relu(image, p[0].bfloat16().contiguous(memory_format=torch.channels_last), p[1].bfloat16(),
                                              [1, 1], [1, 1], [1, 1], 1, True, None, True), [(64, 3, 3, 3), (64,)])]
    for f, shapes in cases:
        ps = [torch.randn(*s, generator=g).cuda().requires_grad_() for s in shapes]
        for p in ps:
            p.grad = torch.zeros_like(p)
        dy = torch.randn_like(f(*ps))
        got = torch.autograd.grad(f(*ps), ps, dy)
        assert all(bool((p.grad == 0).all()) for p in ps)
        f(*ps).backward(dy)
        for p, q in zip(ps, got):  # rounded to bf16 on the way where the gradient is handed over
            assert q.norm() > 0 and (p.grad - q).norm() <= 1e-2 * q.norm()


def test_forward_mode_derivatives_are_those_of_the_plain_composition():
    import torch.autograd.forward_ad as fwad

    import bagua_core_b200 as bb

    C, F = bb._C, torch.nn.functional
    torch.manual_seed(0)
    ids, span = torch.randint(0, 30, (2, 12)).cuda(), torch.randint(0, 12, (2, 3)).cuda()
    b16 = lambda t: t.bfloat16()  # noqa: E731
    cases = [(lambda x, w, b: C.linear(x, w, b, None, True, 1), lambda x, w, b: F.gelu(F.linear(b16(x), b16(w), b16(b))),
              [torch.randn(9, 16), torch.randn(24, 16), torch.randn(24)]),
             (lambda x, r, g, b: C.add_layer_norm(x, r, g, b, 1e-5, True), lambda x, r, g, b: F.layer_norm(x + r, (64,), b16(g), b16(b), 1e-5),
              [b16(torch.randn(5, 64)), b16(torch.randn(5, 64)), torch.randn(64), torch.randn(64)]),
             (lambda *t: C.embed_layer_norm(ids, *t, 1e-5, True),
              lambda t, p, y, g, b: b16(F.layer_norm(F.embedding(ids, t) + p[:12][None] + y[0][None, None], (64,), g, b, 1e-5)),
              [torch.randn(30, 64), torch.randn(20, 64), torch.randn(2, 64), torch.randn(64), torch.randn(64)]),
             (lambda x: C.span_loss(x, span[0], span[1]),
              lambda x: (F.cross_entropy(x.float()[..., 0], span[0]) + F.cross_entropy(x.float()[..., 1], span[1])) / 2,
              [b16(torch.randn(3, 12, 2))])]
    for n, (f, ref, inputs) in enumerate(cases):
        inputs = [t.cuda().requires_grad_() for t in inputs]
        got = []
        for g in (f, ref):
            with fwad.dual_level():
                torch.manual_seed(n)
                got.append(fwad.unpack_dual(g(*[fwad.make_dual(t, torch.randn_like(t)) for t in inputs])).tangent)
        assert (got[0].double() - got[1].double()).norm() <= 2e-2 * got[1].double().norm(), n


def test_hooks_and_replaced_modules_of_the_encoder_are_respected():
    import torch.nn as nn

    from bagua_core_b200.models import BertConfig, BertForQuestionAnswering

    torch.manual_seed(4)
    net = BertForQuestionAnswering(BertConfig(vocab_size=500, hidden=128, layers=2, heads=4, ffn=256, dropout=0.0)).cuda()
    ids, span = torch.randint(0, 500, (3, 40)).cuda(), torch.randint(0, 40, (3, 2)).cuda()

    def loss():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return net(ids, span[:, 0], span[:, 1])

    fused = loss()
    seen, handles = {}, []
    for name, module in net.named_modules():
        if name and name not in ("typ", "layers"):  # its first row is read, it is not called; a list
            handles.append(module.register_forward_hook(lambda m, a, o, name=name: seen.__setitem__(name, (a[0], o))))
    plain = loss()
    assert set(seen) == {n for n, _ in net.named_modules() if n and n not in ("typ", "layers")}
    assert torch.allclose(fused, plain, rtol=1e-5)
    assert bool((seen["layers.0.fc1"][1] < -0.2).any())  # what GELU is applied to, and GELU's values are above that
    for h in handles:
        h.remove()
    assert torch.equal(loss(), fused)
    for name in ("tok", "pos", "ln", "layers.0.ln1", "layers.1.ln2", "layers.0.fc1", "layers.1.drop", "qa"):  # one alone
        seen.clear()
        h = net.get_submodule(name).register_forward_hook(lambda m, a, o: seen.__setitem__("out", o))
        assert torch.allclose(loss(), fused, rtol=1e-5) and seen, name
        h.remove()
    inner = net.qa
    net.qa = nn.Sequential(inner, nn.Identity())
    assert torch.allclose(loss(), fused, rtol=1e-5)
    net.qa = inner
    net.layers[0].drop.p = 0.9  # dropout switched on behind the configuration's back
    assert not torch.allclose(loss(), fused, rtol=1e-3)
    net.layers[0].drop.p = 0.0
    net.tok = nn.Embedding.from_pretrained(net.tok.weight.detach(), freeze=False, padding_idx=int(ids[0, 0]))
    loss().backward()
    assert bool((net.tok.weight.grad[ids[0, 0]] == 0).all())


@pytest.mark.parametrize("bad", ["token", "negative token", "start", "end"])
def test_an_index_outside_its_table_is_an_error(bad):
    """The kernels skip it; the first look of the host behind it says so, and the call after that works again."""
    from bagua_core_b200.models import BertConfig, BertForQuestionAnswering

    net = BertForQuestionAnswering(BertConfig.tiny()).cuda().eval()
    good, span = torch.randint(0, 1000, (2, 16)).cuda(), torch.randint(0, 16, (2, 2)).cuda()
    ids, where = good.clone(), span.clone()
    if bad.endswith("token"):
        ids[1, 3] = 1000 if bad == "token" else -1
    else:
        where[0, int(bad == "end")] = 16

    def loss(i, w):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return net(i, w[:, 0], w[:, 1])

    want = loss(good, span)
    with pytest.raises(RuntimeError, match="which is not in the"):
        assert torch.isnan(loss(ids, where))  # (waits for it, unless it has been noticed already)
        loss(good, span)
    assert torch.equal(loss(good, span), want)
    where[:, 0] = -100  # counts for nothing, and is no error
    loss(good, torch.where(where == 16, 0, where))
    torch.cuda.synchronize()
    assert torch.equal(loss(good, span), want)


def test_linear_follows_the_frameworks_switch_for_partial_sums():
    """The rows are few and k is long, so the library splits k: with the switch off no partial sum is rounded to bf16."""
    import bagua_core_b200 as bb

    settings, saved = torch.backends.cuda.matmul, torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction
    try:
        for M, K, N in ((32, 25088, 4096), (5, 30000, 128), (64, 128, 128), (384, 1024, 4096)):
            torch.manual_seed(K)
            x, w = torch.randn(M, K, device="cuda").bfloat16().requires_grad_(), torch.randn(N, K, device="cuda").bfloat16()
            b = torch.randn(N, device="cuda").bfloat16()
            for allow in (True, False, True):
                settings.allow_bf16_reduced_precision_reduction = allow
                y, ref = bb._C.linear(x, w, b, None, False), torch.nn.functional.linear(x, w, b)
                assert torch.equal(y, ref), (M, K, N, allow)
                dy = torch.randn_like(y)
                (dx,) = torch.autograd.grad(y, x, dy)
                exact = dy.double() @ w.double()
                if not allow:  # one rounding of the result, and fp32 sums
                    assert ((dx.double() - exact).abs() <= 2 ** -8 * exact.abs() + 1e-4 * exact.abs().max()).all()
    finally:
        settings.allow_bf16_reduced_precision_reduction = saved


@pytest.mark.parametrize("batch,seq,V,same", [(16, 512, 30522, 0), (16, 512, 1000, 6000), (16, 384, 50, 0)])
def test_embedding_at_the_largest_batches_of_its_range(batch, seq, V, same):
    test_embedding_sum_and_norm_match_the_plain_composition(batch, seq, V, same)


@pytest.mark.parametrize("hidden", [1032, 1536])
def test_encoders_wider_than_1024_run_fused_and_agree_with_the_plain_composition(hidden):
    from bagua_core_b200.models import BertConfig, BertForQuestionAnswering, bert

    torch.manual_seed(4)
    net = BertForQuestionAnswering(BertConfig(vocab_size=300, hidden=hidden, layers=1, heads=3 if hidden % 24 == 0 and hidden < 1100 else 12,
                                              ffn=264, dropout=0.0)).cuda()
    ids, span = torch.randint(0, 300, (2, 40)).cuda(), torch.randint(0, 40, (2, 2)).cuda()
    out, saved = [], bert._fused
    try:
        for fused in (True, False):
            if not fused:
                bert._fused = lambda x, ln: False
            net.zero_grad()
            before = bb_launches()
            with torch.autocast("cuda", dtype=torch.bfloat16):
                loss = net(ids, span[:, 0], span[:, 1])
            assert not fused or bb_launches() - before >= 6  # embedding, two normalisations' casts, GELU, output layer, loss
            loss.backward()
            out.append((loss.detach(), torch.cat([p.grad.flatten() for p in net.parameters()])))
    finally:
        bert._fused = saved
    (la, ga), (lb, gb) = out
    assert torch.allclose(la, lb, rtol=1e-5)
    assert (ga - gb).norm() <= 1e-2 * gb.norm()


@pytest.mark.parametrize("batch,seq,hidden,heads,layers", [(2, 33, 128, 4, 2), (8, 384, 1024, 16, 2)])
def test_the_fused_encoder_has_the_bits_of_the_plain_composition(batch, seq, hidden, heads, layers):
    """From the ids to the logits every operation rounds where the framework's rounds; the loss, whose sums over rows and
    positions are taken in another order, agrees to fp32 rounding."""
    from bagua_core_b200.models import BertConfig, BertForQuestionAnswering, bert
    from bagua_core_b200.ops import wgrad as W

    torch.manual_seed(2)
    net = BertForQuestionAnswering(BertConfig(vocab_size=3000, hidden=hidden, heads=heads, ffn=4 * hidden, layers=layers, dropout=0.0)).cuda()
    ids, span = torch.randint(0, 3000, (batch, seq)).cuda(), torch.randint(0, seq, (batch, 2)).cuda()
    saved, out = (bert._fused, W.enabled), []
    try:
        for mode in ("plain", "fused", "fused, in place"):
            bert._fused = (lambda x, ln: False) if mode == "plain" else saved[0]
            W.enabled = mode.endswith("in place")
            with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
                out.append((*net(ids), net(ids, span[:, 0], span[:, 1])))
    finally:
        bert._fused, W.enabled = saved
    plain_loss = (torch.nn.functional.cross_entropy(out[0][0], span[:, 0]) + torch.nn.functional.cross_entropy(out[0][1], span[:, 1])) / 2
    for start, end, loss in out[1:]:
        assert torch.equal(start, out[0][0]) and torch.equal(end, out[0][1])
        assert torch.allclose(loss, plain_loss, rtol=1e-6, atol=0)
