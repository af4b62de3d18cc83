"""Single-GPU end-to-end: the flagship training step through `with_bagua` (world size 1)
and the engine scheduler driving GPU buckets with CUDA events."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_smoke_entry():
    import __graft_entry__ as g

    g.smoke()


def test_scheduler_with_cuda_events_single_rank():
    import bagua_core as bc

    dev = torch.device("cuda", 0)
    stream = torch.cuda.Stream()
    uid = bc.BaguaSingleCommunicatorPy.generate_nccl_unique_id_str()
    comm = bc.BaguaSingleCommunicatorPy(0, 1, 0, stream.cuda_stream, uid)
    backend = bc.BaguaCommBackendPy(10, 0)
    flat = torch.randn(3 * 4096, device=dev)
    views = [flat[i * 4096:(i + 1) * 4096] for i in range(3)]
    ts = [bc.BaguaTensorPy(v, f"t{i}") for i, v in enumerate(views)]
    bucket = bc.BaguaBucketPy("b", ts)
    bucket.append_centralized_synchronous_op(comm, None, hierarchical=False, average=True, scattergather=True,
                                             compression="MinMaxUInt8")
    backend.register_ordered_buckets([bucket])
    orig = flat.clone()
    events = []  # the engine borrows the handles: keep the events alive until the wait returns
    for t in ts:
        ev = torch.cuda.Event()
        ev.record()
        events.append(ev)
        backend.mark_communication_ready(t, ev.cuda_event)
    assert backend.wait_pending_comm_ops() == 1
    torch.cuda.current_stream().wait_stream(stream)
    torch.cuda.synchronize()
    # one rank: ByteGrad = quantise/dequantise twice
    assert (flat - orig).abs().max() <= 2 * (orig.max() - orig.min()) / 255
    backend.close()


def test_bert_trains_with_a_bf16_residual_stream():
    """A two-layer BERT through `with_bagua` with ByteGrad under bf16 autocast: the encoder's LayerNorms
    take and return bf16 (statistics in fp32 inside the library kernel), so every projection sees a
    bf16 input; losses stay finite and close to the model with stock fp32-in/fp32-out LayerNorms."""
    import copy
    import os

    import bagua_core_b200.parallel as P
    from bagua_core_b200.models import BertConfig, BertForQuestionAnswering

    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    os.environ.setdefault("MASTER_PORT", "29547")
    dev = torch.device("cuda", 0)
    losses = []
    for stock in (False, True):
        torch.manual_seed(0)
        cfg = BertConfig.tiny()
        cfg.dropout = 0.0
        cfg = copy.copy(cfg)
        cfg.fp32_layernorm_io = stock
        model = BertForQuestionAnswering(cfg).to(dev)
        seen = []
        model.layers[1].qkv.register_forward_hook(lambda m, i, o: seen.append(i[0].dtype))
        P.init_process_group(dev)
        opt = P.FlatSGD(model.parameters(), lr=0.05, momentum=0.9)
        bm = P.with_bagua(model, [opt], P.ByteGradAlgorithm(), bucket_bytes=64 << 10)
        g = torch.Generator().manual_seed(3)
        run = []
        for _ in range(4):
            ids = torch.randint(0, cfg.vocab_size, (4, 32), generator=g).to(dev)
            span = torch.randint(0, 32, (4, 2), generator=g).to(dev)
            opt.zero_grad()
            with torch.autocast("cuda", dtype=torch.bfloat16):
                loss = bm(ids, span[:, 0], span[:, 1])
            loss.backward()
            opt.step()
            run.append(loss.item())
        torch.cuda.synchronize()
        P.destroy_process_group()
        assert all(d == (torch.float32 if stock else torch.bfloat16) for d in seen), seen
        assert all(torch.isfinite(torch.tensor(run)))
        losses.append(run)
    assert all(abs(a - b) < 5e-2 for a, b in zip(*losses)), losses


@pytest.mark.parametrize("early_graph", [False, True])
def test_training_on_a_side_stream_equals_training_on_the_default_stream(early_graph):
    """A model wrapped on the default stream, trained on a stream that lags behind the host: the buckets wait for gradients
    that were added to them there.  `early_graph`: a graph from before the wrapping keeps one layer's accumulation nodes
    on a third stream."""
    import os

    import bagua_core_b200.parallel as P
    from bagua_core_b200.ops import wgrad as W
    from bagua_core_b200.ops.fused_conv import ConvBiasReLU, ConvBiasReLUPool
    from bagua_core_b200.ops.fused_linear import ShadowLinear

    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    os.environ.setdefault("MASTER_PORT", "29549")
    dev = torch.device("cuda", 0)
    saved, results = W.enabled, []
    W.enabled = True
    try:
        for side in (False, True):
            torch.manual_seed(0)
            conv = torch.nn.Sequential(ConvBiasReLU(3, 64, 3, padding=1), ConvBiasReLUPool(64, 64, 3, padding=1), torch.nn.Flatten())
            head = torch.nn.Sequential(ShadowLinear(64 * 16, 64), torch.nn.ReLU(), ShadowLinear(64, 16))
            net = torch.nn.Sequential(conv, head).to(dev).to(memory_format=torch.channels_last)
            third = torch.cuda.Stream()
            with torch.cuda.stream(third):
                keep = head[0](torch.zeros(1, 64 * 16, device=dev)) if early_graph else None
            third.synchronize()
            P.init_process_group(dev)
            opt = P.FlatSGD(net.parameters(), lr=0.05, momentum=0.9)
            bm = P.with_bagua(net, [opt], P.ByteGradAlgorithm(), bucket_bytes=64 << 10)
            x = torch.randn(8, 3, 8, 8, device=dev).contiguous(memory_format=torch.channels_last)
            stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
            stream.wait_stream(torch.cuda.current_stream())
            grads = []
            with torch.cuda.stream(stream):
                for _ in range(3):
                    opt.zero_grad()
                    torch.cuda._sleep(20_000_000)  # about 10 ms: the host is done with the step before the GPU begins it
                    with torch.autocast("cuda", dtype=torch.bfloat16):
                        loss = bm(x).float().square().sum()
                    loss.backward()
                    grads.append([b.flattened.clone() for b in bm.bagua_buckets])
                    opt.step()
            torch.cuda.synchronize()
            results.append((grads, [p.detach().clone() for p in net.parameters()]))
            P.destroy_process_group()
            del keep
    finally:
        W.enabled = saved
    (ga, wa), (gb, wb) = results
    for a, b in zip(sum(ga, []) + wa, sum(gb, []) + wb):
        assert torch.equal(a, b)


@pytest.mark.parametrize("sizes", [[5], [4096, 4097], [1, 70001, 3, 4095, 16384] * 9])
def test_zero_grad_clears_every_bucket_and_nothing_else(sizes):
    """One buffer, and more of them than a launch takes, with tiles that end in the middle."""
    import bagua_core_b200.parallel as P

    m = torch.nn.Module()
    for i, n in enumerate(sizes):
        m.register_parameter("w%d" % i, torch.nn.Parameter(torch.full((n,), float(i), device="cuda")))
    opt = P.FlatSGD(m.parameters(), lr=0.5)
    bagua = P.with_bagua(m, [opt], P.GradientAllReduceAlgorithm(), process_group=P.init_process_group(torch.device("cuda", 0)), bucket_bytes=4)
    assert len(bagua.bagua_buckets) == len(sizes)
    for b in bagua.bagua_buckets:
        b.flattened.fill_(7)
    opt.zero_grad(set_to_none=False)
    for b in bagua.bagua_buckets:
        assert not b.flattened.any()
    opt.step()
    for i, p in enumerate(m.parameters()):
        assert (p == i).all() and not p.grad.any()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs a second GPU")
def test_zero_grad_works_on_the_device_of_its_buckets():
    import bagua_core_b200 as bb

    plan, grads = bb._C.SgdPlan(), []
    for _ in range(3):
        p, g, m = (torch.ones(5000, device="cuda:1") for _ in range(3))
        plan.add(p, g, m, None, 0)
        grads.append(g)
    torch.cuda.synchronize(1)
    with torch.cuda.device(0):
        plan.zero_grad(torch.cuda.current_stream(1).cuda_stream)
    torch.cuda.synchronize(1)
    assert not any(g.any() for g in grads)
