"""CPU tests of the host-side mirror: configuration validation, schedules, graph recording.  They read
like the reference's unit tests (cited) and need no GPU."""
import numpy as np
import pytest
import torch

from metal_candle_b200.graph import ComputationGraph, GraphNode, LazyTensor, NodeId, Operation
from metal_candle_b200.training import (AdamW, AdamWConfig, InvalidConfig, LoRAAdapterConfig, LoRAConfig, LRScheduler,
                                        TargetModule, TrainingConfig, TrainingStep)
from oracle import reference_ops as R


def test_lora_config_defaults_and_validation():
    # src/training/lora.rs:70-121
    c = LoRAConfig()
    assert (c.rank, c.alpha, c.dropout) == (8, 16.0, 0.0) and c.scaling() == 2.0
    for bad, msg in ((LoRAConfig(rank=0), "LoRA rank must be greater than 0"),
                     (LoRAConfig(alpha=0.0), "LoRA alpha must be positive"),
                     (LoRAConfig(dropout=1.0), r"LoRA dropout must be in \[0, 1\)")):
        with pytest.raises(InvalidConfig, match=msg):
            bad.validate()


def test_adapter_config_and_target_modules():
    # src/training/adapter.rs:33-62,96-124
    c = LoRAAdapterConfig()
    assert c.target_modules == [TargetModule.QProj, TargetModule.VProj]
    assert c.is_target(TargetModule.QProj) and not c.is_target(TargetModule.OProj)
    assert TargetModule.from_name("down_proj") is TargetModule.DownProj and TargetModule.from_name("nope") is None
    assert [m.value for m in TargetModule] == ["q_proj", "k_proj", "v_proj", "o_proj", "gate_proj", "up_proj", "down_proj"]
    assert c.to_lora_config().scaling() == 2.0


def test_adamw_config_validation():
    # src/training/optimizer.rs:51-107
    c = AdamWConfig()
    assert (c.learning_rate, c.beta1, c.beta2, c.epsilon, c.weight_decay) == (1e-4, 0.9, 0.999, 1e-8, 0.01)
    for kw, msg in ((dict(learning_rate=0.0), "learning rate must be positive"), (dict(beta1=1.0), "beta1 must be in"),
                    (dict(beta2=-0.1), "beta2 must be in"), (dict(epsilon=0.0), "epsilon must be positive"),
                    (dict(weight_decay=-1.0), "weight decay must be non-negative")):
        with pytest.raises(InvalidConfig, match=msg):
            AdamW(AdamWConfig(**kw))
    opt = AdamW()
    opt.set_lr(3e-4)
    assert opt.learning_rate() == 3e-4 and opt.step_count == 0
    with pytest.raises(Exception, match="not found in optimizer"):
        opt.step("missing", torch.zeros(2), torch.zeros(2))


def test_schedulers_match_oracle_and_reference_values():
    # src/training/scheduler.rs:312-373,401-419
    s = LRScheduler.linear(1000, 1e-3)
    assert s.get_lr(0) == 0.0 and abs(s.get_lr(500) - 5e-4) < 1e-7 and abs(s.get_lr(2000) - 1e-3) < 1e-9
    wc = LRScheduler.warmup_cosine(1000, 10_000, 1e-3, 1e-5)
    co = LRScheduler.cosine(10_000, 1e-3, 1e-5)
    for step in (0, 1, 499, 1000, 1001, 5000, 9999, 10_000, 20_000):
        assert wc.get_lr(step) == float(R.lr_warmup_cosine(step, 1000, 10_000, 1e-3, 1e-5))
        assert co.get_lr(step) == float(R.lr_cosine(step, 10_000, 1e-3, 1e-5))
    assert LRScheduler.constant(1e-4).get_lr(77) == float(np.float32(1e-4))
    LRScheduler.constant(1e-4).validate()
    for bad in (LRScheduler.constant(0.0), LRScheduler.linear(0, 1e-3), LRScheduler.cosine(0, 1e-3, 1e-5),
                LRScheduler.cosine(10, 1e-3, 1e-2), LRScheduler.warmup_cosine(10, 10, 1e-3, 1e-5)):
        with pytest.raises(InvalidConfig):
            bad.validate()


def test_training_config_defaults():
    # src/training/trainer.rs:30-39
    c = TrainingConfig()
    assert c.num_epochs == 3 and c.max_grad_norm == 1.0 and c.lr_scheduler.get_lr(5) == float(np.float32(1e-4))
    st = TrainingStep()
    assert st.step() == 0
    st.reset()
    assert st.step() == 0


def test_operation_names_shapes_and_arity_errors():
    # src/graph/operation.rs:53-166
    assert [Operation.Input().name(), Operation.Matmul().name(), Operation.Add().name(), Operation.Mul().name(),
            Operation.MulScalar(2.0).name(), Operation.LoRA(NodeId(1), NodeId(2), 2.0).name(),
            Operation.Softmax(1).name(), Operation.RMSNorm(1e-5).name()] == \
        ["input", "matmul", "add", "mul", "mul_scalar", "lora", "softmax", "rms_norm"]
    assert Operation.Matmul().output_shape([(2, 3), (3, 4)]) == (2, 4)
    assert Operation.Matmul().output_shape([(5, 2, 3), (3, 4)]) == (5, 2, 4)
    with pytest.raises(ValueError, match="Matmul requires 2 inputs, got 1"):
        Operation.Matmul().output_shape([(2, 3)])
    with pytest.raises(ValueError, match="Matmul dimension mismatch: 2×3 @ 4×5"):
        Operation.Matmul().output_shape([(2, 3), (4, 5)])
    with pytest.raises(ValueError, match="Matmul requires at least 2D tensors"):
        Operation.Matmul().output_shape([(3,), (3, 4)])
    with pytest.raises(ValueError, match="add requires 2 inputs, got 3"):
        Operation.Add().output_shape([(1,), (1,), (1,)])
    with pytest.raises(ValueError, match="Shape mismatch"):
        Operation.Mul().output_shape([(2, 2), (2, 3)])
    with pytest.raises(ValueError, match=r"LoRA requires 3 inputs \(input, a, b\), got 2"):
        Operation.LoRA(NodeId(0), NodeId(1), 1.0).output_shape([(2, 4), (4, 2)])
    # out_features comes from B (the reference returns the input shape here, which is wrong when out != in)
    assert Operation.LoRA(NodeId(0), NodeId(1), 1.0).output_shape([(2, 5, 16), (16, 4), (4, 32)]) == (2, 5, 32)
    with pytest.raises(ValueError, match="softmax requires 1 input, got 2"):
        Operation.Softmax(0).output_shape([(2,), (2,)])
    assert Operation.Softmax(0).output_dtype([torch.bfloat16]) == torch.bfloat16


def test_graph_recording_order_and_merge():
    # src/graph/node.rs:358-565; tests/lazy_execution.rs (graph shapes known before eval)
    a = LazyTensor.from_tensor(torch.ones(2, 3))
    b = a.add_tensor_to_graph(torch.ones(3, 4))
    c = a.matmul(b).mul_scalar(2.0)
    assert c.shape() == (2, 4) and c.dtype() == torch.float32 and c.graph_size() == 4 and not c.is_evaluated()
    assert a.is_evaluated() and a.node_id() == NodeId(0) and repr(c.node_id()) == "NodeId(3)"
    g = c._graph
    assert g.topological_order(c.node_id()) == [NodeId(0), NodeId(1), NodeId(2), NodeId(3)]
    with pytest.raises(ValueError, match=r"Input node NodeId\(9\) not found"):
        g.add_node(Operation.Add(), [NodeId(0), NodeId(9)])
    # operands from another graph are copied in with remapped ids
    other = LazyTensor.from_tensor(torch.ones(2, 4)).mul_scalar(3.0)
    d = c.add(other)
    assert d.graph_size() == 4 + 2 + 1 and d.shape() == (2, 4)
    order = g.topological_order(d.node_id())
    assert order[-1] == d.node_id() and len(order) == 7
    # a diamond is visited once
    e = d.add(d)
    assert len(g.topological_order(e.node_id())) == 8
    # a cycle (only constructible by hand) is reported
    g2 = ComputationGraph("cpu")
    g2.nodes.append(GraphNode(NodeId(0), Operation.MulScalar(1.0), [NodeId(1)], (1,), torch.float32))
    g2.nodes.append(GraphNode(NodeId(1), Operation.MulScalar(1.0), [NodeId(0)], (1,), torch.float32))
    with pytest.raises(ValueError, match="Circular dependency detected at node"):
        g2.topological_order(NodeId(0))
    with pytest.raises(Exception, match="Shape mismatch"):
        a.add(b)


def test_from_slice_and_constructors():
    t = LazyTensor.from_slice([1.0, 2.0, 3.0, 4.0], (2, 2), "cpu")
    assert t.shape() == (2, 2) and t.is_evaluated()
    assert LazyTensor.zeros((3,), torch.float32, "cpu").shape() == (3,)
    assert LazyTensor.ones((3, 2), torch.float32, "cpu").graph_size() == 1
    with pytest.raises(Exception):
        LazyTensor.from_slice([1.0, 2.0], (3,), "cpu")


def test_oracle_dropout_mask_is_a_pure_function_of_seed_and_position():
    """The restated mask of mcb_dropout: keep rate 1 - p, a call at offset k continues the stream of a call at offset 0,
    different seeds give different masks, p = 0 keeps everything; the LoRA training-mode forward scales kept entries
    of x A by 1 / (1 - p) (src/training/lora.rs:325-330 applies candle_nn::ops::dropout to the same tensor)."""
    import numpy as np

    from oracle import reference_ops as R

    whole = R.dropout_mask(100_000, 0.3, 7, 0)
    assert abs(whole.mean() - 0.7) < 5e-3
    assert np.array_equal(R.dropout_mask(1000, 0.3, 7, 5000), whole[5000:6000])
    assert not np.array_equal(R.dropout_mask(1000, 0.3, 8, 0), whole[:1000])
    assert R.dropout_mask(1000, 0.0, 7, 0).all()
    x = np.ones((4, 3)); A = np.ones((3, 2)); B = np.ones((2, 5))
    y = R.lora_forward_dropout(x, A, B, 2.0, 0.5, 11, 0)
    keep = R.dropout_mask(8, 0.5, 11, 0).reshape(4, 2)
    assert np.allclose(y, (np.where(keep, 3.0 / 0.5, 0.0) @ B) * 2.0)


def test_scratch_belongs_to_one_thread_and_stream(monkeypatch):
    """A call's kernels write their scratch memory and read it back: no two streams and no two threads share it, a buffer
    that is outgrown is replaced for its own stream alone, and a capture takes none of them."""
    import threading

    from metal_candle_b200 import backend

    now = {"stream": 1, "capturing": False}
    monkeypatch.setattr(backend, "_stream", lambda: now["stream"])
    monkeypatch.setattr(torch._C, "_cuda_isCurrentStreamCapturing", lambda: now["capturing"])
    monkeypatch.setattr(backend, "_scratch", backend._Scratch())
    cpu = torch.device("cpu")
    a = backend.workspace(cpu, 100)
    assert a.data_ptr() % 1024 == 0 and a.numel() >= 1 << 20
    assert backend.workspace(cpu, 1 << 20) is a and backend.workspace_refs(cpu)[0] is a
    now["stream"] = 2
    assert backend.workspace_refs(cpu) == []
    b = backend.workspace(cpu, 100)
    assert b is not a
    big = backend.workspace(cpu, 3 << 20)
    assert big.numel() >= 3 << 20 and backend.workspace(cpu, 100) is big
    now["stream"] = 1
    assert backend.workspace(cpu, 100) is a
    other = []
    t = threading.Thread(target=lambda: other.append(backend.workspace(cpu, 100)))
    t.start()
    t.join()
    assert other[0] is not a and backend.workspace(cpu, 100) is a
    now["capturing"] = True
    c = backend.workspace(cpu, 100)
    assert c is not a and backend.workspace(cpu, 100) is not c
    now["capturing"] = False
    for s in range(3, 40):   # however many streams a program uses, a thread keeps a few buffers
        now["stream"] = s
        backend.workspace(cpu, 100)
    assert len(backend._scratch.buffers) <= backend._SCRATCH_STREAMS


class _LaunchLog:
    """Stands in for the library: notes the descriptors of each launch instead of making it."""

    def __init__(self):
        self.launches = []

    def mcb_adamw_multi(self, table, n, *rest):
        self.launches.append([(t.p, t.g, t.m, t.v, t.n, t.t) for t in table[:n]])
        return 0


@pytest.fixture
def launch_log(monkeypatch):
    from metal_candle_b200 import backend

    log = _LaunchLog()
    monkeypatch.setattr(backend, "_lib_for", lambda t: log if torch.is_tensor(t) else None)
    monkeypatch.setattr(backend, "_stream", lambda: 0)
    monkeypatch.setattr(backend, "_require_cuda", lambda *t: None)
    return log


def test_adamw_moments_belong_to_the_elements(launch_log):
    """A flat buffer and the view of its first elements start at one address: their moments are not the same, and neither
    is read or written past its end."""
    flat = torch.zeros(100)
    first = flat[:10]
    opt = AdamW(AdamWConfig())
    for order in ([first, flat], [flat, first], [flat[:10].view(2, 5)]):
        opt.step_vars(order, [torch.ones_like(t) for t in order])
        for (p, _, m, v, n, _), t in zip(launch_log.launches[-1], order):
            em, ev = opt.state_of(t)
            assert p == flat.data_ptr() and n == t.numel() == em.numel() == ev.numel() and (m, v) == (em.data_ptr(), ev.data_ptr())
    assert len(opt.state) == 2
    opt.step_var(flat, torch.ones(100))
    assert launch_log.launches[-1][0][4] == 100 and opt.step_count == 6


def test_adamw_refuses_moments_of_another_size(launch_log):
    from metal_candle_b200.training import StateError

    opt, p = AdamW(AdamWConfig()), torch.zeros(8)
    opt.add_parameter("w", torch.zeros(4))
    with pytest.raises(StateError):
        opt.step("w", p, torch.zeros(8))
    opt.step_vars([p], [torch.zeros(8)])
    opt.state[opt._key(p)] = (torch.zeros(8), torch.zeros(7))
    with pytest.raises(StateError):
        opt.step_vars([p], [torch.zeros(8)])
    assert len(launch_log.launches) == 1


def test_adamw_state_is_not_inherited_through_a_reused_address(launch_log):
    """While moments are kept, so is the memory they are known by: a later tensor cannot lie at the same address."""
    opt = AdamW(AdamWConfig())
    seen = set()
    for _ in range(50):
        p = torch.zeros(1000)
        assert p.data_ptr() not in seen
        seen.add(p.data_ptr())
        opt.step_vars([p], [torch.ones(1000)])
        del p
    assert len(opt.state) == 50
    opt.zero_state()
    assert opt.state == {} and opt._held == {}


class _OnDevice(torch.Tensor):
    """A CPU tensor that says it is on the GPU."""

    is_cuda = property(lambda self: True)


def _layer_model():
    """One layer with q and v adapters and nothing behind it but shapes: `prepare` launches nothing."""
    from types import SimpleNamespace

    from metal_candle_b200 import _lib
    from metal_candle_b200.qwen import ModelConfig, Qwen

    def dev(*shape, dtype=torch.bfloat16):
        return torch.zeros(*shape, dtype=dtype).as_subclass(_OnDevice)

    cfg = ModelConfig(vocab_size=320, hidden_size=256, intermediate_size=384, num_hidden_layers=1, num_attention_heads=4,
                      num_key_value_heads=2, max_position_embeddings=256, rms_norm_eps=1e-6, rope_theta=1.0e6)
    m = Qwen.__new__(Qwen)
    m.config, m.dtype, m.device, m.lib = cfg, torch.bfloat16, torch.device("cpu"), _lib.load()
    m.fuse_qkv = m.fuse_swiglu_bwd = True
    L = {"input_layernorm": dev(256), "post_attention_layernorm": dev(256)}
    for name, out, inp in (("q_proj", 256, 256), ("k_proj", 128, 256), ("v_proj", 128, 256), ("o_proj", 256, 256), ("gate_proj", 384, 256),
                           ("up_proj", 384, 256), ("down_proj", 256, 384)):
        lora = None
        if name in ("q_proj", "v_proj"):
            lora = SimpleNamespace(lora_a=dev(inp, 4, dtype=torch.float32), lora_b=dev(4, out, dtype=torch.float32), config=LoRAConfig(rank=4))
        L[name] = SimpleNamespace(weight=dev(out, inp), weight_t=dev(inp, out), bias=dev(out) if name in ("q_proj", "k_proj", "v_proj") else None,
                                  lora=lora, in_f=inp, out_f=out)
    m.layers, m._on_device = [L], dev
    return m, L


def _wrong_norm(m, L):
    L["input_layernorm"] = torch.ones(256, dtype=torch.bfloat16)


def _wrong_second_norm(m, L):
    L["post_attention_layernorm"] = torch.ones(256, dtype=torch.bfloat16)


def _wrong_biases(m, L):
    for name in ("q_proj", "k_proj", "v_proj"):
        L[name].bias = torch.zeros(L[name].out_f, dtype=torch.bfloat16)


def _float32_biases(m, L):
    for name in ("q_proj", "k_proj", "v_proj"):
        L[name].bias = m._on_device(L[name].out_f, dtype=torch.float32)


def _short_bias(m, L):
    L["q_proj"].bias = m._on_device(8)


def _narrow_qkv(m, L):
    for name in ("q_proj", "k_proj", "v_proj"):
        L[name].weight = m._on_device(L[name].out_f, 128)


def _shifted_qkv(m, L):
    for name, out in (("q_proj", 128), ("k_proj", 256)):
        L[name].weight, L[name].out_f = m._on_device(out, 256), out
    L["q_proj"].lora.lora_b = m._on_device(4, 128, dtype=torch.float32)


def _narrow_mlp(m, L):
    for name in ("gate_proj", "up_proj"):
        L[name].weight, L[name].weight_t, L[name].out_f = m._on_device(256, 256), m._on_device(256, 256), 256


# A layer goes to the library as addresses: whatever the calls per kernel refuse or read by its own shape has to stay with them.
@pytest.mark.parametrize("spoil", [None, _wrong_norm, _wrong_second_norm, _wrong_biases, _float32_biases, _short_bias, _narrow_qkv, _shifted_qkv,
                                   _narrow_mlp], ids=lambda f: f.__name__ if f else "sound")
def test_layer_call_takes_only_tensors_of_the_layers_own_shape_and_device(monkeypatch, spoil):
    from metal_candle_b200 import backend
    from metal_candle_b200.qwen import _LayerCalls

    monkeypatch.setattr(backend, "transpose_2d", lambda w: w.t().contiguous())
    monkeypatch.setattr(backend, "interleave_gate_up", lambda g, u: torch.cat([g, u], 0))
    m, L = _layer_model()
    if spoil is not None:
        spoil(m, L)
    calls = _LayerCalls(m, 1, 16, backward=False)
    prepared = calls.prepare(0)
    assert (prepared is None) == (spoil is not None)
