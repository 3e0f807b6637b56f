"""A wait that ran out is raised before the results it concerns are handed out.  Nothing fails here: the error word is set
from the host, as a kernel that gives up would set it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from velox_b200.csrc import ops as o
    return o


@pytest.fixture(autouse=True)
def clean():
    ops().check_device_errors()
    yield
    torch.cuda.synchronize()
    ops()._error_word(torch.device(DEV)).zero_()
    ops().check_device_errors()


def set_word():
    ops()._error_word(torch.device(DEV)).fill_(8)


def products():
    a, w = torch.randn(24, 1024, device=DEV), torch.randn(256, 1024, device=DEV)
    ab, wb = a.bfloat16(), w.bfloat16()
    return {"turned": lambda: ops().gemm_turned(ab, wb),
            "turned gated": lambda: ops().gemm_turned(ab, wb, gated_activation="silu"),
            "float32": lambda: ops().gemm_nt_simt(a, w),
            "float32 heads": lambda: ops().gemm_heads(a.view(24, 1, 1024), w.view(1, 256, 1024), torch.empty(24, 1, 256, device=DEV)),
            "float32 members": lambda: ops().gemm_members(a.view(1, 24, 1024), w.view(1, 256, 1024)),
            "tcgen05": lambda: ops().gemm_tcgen05(ab, wb)}


@pytest.mark.parametrize("name", ["turned", "turned gated", "float32", "float32 heads", "float32 members", "tcgen05"])
def test_products_with_bounded_waits_are_checked(name):
    o = ops()
    call = products()[name]
    call()
    assert o.bounded_wait_pending()
    o.check_pending_device_errors()
    assert not o.bounded_wait_pending()
    call()
    set_word()
    with pytest.raises(o.KernelError, match="gave up a wait"):
        o.check_pending_device_errors()
    o.check_pending_device_errors()   # (reported once)


def test_a_kernel_writes_the_error_word_and_the_host_reads_it():
    """The word lies in host memory: what a kernel stores there (the sampler its token id, 8) is there when the kernel has ended."""
    o = ops()
    logits = torch.zeros(1, 64, device=DEV)
    logits[0, 8] = 1.0
    word = o._error_word(torch.device(DEV))
    assert int(word[0]) == 0 and word.data_ptr() == o._error_address(torch.device(DEV))
    o._check(o.library().vx_sample(o._ptr(logits), 64, 1, 64, None, None, None, o._ptr(word), o._stream()), "sample")
    torch.cuda.synchronize()
    assert int(word[0]) == 8
    with pytest.raises(o.KernelError, match="code 8"):
        o.check_device_errors()
    assert int(word[0]) == 0


def engine(dtype, vocab=512):
    from velox_b200 import Engine, EngineConfig
    from velox_b200.config import Qwen3Config
    raw = dict(vocab_size=vocab, hidden_size=1024, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=4, head_dim=128,
               attention_bias=False, num_key_value_heads=2, max_position_embeddings=256, tie_word_embeddings=False, rope_theta=10000.0,
               rms_norm_eps=1e-6, hidden_act="silu", architectures=["Qwen3ForCausalLM"], model_type="qwen3")
    return Engine(model_config=Qwen3Config.from_dict(raw), random_seed=1,
                  config=EngineConfig(dtype=dtype, page_size=16, num_pages=64, max_running_requests=16, max_model_len=64))


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_a_decode_step_hands_out_no_token_of_a_failed_wait(dtype):
    """Twelve requests decode; then the word is set while a step's results are under way: that very step raises, the last one of a
    request (after which nothing would look again) as well."""
    from velox_b200 import SamplingParams
    e = engine(dtype)
    for i in range(12):
        e.add_request([1 + i, 7, 9], SamplingParams(max_tokens=4))
    for _ in range(3):
        e.step()
    e.on_logits = lambda ids, logits: set_word()
    with pytest.raises(ops().KernelError, match="gave up a wait"):
        e.step()


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_run_step_hands_out_no_logits_of_a_failed_wait(dtype):
    from velox_b200.engine import StepEntry
    e = engine(dtype)
    for i in range(12):
        e.cache.add_request(i)
    entries = [StepEntry(i, [3 + i], [0]) for i in range(12)]
    for _ in range(2):
        e.run_step(entries)
    logits = e.runner.step(entries)
    assert e.runner.pending_error_check and logits is not None
    set_word()
    with pytest.raises(ops().KernelError, match="gave up a wait"):
        e.runner.check_errors()
    assert not e.runner.pending_error_check


def test_the_end_of_waits_of_a_graph_is_that_of_its_latest_replay():
    """The host waits for the event that a replay records behind its last kernel with bounded waits: what comes before it has then run,
    in that very replay, though the stream is still busy with what comes after."""
    o = ops()
    x, big = torch.zeros(1, dtype=torch.int32, device=DEV), torch.randn(4096, 4096, device=DEV).bfloat16()
    end = o.EndOfWaits(captured=True)

    def work():
        for _ in range(20):
            torch.mm(big, big)
        x.add_(1)
        end.record()
        for _ in range(20):
            torch.mm(big, big)

    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        work()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        work()
    x.zero_()
    torch.cuda.synchronize()
    busy = 0
    for i in range(1, 21):
        graph.replay()
        end.event.synchronize()
        busy += not torch.cuda.current_stream().query()
        with torch.cuda.stream(side):
            assert int(x.item()) == i
    assert busy > 0


def test_a_captured_step_is_checked_at_its_end_of_waits():
    """Decode steps from a graph: the end noted last is the graph's own, and covers all that it launched."""
    from velox_b200.engine import StepEntry
    o, e = ops(), engine("bfloat16", vocab=32784)   # (the head is the library's: no waits)
    for i in range(12):
        e.cache.add_request(i)
    for k in range(3):
        e.runner.step([StepEntry(i, [3 + i], [0]) for i in range(12)])
        if k:
            assert o._END_OF_WAITS[0] == o.bounded_wait_launches()
            g = next(iter(e.runner.graphs.graphs.values()))
            assert o._END_OF_WAITS[1] is g.end_of_waits.event
        e.runner.check_errors()
        assert not e.runner.pending_error_check


def test_a_captured_step_without_bounded_waits_records_no_end():
    from velox_b200.engine import StepEntry
    o, e = ops(), engine("bfloat16", vocab=32784)
    for i in range(2):
        e.cache.add_request(i)
    for _ in range(3):
        e.runner.step([StepEntry(i, [3 + i], [0]) for i in range(2)])
        assert not e.runner.pending_error_check
    g = next(iter(e.runner.graphs.graphs.values()))
    assert g.graph is not None and g.bounded_wait_launches == 0 and g.end_of_waits.launches == -1


def test_a_step_that_the_caller_captures_notes_no_end_of_waits():
    """Checks afterwards wait for the stream, as they do for any
    kernel with bounded waits behind which no end was noted."""
    from velox_b200.engine import StepEntry
    from velox_b200.engine.batch import build_step_context
    o, e = ops(), engine("bfloat16", vocab=32784)
    for i in range(12):
        e.cache.add_request(i)
    entries = [StepEntry(i, [3 + i], [0]) for i in range(12)]
    for i in range(12):
        e.cache.reserve(i, 1)
    ctx = build_step_context(entries, e.cache, e.device, 32784, e.runner.short_max)
    e.runner.run(ctx)
    e.runner.check_errors()
    noted = o._END_OF_WAITS
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        e.runner.run(ctx)
    assert o._END_OF_WAITS is noted and e.runner.pending_error_check
    graph.replay()
    set_word()
    with pytest.raises(o.KernelError, match="gave up a wait"):
        e.runner.check_errors()
