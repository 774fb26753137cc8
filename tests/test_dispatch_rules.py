"""What the dispatchers decide and hand on, without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from vllm_lite_b200.csrc import ops
from vllm_lite_b200.parts import attention_dispatch
from vllm_lite_b200.parts.base import StepBatch, Workspace


def decode_call(monkeypatch, *, tokens, spec, bound, dtype=torch.bfloat16, **step):
    """The arguments with which a decode step of `tokens` requests reaches `ops.flash_decode`."""
    seen = {}
    monkeypatch.setattr(ops, "sm_pairs", lambda: 74)
    monkeypatch.setattr(ops, "flash_decode_max_cluster", lambda hd: 8)
    monkeypatch.setattr(ops, "flash_decode", lambda *args, **kw: seen.update(kw, part_acc=args[13], part_ml=args[14]))
    q = torch.empty(tokens, 8, dtype=dtype)
    batch = SimpleNamespace(workspace=Workspace("cpu"), tag="", err=None, req_index=None, positions=None, max_query_len=1, query_tiles=None,
                            single_tokens=None, **step)
    group = SimpleNamespace(page_size=64, max_context=bound, block_table=None)
    cache = SimpleNamespace(k=None, v=None)
    attention_dispatch.run(q, None, cache, group, batch, SimpleNamespace(**spec), 1.0)
    return seen


QWEN = dict(num_heads=32, num_kv_heads=8, head_dim=128, window=None)


@pytest.mark.parametrize("settled", [True, False])
def test_a_step_says_whether_its_description_may_be_read_early(monkeypatch, settled):
    assert decode_call(monkeypatch, tokens=64, spec=QWEN, bound=4096, settled=settled)["settled"] is settled


def test_a_step_may_not_be_read_early_unless_it_says_so(monkeypatch):
    assert decode_call(monkeypatch, tokens=64, spec=QWEN, bound=4096)["settled"] is False
    assert StepBatch.__dataclass_fields__["settled"].default is False


# where the measured times of the two decode kernels cross (requests, KV heads, head size, bound), page size 64
@pytest.mark.parametrize("tokens,heads,size,bound,streams", [
    (48, 8, 128, 1024, False), (64, 8, 128, 1024, False), (24, 8, 128, 2048, False), (32, 8, 128, 2048, True), (64, 8, 128, 2048, True),
    (8, 8, 128, 4096, False), (12, 8, 128, 4096, True), (16, 8, 128, 4096, True), (16, 4, 128, 4096, False), (32, 4, 128, 4096, True),
    (4, 8, 128, 8192, False), (8, 8, 128, 8192, True), (12, 4, 128, 8192, True), (4, 8, 128, 16384, True), (4, 4, 128, 30000, True),
    (1, 8, 128, 32768, False), (64, 8, 128, 512, False), (64, 8, 64, 4096, False), (8, 8, 64, 16384, False)])
def test_which_decode_kernel_serves_a_step(tokens, heads, size, bound, streams):
    assert ops.flash_decode_streams(torch.bfloat16, tokens, heads, size, 64, bound) is streams
    assert not ops.flash_decode_streams(torch.bfloat16, tokens, heads, size, 32, bound)      # short pages: small boxes
    assert not ops.flash_decode_streams(torch.float32, tokens, heads, size, 64, bound)


def shared(heads, rank, window=None):
    return dict(num_heads=heads, num_kv_heads=1, head_dim=rank, window=window, shared_row=True)


# halved while all blocks still run at once (148 SMs), and with a window while the launch holds few blocks outside it
@pytest.mark.parametrize("tokens,heads,rank,window,bound,chunk", [
    (2, 16, 256, None, 4096, 128), (16, 16, 256, None, 1024, 128), (32, 16, 256, None, 1024, 256), (16, 16, 256, None, 2048, 256),
    (16, 32, 256, None, 1024, 256), (32, 16, 256, None, 4096, 1024), (8, 16, 256, None, 16384, 1024), (64, 16, 256, None, 1024, 256),
    (8, 16, 256, 1024, 16384, 128), (16, 16, 256, 1024, 16384, 256), (16, 16, 256, 1024, 4096, 128), (32, 16, 128, None, 1024, 128),
    (32, 16, 128, 1024, 16384, 128), (64, 16, 128, 1024, 16384, 256), (64, 16, 128, None, 16384, 1024)])
def test_chunks_of_a_shared_row(monkeypatch, tokens, heads, rank, window, bound, chunk):
    got = decode_call(monkeypatch, tokens=tokens, spec=shared(heads, rank, window), bound=bound)
    assert got["chunk"] == chunk and got["arrivals"] is None and got["stream_kernel"] is False


@pytest.mark.parametrize("tokens", [1, 2, 4, 8, 16, 32, 36, 64])
@pytest.mark.parametrize("heads,rank,window", [(16, 256, 1024), (16, 256, 64), (32, 128, 1024), (64, 256, 2048), (16, 256, None), (16, 128, None)])
def test_scratch_of_a_shared_row_stays_small(monkeypatch, tokens, heads, rank, window):
    """Shorter chunks must not multiply the scratch, which nobody reserves: at most 64 MB where they are shortened."""
    whole = 1024 if not window or window > 2048 else (256 if window <= 1024 else 512)
    got = decode_call(monkeypatch, tokens=tokens, spec=shared(heads, rank, window), bound=131072)
    assert got["chunk"] == whole or 4 * got["part_acc"].numel() <= 64 << 20


def test_counters_are_zero_again_behind_an_error_that_was_raised():
    from vllm_lite_b200.engine.runner import ModelRunner, StepError
    runner = ModelRunner.__new__(ModelRunner)            # no device: the error word and the workspace are all that is read
    runner.err, runner.workspace = torch.tensor([0x2008], dtype=torch.int32), Workspace("cpu")
    counters = runner.workspace.zeros("attn.arrivals", 5, torch.int32)
    kept = runner.workspace.get("attn.out", (4,), torch.float32).fill_(3.0)
    counters[2] = 4                                      # as a block leaves it whose wait ran out before its last arrival
    with pytest.raises(StepError, match="wait"):
        runner.check_device_errors()
    assert not counters.any() and int(runner.err) == 0
    assert runner.workspace.zeros("attn.arrivals", 5, torch.int32) is counters and bool((kept == 3).all())
    runner.check_device_errors()                         # nothing left to raise


# single slots, one run, a few runs, scattered ones (the last of the pool and the first among them), a list in no order
@pytest.mark.parametrize("slots", [[], [5], [3, 4, 5, 6], [9, 1, 0], [0, 2, 4, 6], list(range(63, -1, -2)), list(range(64)), [63, 0, 31, 7, 8, 12]])
def test_fresh_slots_are_zeroed_in_few_launches(slots):
    from torch.utils._python_dispatch import TorchDispatchMode

    from vllm_lite_b200.cache.storage import CacheStorage
    writes = []

    class Count(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if any(name in str(func) for name in ("zero_", "fill_", "index_put_", "copy_")):
                writes.append(str(func))
            return func(*args, **(kwargs or {}))

    state = [torch.full((2, 64, 3), 7.0), torch.full((1, 64, 2, 2), 7, dtype=torch.int32), torch.full((3, 64), 7.0, dtype=torch.bfloat16)]
    with Count():
        CacheStorage.zero_slots(SimpleNamespace(state=state), slots)
    for t in state:
        for s in range(64):
            assert bool((t[:, s] == (0 if s in slots else 7)).all()), s
    assert len(writes) <= 3 * len(state)


@pytest.mark.parametrize("counts,heads,dim,pays", [
    ([95, 40], 32, 64, False), ([96], 32, 64, False), ([96, 96], 32, 64, True), ([127], 32, 64, False), ([128], 8, 64, True),
    ([96] * 4, 8, 64, False), ([96] * 8, 8, 64, True), ([96, 1, 1, 1, 1, 1, 1, 1], 8, 64, False), ([128, 96], 4, 64, True),
    ([96], 16, 128, False), ([159], 16, 128, False), ([160], 16, 128, True), ([96], 24, 128, True), ([96, 96], 16, 128, True),
    ([223], 8, 128, False), ([224], 4, 96, True), ([127], 32, 32, False), ([128], 128, 32, True), ([191, 128], 128, 32, False),
    ([192, 128], 128, 32, True), ([], 32, 64, False)])
def test_which_portions_of_a_time_mixing_are_cut_into_chunks(counts, heads, dim, pays):
    assert ops.decay_chunks_pay(counts, heads, dim) is pays


@pytest.mark.parametrize("tokens,heads,dim,pays", [(1, 4, 64, True), (1, 32, 32, True), (1, 16, 128, False), (2, 16, 128, False),
                                                   (3, 16, 128, True), (1, 32, 128, False), (2, 32, 128, True), (4, 8, 96, False), (5, 8, 96, True)])
def test_which_single_tokens_of_a_time_mixing_take_a_block_a_head(tokens, heads, dim, pays):
    assert ops.decay_step_pays(tokens, heads, dim) is pays


@pytest.mark.parametrize("heads,dim", [(32, 64), (16, 128), (2, 16), (7, 100)])
def test_only_bfloat16_steps_reserve_room_for_chunks_of_a_time_mixing(heads, dim):
    from vllm_lite_b200.cache.sizing import _mixer_width
    from vllm_lite_b200.parts.spec import TimeMixSpec
    spec, tokens = TimeMixSpec(heads * dim, heads, dim, 16, 1e-5), 4096
    walk = _mixer_width(spec, 4)
    assert walk == 5 * spec.hidden_size + 12 * heads * dim + 2 * 16        # the products, mixes, gate and rows alone
    for n in (96, 129, 200, 1000, 4096):                 # portions whose last chunks are as short as they come, and one long one
        chunks = ops.decay_chunks_of([n] * (tokens // n))
        assert 4 * ops.decay_chunk_floats(chunks, heads, dim, dim) <= 2 * (_mixer_width(spec, 2) - walk) * tokens


def test_constants_that_the_chunked_time_mixing_and_its_caller_share():
    import ctypes

    from vllm_lite_b200.csrc import build
    lib = build.load("decay_chunks")
    lib.vl_decay_chunk_floats.restype = ctypes.c_longlong
    assert lib.vl_decay_min_chunk() == ops.DECAY_MIN_CHUNK
    for sizes in ((1, 1, 4, 4), (7, 32, 64, 64), (3, 5, 100, 68), (4096, 16, 128, 128)):
        assert lib.vl_decay_chunk_floats(*sizes) == ops.decay_chunk_floats(*sizes)


@pytest.mark.parametrize("sizes", [(1, 1, 4, 4), (7, 32, 64, 64), (3, 5, 100, 68), (4096, 16, 128, 128)])
def test_the_delta_rules_scratch_is_what_its_caller_brings(sizes):
    import ctypes
    from vllm_lite_b200.csrc import build
    floats = build.load("delta").vl_delta_chunk_floats
    floats.restype = ctypes.c_longlong
    assert floats(*sizes) == ops.delta_chunk_floats(*sizes)


# where the measured times cross (148 SMs): the weight-streaming product up to 8 rows, a tile of W an SM, the library
@pytest.mark.parametrize("M,N,K,few", [
    (8, 2048, 2048, False), (9, 2048, 2048, True), (16, 7104, 2048, True), (16, 7120, 2048, False), (17, 4736, 2048, True), (24, 4752, 8192, False),
    (25, 6144, 4096, True), (32, 6144, 2048, False), (32, 7120, 4096, False), (33, 2368, 512, True), (48, 2384, 512, False), (49, 64, 512, False),
    (12, 2048, 2052, False)])
def test_which_products_of_few_rows_take_a_tile_an_sm(monkeypatch, M, N, K, few):
    monkeypatch.setattr(ops, "sm_pairs", lambda: 74)
    assert ops.gemm_bf16_few_ok(M, N, K) is few


@pytest.mark.parametrize("tokens,pairs,experts,K,big", [(64, 4096, 32, 2048, False), (65, 192, 32, 2048, True), (65, 191, 32, 2048, False),
                                                        (100, 800, 128, 2048, True), (100, 764, 128, 2048, False), (512, 4096, 64, 2044, False)])
def test_which_experts_products_run_on_tcgen05(tokens, pairs, experts, K, big):
    assert ops.gemm_grouped_tc5_ok(torch.bfloat16, tokens, pairs, experts, K) is big
    assert not ops.gemm_grouped_tc5_ok(torch.float32, tokens, pairs, experts, K)


def test_few_rows_an_expert_keep_the_full_exponential():
    assert ops.gemm_grouped_tc5_fine(1023, 4) and not ops.gemm_grouped_tc5_fine(1024, 4)
    assert ops.gemm_grouped_tc5_fine(96 * 32 - 1, 32) and not ops.gemm_grouped_tc5_fine(96 * 32, 32)


# Products of paired blocks never run among programmatic launches: up to 64 tokens none is chosen, beyond them a recorded step asks the model.
def test_no_product_of_paired_blocks_among_programmatic_launches(monkeypatch):
    from vllm_lite_b200.engine.runner import PDL_MAX_TOKENS, launches_dependent
    monkeypatch.setattr(ops, "sm_pairs", lambda: 74)
    for T in (1, 2, PDL_MAX_TOKENS - 1, PDL_MAX_TOKENS):
        assert not any(ops.gemm_grouped_tc5_ok(torch.bfloat16, T, T * top, E, 2048) for top in (1, 2, 8, 64) for E in (1, 2, 8, 128))
    for M in range(1, ops.TC5_MIN_M_FULL):
        assert not any(ops.gemm_bf16_tc5_ok(M, 4096, fused, N) for fused in (False, True) for N in (None, 256, 24576))
    yes, no = (lambda tokens: True), (lambda tokens: False)
    assert launches_dependent(PDL_MAX_TOKENS, True, yes) and launches_dependent(PDL_MAX_TOKENS, False, yes)
    assert not launches_dependent(PDL_MAX_TOKENS + 1, True, yes) and launches_dependent(PDL_MAX_TOKENS + 1, True, no)
    assert not launches_dependent(PDL_MAX_TOKENS + 1, False, no)


def test_a_recorded_step_asks_the_model_for_paired_products(monkeypatch):
    from types import SimpleNamespace
    from vllm_lite_b200.engine.runner import ModelRunner
    from vllm_lite_b200.parts.base import BuildContext
    from vllm_lite_b200.parts.experts import RoutedExperts
    from vllm_lite_b200.parts.model import CausalLM

    class Launched(Exception):
        pass

    def forward(batch, caches):
        raise Launched

    E, top, H, I = 8, 2, 64, 16
    ctx = BuildContext(torch.device("cpu"), torch.bfloat16)
    from vllm_lite_b200.parts.spec import RoutedExpertsSpec
    spec = RoutedExpertsSpec(hidden_size=H, intermediate_size=I, num_experts=E, top=top)
    weights = {n: torch.zeros(d.shape, dtype=torch.bfloat16) for n, d in RoutedExperts.declare(spec).items()}
    part = RoutedExperts(spec, weights, ctx)
    assert ctx.paired == [part.may_pair]
    model = CausalLM.__new__(CausalLM)
    model.ctx, model.forward = ctx, forward
    runner = ModelRunner.__new__(ModelRunner)
    runner.model, runner.storage, runner._graphs = model, SimpleNamespace(call_caches=[]), {}
    states = []
    monkeypatch.setattr(ops, "set_pdl", states.append)
    for tokens, paired in ((64, False), (128, True), (256, True), (512, True)):
        assert part.may_pair(tokens) is paired and model.may_pair(tokens) is paired
        with pytest.raises(Launched):
            runner._forward_graph(SimpleNamespace(graph_bucket=tokens, num_tokens=tokens, groups=[]))
        assert states.pop() is not paired
    ctx.paired.clear()                                   # a dense model: only where its own products may be paired ones
    for tokens, on in ((256, True), (512, False), (4096, False)):
        with pytest.raises(Launched):
            runner._forward_graph(SimpleNamespace(graph_bucket=tokens, num_tokens=tokens, groups=[]))
        assert states.pop() is on


# What a pre-norm block asks of its parts: the sum into the stream, where both neighbours should factor the norm between them; the float32 sums, where
# they could but take a faster product; else a result in the activation dtype.
@pytest.mark.parametrize("can,should", [((1, 1), (1, 1)), ((1, 1), (0, 1)), ((1, 1), (1, 0)), ((1, 1), (0, 0)), ((1, 0), (1, 0)), ((0, 0), (0, 0))])
@pytest.mark.parametrize("nxt", [None, True, False])
def test_a_pre_norm_block_never_rounds_what_it_could_add_in_float32(can, should, nxt):
    from vllm_lite_b200.parts.base import Residual
    from vllm_lite_b200.parts.block import PreNormBlock

    class Part:
        def __init__(self, i):
            self.i, self.asked = i, None

        def can_factor_norms(self, M):
            return bool(can[self.i])

        def factors_norms(self, M):
            return bool(should[self.i])

        def __call__(self, h, *rest, sink=None, sums=False):
            self.asked = "sink" if sink is not None else "sums" if sums else "rounded"
            return self.asked

    class Norm(SimpleNamespace):
        def __call__(self, x, delta, step, tag):
            return tag

    block = PreNormBlock.__new__(PreNormBlock)
    block.mixer, block.ffn = Part(0), Part(1)
    block.norm1, block.norm2 = (Norm(factorable=True, weight=None, spec=SimpleNamespace(eps=0.0, size=0)) for _ in range(2))
    residual, after = Residual(None), Norm(weight=None, spec=SimpleNamespace(eps=0.0, size=0))
    block(residual, SimpleNamespace(num_tokens=12), None, next_norm=None if nxt is None else (after, nxt))
    assert block.mixer.asked == ("rounded" if not all(can) else "sink" if all(should) else "sums")
    assert block.ffn.asked == ("rounded" if nxt is None or not can[1] else "sink" if nxt and should[1] else "sums")
    assert (residual.normed_for is after) == (block.ffn.asked == "sink") == (residual.pending is None)


def test_layers_of_4096_columns_leave_their_sums(monkeypatch):
    """Nine to sixteen rows: the product that takes a tile an SM, and no less of the residual than the weight-streaming product adds."""
    from vllm_lite_b200.parts.linear import Linear
    monkeypatch.setattr(ops, "sm_pairs", lambda: 74)
    wide, narrow = (Linear(torch.empty(64, K, dtype=torch.bfloat16)) for K in (4096, 2048))
    for M in (1, 8, 9, 16, 17):
        assert wide.can_factor_norms(M) is narrow.can_factor_norms(M) is (M <= 16)
        assert narrow.factors_norms(M) is (M <= 16) and wide.factors_norms(M) is (M <= 8)


# The tcgen05 products: plain ones from 2,048 rows, the fused activation from 1,024, and from 512 where at most a quarter of the tiles is padding or
# places without a tile (74 pairs of SMs; gate/up of 24,576 rows of W: 96 tiles for 256 rows).
@pytest.mark.parametrize("M,N,fused,takes", [
    (511, 24576, True, False), (512, 24576, True, True), (536, 24576, True, False), (768, 24576, True, True), (900, 24576, True, False),
    (1023, 24576, True, True), (1024, 24576, True, True), (1024, 512, True, True), (512, 512, True, False), (768, None, True, False),
    (1023, None, True, False), (1024, None, True, True), (1024, 24576, False, False), (2047, 24576, False, False), (2048, 64, False, True)])
def test_which_products_run_on_tcgen05(monkeypatch, M, N, fused, takes):
    monkeypatch.setattr(ops, "sm_pairs", lambda: 74)
    assert ops.gemm_bf16_tc5_ok(M, 4096, fused, N) is takes
    assert not ops.gemm_bf16_tc5_ok(M, 4100, fused, N)


def test_a_fused_activation_is_promised_where_a_kernel_takes_it(monkeypatch):
    """`fuses_swiglu` and the product itself ask the same rules: what is promised finds a kernel, and what is not has none."""
    from vllm_lite_b200.parts import matmul
    monkeypatch.setattr(ops, "sm_pairs", lambda: 74)
    for name in ("gemm_bf16_few", "gemm_bf16_small_m", "gemm_bf16_tc5", "gemm_bf16_tc5_pair"):
        monkeypatch.setattr(ops, name, lambda *a, _n=name, **k: _n)
    for N in (64, 2048, 4752, 7120, 24576):
        for K in (64, 4096, 4100):
            w = torch.empty(N, K, dtype=torch.bfloat16, device="meta")
            for M in (1, 8, 9, 16, 17, 32, 33, 48, 49, 64, 511, 512, 536, 768, 1023, 1024, 4096):
                a = torch.empty(M, K, dtype=torch.bfloat16, device="meta")
                if matmul.fuses_swiglu(M, K, N):
                    assert matmul.gemm_bf16(a, w, None, swiglu=True).startswith("gemm_bf16_")
                else:
                    with pytest.raises(ValueError):
                        matmul.gemm_bf16(a, w, None, swiglu=True)
