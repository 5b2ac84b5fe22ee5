"""The one-rank kernels, batch (csrc/mm_batch.cuh) and decode (csrc/mm_decode.cuh), at the sizes where it can go wrong, against the CPU oracle: row counts around
the 16-row groups and the tile limits (128 rows, 96 with E4M3 tokens), more tokens than SMs, masked slots, the largest
launch, experts without rows. Tolerances are the layer's: relative RMSE 0.3 %, counts and slot maps exact."""
import pytest
import torch

import hopper_megamoe_basedondeepgemm_b200 as mm
from hopper_megamoe_basedondeepgemm_b200 import _lib
from oracle import megamoe_oracle as O
from tests import util_moe as U
from tests.test_gpu_frontend import _canon
from tests.test_gpu_layer import REL_RMSE_TOL, check_against_oracle, run_layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
@pytest.mark.parametrize('e_local,topk,tokens', [
    (8, 1, 17),           # one entry more than decode mode takes
    (2, 2, 16), (2, 2, 17),         # exactly one 16-row group per expert, and one row beyond it
    (2, 2, 96), (2, 2, 97),         # the E4M3 tile limit
    (2, 2, 128), (2, 2, 129),       # the tile limit of the 4-bit formats
    (64, 3, 31),          # the most experts, an odd number of routes, many experts with one row or none
    (4, 3, 301),          # more tokens than SMs, several tiles per expert
])
def test_row_counts_around_the_tile_edges(fmt, e_local, topk, tokens):
    y, stats, ref, buf, _ = run_layer(fmt, e_local, 512, 256, topk, tokens, 'random', 'umma', seed=tokens, std=0.02)
    assert buf.device_status()[1][3] == (96 if fmt == 'fp8' else 128)          # the batch kernel ran
    check_against_oracle(y, stats, ref, buf, fmt, 256)


@pytest.mark.parametrize('e_local,hidden,inter,topk,tokens', [
    (4, 4096, 768, 2, 8), (3, 512, 256, 3, 5), (2, 1536, 1280, 2, 1),          # decode kernel: the widest token tile; units per task odd and even
    (4, 4096, 256, 2, 170), (3, 1536, 768, 3, 31), (8, 512, 256, 2, 12),       # batch kernel: 96-row records (fewest weight stages), 32- and 16-row ones
])
def test_widened_units_over_ring_depths_and_odd_unit_counts(e_local, hidden, inter, topk, tokens):
    y, stats, ref, buf, _ = run_layer('fp8', e_local, hidden, inter, topk, tokens, 'random', 'umma', seed=tokens, std=0.02)
    check_against_oracle(y, stats, ref, buf, 'fp8', inter)


@pytest.mark.parametrize('num_sms', [5, 0])
@pytest.mark.parametrize('hidden,inter', [(512, 768), (1536, 256), (4096, 256)])
def test_shapes_and_small_grids(hidden, inter, num_sms):
    """K units that fill no pair, an L1 task shorter than an L2 task, the largest hidden size; a grid of a few SMs."""
    y, stats, ref, buf, _ = run_layer('mxfp4', 6, hidden, inter, 4, 23, 'random', 'umma', seed=hidden, std=0.02, num_sms=num_sms,
                                      masked_ratio=0.3, t_max=64)
    assert buf.device_status()[1][3] == 128
    check_against_oracle(y, stats, ref, buf, 'mxfp4', inter)


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4'])
@pytest.mark.parametrize('num_sms,e_local,hidden,inter,topk,tokens', [
    (6, 2, 512, 512, 2, 9), (5, 2, 512, 512, 2, 9),           # 48 units of weights: eight per SM, and more; first units of a tile per SM and the loader's
    (5, 2, 1024, 256, 2, 9),                                  # less than two tiles per SM: the loader's alone
    (2, 3, 512, 256, 3, 9), (1, 3, 4096, 256, 3, 9),          # tiles of two units, and of sixteen
    (2, 24, 512, 256, 1, 40),                                 # experts without rows among those whose weights may be asked for
    (20, 16, 512, 256, 16, 128), (20, 16, 512, 256, 16, 129),         # 2048 routing entries, and more
])
@pytest.mark.parametrize('masked', [0.0, 0.4])
def test_weights_asked_ahead_on_both_sides_of_the_lines(fmt, num_sms, e_local, hidden, inter, topk, tokens, masked):
    y, stats, ref, buf, _ = run_layer(fmt, e_local, hidden, inter, topk, tokens, 'random', 'umma', seed=tokens, std=0.02, num_sms=num_sms, masked_ratio=masked)
    check_against_oracle(y, stats, ref, buf, fmt, inter)


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
@pytest.mark.parametrize('num_sms,e_local,inter,topk,tokens', [
    (1, 8, 256, 4, 10), (1, 8, 256, 4, 11),        # 40 and 44 rows of 512 columns on one SM: 40 KB, and more
    (4, 14, 256, 2, 100), (4, 13, 256, 2, 100),    # 14 tasks of one unit per SM, the least that leaves ten in front of four, and 13
    (3, 4, 512, 3, 90), (1, 2, 256, 2, 40),        # two units to a task; fewer tiles than would go column block by column block
])
def test_column_tasks_on_both_sides_of_the_lines(fmt, num_sms, e_local, inter, topk, tokens):
    y, stats, ref, buf, _ = run_layer(fmt, e_local, 512, inter, topk, tokens, 'random', 'umma', seed=tokens, std=0.02, num_sms=num_sms)
    check_against_oracle(y, stats, ref, buf, fmt, inter)


def _small_layer(fmt, e, hidden, inter, topk, tokens, seed, masked=0.0):
    w, _, _ = O.make_expert_weights(e, hidden, inter, fmt, seed=seed, std=0.05)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, tokens, topk, hidden, inter, act_format=fmt)
    idx, tw = U.random_routing(tokens, e, topk, seed + 1, masked)
    _, inp, sfb = U.make_rank_inputs(tokens, hidden, fmt, seed + 2, idx, tw)
    U.write_inputs(buf, inp, sfb)
    return w, l1, l2, buf, inp, sfb


# (a clamp far inside the values' range would not do: it makes rows of equal products, and one rounding tie they share then
# moves the whole output by 2 %, with the multi-rank kernel just as much)
@pytest.mark.parametrize('fast_math,clamp', [(True, None), (False, 0.5)])
def test_largest_launch_exact_math_and_clamp(fast_math, clamp):
    """4096 routing entries, twice on one buffer (the second launch counts in the other set of arrival counters)."""
    fmt, e, hidden, inter, topk, tokens = 'mxfp4', 64, 512, 256, 8, 512
    w, l1, l2, buf, inp, _ = _small_layer(fmt, e, hidden, inter, topk, tokens, 900, 0.05)
    ref = O.moe_layer_reference([inp], [w], fmt, e, clamp=clamp)
    y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    for _ in range(2):
        mm.fp4_fp4_mega_moe(y.zero_(), l1, l2, buf, activation_clamp=clamp, fast_math=fast_math, timeout_ms=500.0)
        assert buf.device_status()[0] == 0
        assert O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL


def test_all_slots_masked_gives_zeros():
    _, l1, l2, buf, _, _ = _small_layer('mxfp4', 4, 512, 256, 4, 20, 910)
    buf.topk_idx.fill_(-1)
    y = torch.full((20, 512), 3.0, dtype=torch.bfloat16, device='cuda')
    mm.fp4_fp4_mega_moe(y, l1, l2, buf, timeout_ms=500.0)
    assert buf.device_status()[0] == 0 and float(y.abs().max()) == 0.0


def test_route_to_a_missing_expert_is_reported_and_the_buffer_recovers():
    w, l1, l2, buf, inp, sfb = _small_layer('mxfp4', 4, 512, 256, 2, 20, 920)
    ref = O.moe_layer_reference([inp], [w], 'mxfp4', 4, clamp=None)
    y = torch.empty((20, 512), dtype=torch.bfloat16, device='cuda')
    buf.topk_idx[7, 1] = 4
    mm.fp4_fp4_mega_moe(y, l1, l2, buf, timeout_ms=500.0)
    st, words = buf.device_status()
    assert st == 4 and (words[0] & 0xFF) == 9                  # the status a route nobody serves has always had
    buf.reset()
    U.write_inputs(buf, inp, sfb)
    mm.fp4_fp4_mega_moe(y, l1, l2, buf, timeout_ms=500.0)
    assert buf.device_status()[0] == 0 and O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL


def test_decode_and_batch_launches_alternate_on_one_buffer():
    """Both kernels share the buffer's launch numbering and clear each other's counters."""
    fmt, e, hidden, inter, topk = 'fp8', 4, 512, 256, 2
    w, _, _ = O.make_expert_weights(e, hidden, inter, fmt, seed=1, std=0.05)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, 64, topk, hidden, inter, act_format=fmt)
    for it, tokens in enumerate([40, 3, 40, 8, 9, 1, 2, 64]):
        idx, tw = U.random_routing(tokens, e, topk, 930 + it)
        _, inp, sfb = U.make_rank_inputs(tokens, hidden, fmt, 940 + it, idx, tw)
        ref = O.moe_layer_reference([inp], [w], fmt, e, clamp=None)
        U.write_inputs(buf, inp, sfb)
        y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
        mm.fp8_fp4_mega_moe(y, l1, l2, buf, timeout_ms=500.0)
        st, words = buf.device_status()
        assert st == 0 and words[1] == it + 1 and (words[3] != 0) == (tokens * topk > 16)
        assert O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL, (it, tokens)


def test_layout_holds_the_packed_images():
    """An expert's rows are rounded up to 16 in the images: the regions hold the worst case of every format."""
    import ctypes
    lib = _lib.load()
    for fmt, atoms, planes in (('mxfp4', 1, 2), ('nvfp4', 1, 4), ('fp8', 2, 2)):
        cfg, L = _lib.MMConfig(1, 0, 64, 512, 8, 3072, 1280, _lib.FMT[fmt], 148), _lib.MMLayout()
        assert lib.mm_get_layout(ctypes.byref(cfg), ctypes.byref(L)) == 0
        groups, tiles = (4096 + 15 * 64 + 15) // 16, 64 + 4096 // 64
        need = lambda units: units * (groups * 2048 * atoms + tiles * planes * 512)      # noqa: E731
        assert L.tile_capacity * L.token_tile_bytes >= need(12) and L.tile_capacity * L.mid_tile_bytes >= need(5)


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
@pytest.mark.parametrize('e_local,topk,tokens,hidden,inter', [
    (1, 1, 1, 512, 256),            # one row, one expert
    (64, 8, 2, 1024, 256),          # sixteen rows, (almost) all on experts of their own
    (16, 1, 16, 512, 512),          # one route per token
    (2, 2, 8, 1536, 256),           # eight rows per expert
    (20, 5, 3, 512, 2048),          # an odd entry count; an L2 task longer than an L1 task
    (48, 8, 1, 3072, 1280),         # the benchmark's layer: remainder tiles split over the SMs
])
def test_decode_kernel(fmt, e_local, topk, tokens, hidden, inter):
    """At most 16 routing entries on one rank (csrc/mm_decode.cuh), a few slots masked."""
    y, stats, ref, buf, _ = run_layer(fmt, e_local, hidden, inter, topk, tokens, 'random', 'umma', seed=7 * tokens, std=0.02,
                                      masked_ratio=0.15 if tokens > 1 else 0.0)
    check_against_oracle(y, stats, ref, buf, fmt, inter)


@pytest.mark.parametrize('num_sms', [3, 0])
def test_decode_kernel_small_grid_masked_and_missing_expert(num_sms):
    fmt, e, hidden, inter, topk, tokens = 'mxfp4', 6, 1024, 512, 4, 4
    w, _, _ = O.make_expert_weights(e, hidden, inter, fmt, seed=50, std=0.05)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, 16, topk, hidden, inter, act_format=fmt, num_sms=num_sms)
    y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    idx, tw = U.random_routing(tokens, e, topk, 51)
    _, inp, sfb = U.make_rank_inputs(tokens, hidden, fmt, 52, idx, tw)
    ref = O.moe_layer_reference([inp], [w], fmt, e, clamp=10.0)
    for case in ('plain', 'masked', 'missing', 'plain'):
        U.write_inputs(buf, inp, sfb)
        if case == 'masked':
            buf.topk_idx.fill_(-1)
        if case == 'missing':
            buf.topk_idx[1, 2] = e
        mm.fp4_fp4_mega_moe(y.fill_(1.0), l1, l2, buf, activation_clamp=10.0, timeout_ms=300.0)
        st, words = buf.device_status()
        if case == 'missing':
            assert st == 4 and (words[0] & 0xFF) == 9
            buf.reset()
        else:
            assert st == 0
        if case == 'plain':
            assert O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL
        if case == 'masked':
            assert float(y.abs().max()) == 0.0


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
@pytest.mark.parametrize('tokens', [1, 2, 3, 160])
@pytest.mark.parametrize('score_mode', [0, 1])
def test_from_hidden_states_in_the_decode_and_batch_kernels(fmt, tokens, score_mode):
    """One and two tokens (decode kernel), three, and more tokens than SMs with four experts per logit block: routing exact,
    the quantised views as the stand-alone frontend writes them, the layer's output against the oracle."""
    e, hidden, inter = 64, 1024, 256
    g = torch.Generator().manual_seed(60 + tokens)
    x = torch.randn((tokens, hidden), generator=g).to(torch.bfloat16)
    if tokens > 1:
        x[1] = 0
    wr = (torch.randn((e, hidden), generator=g) / hidden ** 0.5).to(torch.bfloat16)
    bias = (0.3 * torch.rand(e, generator=g)) if score_mode else None
    w, gs1, gs2 = O.make_expert_weights(e, hidden, inter, fmt, seed=61, std=0.02)
    x_gs, mid_gs = (1.0 / 64.0, 1.0 / 512.0) if fmt == 'nvfp4' else (1.0, 1.0)
    buf = mm.get_symm_buffer_for_mega_moe(None, e, tokens, 8, hidden, inter, act_format=fmt)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    ws = torch.zeros(mm.fe_workspace_bytes(buf), dtype=torch.uint8, device='cuda')
    y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    stats = torch.zeros(e, dtype=torch.int32, device='cuda')
    bias_d = bias.cuda() if bias is not None else None
    mm.mega_moe_from_hidden(y, x.cuda(), wr.cuda(), l1, l2, buf, ws, cumulative_local_expert_recv_stats=stats, activation_clamp=10.0,
                            score_mode=score_mode, expert_bias=bias_d, x_global_scale=x_gs, l1_global_scale=gs1, l2_global_scale=gs2,
                            mid_global_scale=mid_gs, timeout_ms=500.0)
    st, words = buf.device_status()
    assert st == 0, [hex(v) for v in words[:4]]
    idx, tw = O.route_from_logits(O.router_logits_device_order(x, wr), x, 8, 'sigmoid_bias' if score_mode else 'softmax', bias)
    assert torch.equal(buf.topk_idx[:tokens].cpu(), idx) and torch.allclose(buf.topk_weights[:tokens].cpu(), tw, rtol=2e-6, atol=1e-7)
    fused = [t[:tokens].view(torch.uint8).clone() for t in (buf.x, buf.x_sf, buf.topk_weights)]
    for t in (buf.x, buf.x_sf, buf.topk_weights):                 # (what the second call left out would be the first one's)
        t.view(torch.uint8).fill_(0xAA)
    mm.fe_forward_into_buffer(x.cuda(), wr.cuda(), buf, ws, score_mode=score_mode, expert_bias=bias_d, x_global_scale=x_gs)
    assert all(torch.equal(a, t[:tokens].view(torch.uint8)) for a, t in zip(fused, (buf.x, buf.x_sf, buf.topk_weights)))
    q, sf, _ = O.quantise_tokens(x, fmt, rounding='rne', sf_rule='mul', global_scale=x_gs)
    ref = O.moe_layer_reference([O.RankInput(q, sf, idx, tw)], [w], fmt, e, clamp=10.0, x_global_scale=x_gs, w1_global_scale=gs1,
                                w2_global_scale=gs2, mid_global_scale=mid_gs)
    assert torch.equal(stats.cpu(), ref.counts[0])
    assert O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL


@pytest.mark.parametrize('tokens,t_max', [(512, 512), (3, 16), (1, 1)])
def test_more_rows_than_the_buffer_has_room_for_is_reported(tokens, t_max):
    """A buffer has room for tokens x min(routes, experts) rows. Two experts, eight routes each of which names one of them: four
    times as many rows (batch kernel; with one token of a buffer for one token the decode kernel) are refused on the device, as many
    as there is room for (24 rows of 32 here) are served, and the buffer recovers."""
    fmt, e, hidden, inter, topk = 'mxfp4', 2, 512, 256, 8
    w, _, _ = O.make_expert_weights(e, hidden, inter, fmt, seed=71, std=0.05)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    buf = mm.SymmBuffer(None, e, t_max, topk, hidden, inter, act_format=fmt)
    assert int(buf.layout.rx_cap_rows) == 2 * t_max
    full = torch.arange(tokens * topk).reshape(tokens, topk) % e
    weights = torch.full((tokens, topk), 0.125)
    _, inp, sfb = U.make_rank_inputs(tokens, hidden, fmt, 72, full, weights)
    y = torch.zeros((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    U.write_inputs(buf, inp, sfb)
    before = buf.inputs.clone()
    mm.fp4_fp4_mega_moe(y, l1, l2, buf, timeout_ms=500.0)
    st, words = buf.device_status()
    if tokens * topk <= 2 * t_max:
        ref = O.moe_layer_reference([inp], [w], fmt, e, clamp=None)
        assert st == 0 and O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL
        return
    assert st == 5 and (words[0] & 0xFF) == 10 and torch.equal(buf.inputs, before)
    buf.reset()
    inp.topk_idx[:, 2:] = -1                                       # one row per token and expert
    ref = O.moe_layer_reference([inp], [w], fmt, e, clamp=None)
    U.write_inputs(buf, inp, sfb)
    for _ in range(2):
        mm.fp4_fp4_mega_moe(y, l1, l2, buf, timeout_ms=500.0)
        assert buf.device_status()[0] == 0 and O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL


@pytest.mark.parametrize('between', [20, 3])
def test_a_launch_that_fails_at_routing_leaves_clean_counters(between):
    """The launch after one that failed (a route to a missing expert, in a batch-size and in a decode-size launch) counts in the set
    that the failed launch had to clear: its results are right without a reset. The status keeps the first failure."""
    fmt, e, hidden, inter, topk, tokens = 'mxfp4', 4, 512, 256, 2, 20
    w, l1, l2, buf, inp, sfb = _small_layer(fmt, e, hidden, inter, topk, tokens, 925)
    y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    for it in range(4):
        idx, tw = U.random_routing(tokens, e, topk, 926 + it)
        _, inp, sfb = U.make_rank_inputs(tokens, hidden, fmt, 930 + it, idx, tw)
        ref = O.moe_layer_reference([inp], [w], fmt, e, clamp=None)
        U.write_inputs(buf, inp, sfb)
        mm.fp4_fp4_mega_moe(y, l1, l2, buf, timeout_ms=500.0)
        torch.cuda.synchronize()
        assert O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL, it
        buf.topk_idx[1, 1] = e
        mm.fp4_fp4_mega_moe(torch.empty((between, hidden), dtype=torch.bfloat16, device='cuda'), l1, l2, buf, timeout_ms=500.0)
        st, words = buf.device_status()
        assert st == 4 and (words[0] & 0xFF) == 9


def _exact_sum_weights(e, n, k, fmt, g):
    """Random E2M1 codes under scales that are powers of two close together: every sum of products is exact, in any order."""
    q = torch.randint(0, 256, (e, n, k // 2), generator=g).to(torch.uint8)
    vec = 16 if fmt == 'nvfp4' else 32
    sf = torch.randint(0, 3, (e, n, k // vec), generator=g)
    words = (((sf + 5) * 8) if fmt == 'nvfp4' else sf + 120).to(torch.uint8).view(torch.int32)
    sf_mn = torch.empty((e, words.shape[-1], n), dtype=torch.int32).permute(0, 2, 1)
    sf_mn.copy_(words)
    return q.view(torch.int8).cuda(), sf_mn.cuda()


@pytest.mark.parametrize('tokens', [2, 23])                     # the decode and the batch kernel
@pytest.mark.parametrize('fmt,weights,scales', [
    ('mxfp4', 'plain', (1.0, 1.0, 1.0, 1.0)), ('mxfp4', 'odd', (1.0, 1.0, 1.0, 1.0)), ('fp8', 'plain', None), ('fp8', 'odd', None),
    ('nvfp4', 'plain', (1.0 / 64, 1.0 / 64, 1.0, 1.0 / 512)),
    ('nvfp4', 'plain', (1.0 / 64, 1.0 / 64, 1.0, 0.0123)),       # a divisor that is no power of two
    ('nvfp4', 'plain', (1.0 / 64, 1.0 / 8, 1.0, 1e-3)),          # gates far below zero: outputs that are zeros of either sign
    ('nvfp4', 'plain', (1.0 / 64, 0.22, 1.0, 1.0 / 512)),        # ... and about where exp(-gate) leaves fp32
    ('nvfp4', 'plain', (1e10, 1e9, 1e-9, 1.0)),                  # outputs beyond fp32
    ('nvfp4', 'plain', (1.0, 1e15, 1.0, 1e-15)),                 # quotients beyond fp32
    ('nvfp4', 'plain', (1.0, 1.0, 1.0, 3e-39)), ('nvfp4', 'plain', (1.0, 1.0, 1.0, 1e38)),         # divisors without a normal reciprocal
    ('nvfp4', 'plain', (1e-12, 1e-10, 1.0, 1e-20)),              # quotients around the smallest ones that are corrected
    ('nvfp4', 'odd', (1.0 / 64, 1.0 / 64, 1.0, 1.0 / 512)),
])
@pytest.mark.parametrize('fast_math', [True, False])
def test_intermediate_rows_equal_those_of_the_multi_rank_kernel(fmt, weights, scales, tokens, fast_math):
    """The one-rank kernels' SwiGLU and requantisation take other instructions than the general kernel (a refined reciprocal, division by
    a known divisor). From the same accumulators they give the same bytes, also for zeros, infinities and NaN."""
    e, topk, hidden, inter = 8, 4, 512, 256
    g = torch.Generator().manual_seed(80 + tokens)
    l1, l2 = mm.transform_weights_for_mega_moe(_exact_sum_weights(e, 2 * inter, hidden, fmt, g), _exact_sum_weights(e, hidden, inter, fmt, g))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, 32, topk, hidden, inter, act_format=fmt)
    idx, tw = U.random_routing(tokens, e, topk, 81)
    if weights == 'odd':
        special = torch.tensor([float('nan'), float('inf'), -float('inf'), 0.0, -0.0, -1e20, 1e-36, -1.0])
        tw = special[torch.randint(0, len(special), tw.shape, generator=g)]
    if fmt == 'fp8':
        xq = torch.randint(-4, 5, (tokens, hidden), generator=g).float().to(torch.float8_e4m3fn).view(torch.uint8)
        sfb = torch.full((tokens, hidden // 32), 127)
    else:
        xq = torch.randint(0, 256, (tokens, hidden // 2), generator=g).to(torch.uint8)
        sfb = torch.full((tokens, hidden // 32), 121) if fmt == 'mxfp4' else torch.full((tokens, hidden // 16), 5 * 8)
    lib, got = _lib.load(), []
    knobs = lib.mm_get_tuning(_lib.TUNE['knobs'])
    kw = dict(zip(('x_global_scale', 'l1_global_scale', 'l2_global_scale', 'mid_global_scale'), scales)) if scales else {}
    try:
        for k in (knobs, knobs & ~(16 | 64)):                    # (without the tile images and the decode kernel: the multi-rank kernel)
            mm.set_tuning(knobs=k)
            buf.x[:tokens].view(torch.uint8).copy_(xq)
            buf.x_sf[:tokens].view(torch.uint8).copy_(sfb.to(torch.uint8))
            buf.topk_idx[:tokens].copy_(idx)
            buf.topk_weights[:tokens].copy_(tw)
            y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
            (mm.fp8_fp4_mega_moe if fmt == 'fp8' else mm.fp4_fp4_mega_moe)(y, l1, l2, buf, fast_math=fast_math, timeout_ms=500.0, **kw)
            assert buf.device_status()[0] == 0
            recs = buf.received_records()[0]
            rows, sf = buf.l2_acts_payload().cpu(), buf.l2_acts_sf_payload().cpu()[:, :inter // (16 if fmt == 'nvfp4' else 32)]
            live, base = [], 0
            for ex in range(e):
                n = sum(1 for r in recs if r[0] == ex)
                live += range(base, base + n)
                base += (n + 15) // 16 * 16
            got.append((y.view(torch.int16).cpu(), rows[live], sf[live]))
    finally:
        mm.set_tuning(knobs=knobs)
    for a, b, what in zip(got[0], got[1], ('y', 'codes', 'scale bytes')):
        assert a.shape == b.shape and torch.equal(a, b), (what, int((a != b).sum()), a.numel())


@pytest.mark.parametrize('fmt', ['mxfp4', 'fp8'])
@pytest.mark.parametrize('num_sms,tokens', [(1, 1), (1, 2), (2, 2), (1, 3)])
def test_from_hidden_states_on_one_or_two_sms_fills_every_view(fmt, num_sms, tokens):
    """The routing and the quantised tokens land in the buffer's views whatever the grid: fewer SMs than tokens, in both kernels."""
    e, hidden, inter = 8, 512, 256
    g = torch.Generator().manual_seed(90)
    x = torch.randn((tokens, hidden), generator=g).to(torch.bfloat16).cuda()
    wr = (torch.randn((e, hidden), generator=g) / hidden ** 0.5).to(torch.bfloat16).cuda()
    w, _, _ = O.make_expert_weights(e, hidden, inter, fmt, seed=91, std=0.02)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, 16, 8, hidden, inter, act_format=fmt, num_sms=num_sms)
    ws = torch.zeros(mm.fe_workspace_bytes(buf), dtype=torch.uint8, device='cuda')
    y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    views = (buf.x, buf.x_sf, buf.topk_idx, buf.topk_weights)
    for v in views:
        v.view(torch.uint8).fill_(0x55)
    mm.mega_moe_from_hidden(y, x, wr, l1, l2, buf, ws, timeout_ms=500.0)
    assert buf.device_status()[0] == 0
    got = [v[:tokens].view(torch.uint8).clone() for v in views]
    for v in views:
        v.view(torch.uint8).fill_(0xAA)
    mm.fe_forward_into_buffer(x, wr, buf, ws)
    for a, v in zip(got, views):
        assert torch.equal(a, v[:tokens].view(torch.uint8))


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
@pytest.mark.parametrize('tokens,e,hidden', [
    (1, 16, 4096), (2, 48, 512), (3, 48, 4096),                       # one token to an item: rows of one and of eight chunks a lane, more than are in flight
    (24, 48, 512), (25, 48, 1536), (148, 48, 512), (149, 48, 1024),   # both sides of the lines between the item sizes (on 148 SMs)
    (256, 16, 512), (256, 64, 1024),
])
def test_frontend_of_the_one_rank_kernels_matches_the_stand_alone_one(fmt, tokens, e, hidden):
    """Routing and quantised tokens, bit for bit, whatever the items the partial logits are cut into; routing and quantised tokens of the oracle."""
    g = torch.Generator().manual_seed(190 + tokens)
    x = torch.randn((tokens, hidden), generator=g).to(torch.bfloat16)
    x[tokens // 2] = 0
    x = x.cuda()
    wr = (torch.randn((e, hidden), generator=g) / hidden ** 0.5).to(torch.bfloat16).cuda()
    inter = 256
    stream = lambda n, k: (torch.zeros((e, n // 128, k // 256, 18432 if fmt == 'nvfp4' else 17408), dtype=torch.uint8, device='cuda'),      # noqa: E731
                           torch.tensor([n, k, 16 if fmt == 'nvfp4' else 32]))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, tokens, 8, hidden, inter, act_format=fmt)
    ws = torch.zeros(mm.fe_workspace_bytes(buf), dtype=torch.uint8, device='cuda')
    y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    kw = dict(x_global_scale=1.0 / 64.0) if fmt == 'nvfp4' else {}
    views = (buf.x, buf.x_sf, buf.topk_idx, buf.topk_weights)
    for v in views:
        v.view(torch.uint8).fill_(0x55)
    mm.mega_moe_from_hidden(y, x, wr, stream(2 * inter, hidden), stream(hidden, inter), buf, ws, timeout_ms=500.0, **kw)
    assert buf.device_status()[0] == 0
    got = [v[:tokens].view(torch.uint8).clone() for v in views]
    idx, _ = O.route_from_logits(O.router_logits_device_order(x.cpu(), wr.cpu()), x.cpu(), 8)
    assert torch.equal(buf.topk_idx[:tokens].cpu(), idx)
    q, _, sfb = O.quantise_tokens(x.cpu(), fmt, rounding='rne', sf_rule='mul', global_scale=kw.get('x_global_scale', 1.0))
    assert torch.equal(_canon(got[0].cpu(), fmt), _canon(q, fmt)) and torch.equal(got[1].cpu().view(tokens, -1), sfb)
    for v in views:
        v.view(torch.uint8).fill_(0xAA)
    mm.fe_forward_into_buffer(x, wr, buf, ws, **kw)
    for a, v in zip(got, views):
        assert torch.equal(a, v[:tokens].view(torch.uint8))


MULTI_RANK, BATCH, DECODE = 1, 2, 3             # status word 4


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
@pytest.mark.parametrize('topk,tokens,hidden,inter,kernel', [
    (1, 1, 512, 256, DECODE), (1, 16, 512, 512, DECODE), (8, 2, 1024, 256, DECODE), (5, 3, 512, 2048, DECODE), (8, 1, 3072, 1280, DECODE),
    (2, 8, 1536, 256, DECODE), (1, 17, 512, 256, BATCH), (8, 3, 1024, 256, BATCH), (16, 256, 2048, 256, BATCH),
])
def test_which_kernel_a_launch_takes(fmt, topk, tokens, hidden, inter, kernel):
    """The dispatch rule at its line (16 routing entries), over the shapes of the decode tests, and with inputs in host memory, which
    stay with the multi-rank kernel; a launch without tokens does too."""
    e = 16
    stream = lambda n, k: (torch.zeros((e, n // 128, k // 256, 18432 if fmt == 'nvfp4' else 17408), dtype=torch.uint8, device='cuda'),      # noqa: E731
                           torch.tensor([n, k, 16 if fmt == 'nvfp4' else 32]))
    l1, l2 = stream(2 * inter, hidden), stream(hidden, inter)
    buf = mm.get_symm_buffer_for_mega_moe(None, e, tokens, topk, hidden, inter, act_format=fmt)
    buf.topk_idx[:tokens].copy_(U.random_routing(tokens, e, topk, 100)[0])
    call = mm.fp8_fp4_mega_moe if fmt == 'fp8' else mm.fp4_fp4_mega_moe
    y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    call(y, l1, l2, buf, timeout_ms=500.0)
    st, words = buf.device_status()
    assert st == 0 and words[4] == kernel
    mirror, views = buf.host_inputs()
    views['topk_idx'].fill_(-1)
    for out, kw in ((y, dict(host_inputs=mirror)), (y[:0], {})):
        call(out, l1, l2, buf, timeout_ms=500.0, **kw)
        st, words = buf.device_status()
        assert st == 0 and words[4] == MULTI_RANK


@pytest.mark.parametrize('fmt', ['mxfp4', 'fp8'])
def test_launches_with_mapped_inputs_alternate_with_the_one_rank_kernels(fmt):
    """Inputs in host memory stay with the multi-rank kernel, which shares buffer, launch numbers and counters with the other two."""
    e, hidden, inter, topk = 4, 512, 256, 2
    w, _, _ = O.make_expert_weights(e, hidden, inter, fmt, seed=110, std=0.05)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, 64, topk, hidden, inter, act_format=fmt)
    call = mm.fp8_fp4_mega_moe if fmt == 'fp8' else mm.fp4_fp4_mega_moe
    mirror, views = buf.host_inputs()
    order = [(40, 0), (40, 1), (40, 0), (3, 1), (3, 0), (64, 1), (64, 0), (5, 0), (5, 1), (40, 0), (40, 1), (64, 0), (33, 0), (2, 1), (50, 0)]
    for it, (tokens, mapped) in enumerate(order):
        idx, tw = U.random_routing(tokens, e, topk, 111 + it)
        _, inp, sfb = U.make_rank_inputs(tokens, hidden, fmt, 130 + it, idx, tw)
        ref = O.moe_layer_reference([inp], [w], fmt, e, clamp=None)
        if mapped:
            for name, v in (('x', inp.x_q.view(buf.x.dtype)), ('x_sf', sfb.contiguous().view(torch.int32)), ('topk_idx', idx), ('topk_weights', tw)):
                views[name].view(torch.uint8)[:tokens].copy_(v.contiguous().view(torch.uint8))
        else:
            U.write_inputs(buf, inp, sfb)
        y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
        call(y, l1, l2, buf, timeout_ms=500.0, **(dict(host_inputs=mirror) if mapped else {}))
        st, words = buf.device_status()
        assert st == 0 and words[1] == it + 1 and words[4] == (MULTI_RANK if mapped else (BATCH if tokens * topk > 16 else DECODE))
        assert O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL, (it, tokens, mapped)


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
def test_partial_sums_of_the_multi_rank_kernel_are_not_taken_for_the_decode_kernels(fmt):
    """The multi-rank kernel keeps plain fp32 sums in the split-tile region: 32 KB per SM, any bit pattern, the next launch's number
    among them. The decode kernel's flagged words lie elsewhere in the region."""
    e, hidden, inter, topk, tokens = 8, 1024, 512, 8, 1
    w, gs1, gs2 = O.make_expert_weights(e, hidden, inter, fmt, seed=150, std=0.05)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, 16, topk, hidden, inter, act_format=fmt)
    idx, tw = U.random_routing(tokens, e, topk, 151)
    _, inp, sfb = U.make_rank_inputs(tokens, hidden, fmt, 152, idx, tw)
    ref = O.moe_layer_reference([inp], [w], fmt, e, clamp=None, w1_global_scale=gs1, w2_global_scale=gs2)
    U.write_inputs(buf, inp, sfb)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    off = int(buf.layout.off_red)
    sums = buf.buffer[off:off + sms * 32768].view(torch.int32)
    y = torch.empty((tokens, hidden), dtype=torch.bfloat16, device='cuda')
    call = mm.fp8_fp4_mega_moe if fmt == 'fp8' else mm.fp4_fp4_mega_moe
    kw = dict(l1_global_scale=gs1, l2_global_scale=gs2) if fmt == 'nvfp4' else {}
    for launch in range(1, 9):
        sums.fill_(launch)
        call(y, l1, l2, buf, timeout_ms=500.0, **kw)
        st, words = buf.device_status()
        assert st == 0 and words[4] == DECODE and words[1] == launch
        assert bool((sums == launch).all()) and O.rel_rmse(y.cpu(), ref.y[0]) <= REL_RMSE_TOL


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
def test_first_weight_request_of_the_decode_kernel(fmt):
    """Slot 13 of the stamps and slot 5 of an SM's record are the times of a weight request, not of the routing: an SM that asks for no
    weights has none, whatever the launch before it left there, nor has a launch that fails at routing."""
    e, hidden, inter, topk = 8, 512, 256, 2
    w, _, _ = O.make_expert_weights(e, hidden, inter, fmt, seed=170, std=0.05)
    l1, l2 = mm.transform_weights_for_mega_moe(*U.to_operator_weights(w, fmt, 'cuda'))
    buf = mm.get_symm_buffer_for_mega_moe(None, e, 16, topk, hidden, inter, act_format=fmt)
    call = mm.fp8_fp4_mega_moe if fmt == 'fp8' else mm.fp4_fp4_mega_moe
    y = torch.empty((1, hidden), dtype=torch.bfloat16, device='cuda')
    idx, tw = U.random_routing(1, e, topk, 171)
    _, inp, sfb = U.make_rank_inputs(1, hidden, fmt, 172, idx, tw)
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def launch(route):
        U.write_inputs(buf, inp, sfb)
        if route is not None:
            buf.topk_idx[:1] = route
        call(y, l1, l2, buf, timeout_ms=500.0)
        st, words = buf.device_status()
        assert words[4] == DECODE
        return st, buf.phase_stamps(), buf.sm_phases()[:sms]

    st, s, ph = launch(-1)                                          # no unit on any SM
    assert st == 0 and s[13] == 0 and bool((ph[:, 5] == 0).all())
    st, s, ph = launch(None)                                        # eight L1 tiles of two units, eight L2 tiles of one: part of the SMs
    on = ph[:, 5] != 0
    assert st == 0 and 0 < int(on.sum()) < sms and int(ph[on, 5].min()) == s[13]
    assert bool((ph[on, 4] <= ph[on, 5]).all()) and bool((ph[on, 5] <= ph[on, 6]).all())       # scheduled, requested, landed
    assert s[12] <= s[13] <= s[14] <= s[8]
    st, s, _ = launch(-1)
    assert st == 0 and s[13] == 0
    launch(None)
    st, s, _ = launch(e)                                            # no such expert
    assert st == 4 and s[13] == 0
