"""CPU-side checks: the library loads and exports the declared C ABI, the buffer layout, the weight pre-tiling."""
import ctypes
import os
import re

import pytest
import torch

import hopper_megamoe_basedondeepgemm_b200 as mm
from hopper_megamoe_basedondeepgemm_b200 import _lib, quant
from oracle import megamoe_oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_library_exports_every_declared_symbol():
    lib = _lib.load()
    header = open(os.path.join(ROOT, 'include', 'megamoe_b200.h')).read()
    declared = set(re.findall(r'\b(mm_[a-z0-9_]+)\s*\(', header))
    assert declared == set(_lib.EXPORTS)
    for name in declared:
        assert getattr(lib, name) is not None


def _layout(**kw):
    lib = _lib.load()
    cfg = _lib.MMConfig(kw.get('ranks', 8), kw.get('rank', 0), kw.get('experts', 384), kw.get('tmax', 128), 8,
                        kw.get('hidden', 3072), kw.get('inter', 1280), _lib.FMT[kw.get('fmt', 'mxfp4')], 148)
    L = _lib.MMLayout()
    return lib.mm_get_layout(ctypes.byref(cfg), ctypes.byref(L)), L


def test_layout_regions_are_ordered_and_sized():
    st, L = _layout()
    assert st == 0
    offs = [L.off_ctrl, L.off_x, L.off_x_sf, L.off_topk_idx, L.off_topk_weights, L.off_rx, L.off_mid,
            L.off_mid_sf, L.off_comb, L.off_red, L.off_cnt, L.off_logits, L.off_token_tiles, L.off_mid_tiles, L.off_arrive,
            L.total_bytes]
    assert offs == sorted(offs) and all(o % 1024 == 0 for o in offs)
    # tile images (launches with more than 16 received rows): one per 16 rows of the intermediate pool at most; per tile 32
    # row records of 16 B (token tiles), then per 256-element K unit a record of 32 rows x 128 B + two scale-word slot planes
    rec32 = 32 * 128 + 2 * 32 * 16
    assert L.tile_capacity == L.mid_rows // 16
    assert L.token_tile_bytes == 32 * 16 + (3072 // 256) * rec32 and L.mid_tile_bytes == (1280 // 256) * rec32
    assert L.off_mid_tiles - L.off_token_tiles >= L.tile_capacity * L.token_tile_bytes
    assert L.off_arrive - L.off_mid_tiles >= L.tile_capacity * L.mid_tile_bytes
    assert L.total_bytes - L.off_arrive >= 2 * 2 * L.tile_capacity * 4
    assert L.x_row_bytes == 1536 and L.x_sf_row_bytes == 96 and L.rx_row_bytes == 1536 + 96 + 16
    assert L.rx_cap_rows == 128 * 8 and L.mid_row_bytes == 640 and L.mid_sf_row_bytes == 48
    assert L.rx_region_bytes >= 32 + 2 * L.rx_cap_rows * L.rx_row_bytes
    assert L.off_mid - L.off_rx >= 2 * 8 * L.rx_region_bytes
    st, L2 = _layout(fmt='nvfp4')
    assert st == 0 and L2.x_sf_row_bytes == 192 and L2.mid_sf_row_bytes == 80 and L2.sf_vec == 16


def test_layout_rejects_bad_shapes():
    assert _layout(hidden=3000)[0] == 2        # unsupported
    assert _layout(experts=385)[0] == 1        # invalid: not divisible by ranks
    assert _layout(ranks=16, experts=384)[0] == 1
    assert _layout(ranks=1, experts=384)[0] == 2   # more than 64 local experts
    assert _layout(fmt='fp8')[0] in (0, 2)


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4'])
def test_pretiled_stream_decodes_back_to_the_weights(fmt):
    """Walk the stream with the address arithmetic the kernel uses and recover every weight byte and scale byte."""
    vec = quant.SF_VEC[fmt]
    torch.manual_seed(0)
    e, n, k = 2, 256, 512
    w = (torch.randn(e, n, k) * 0.05).to(torch.bfloat16)
    q, sf_mn = quant.cast_grouped_weights_to_fp4(w, fmt)
    stream = quant.pretile_weights(q, sf_mn, vec)
    planes = 256 // (4 * vec)
    assert stream.shape == (e, n // 128, k // 256, 16384 + planes * 512)
    qb = q.view(torch.uint8)
    sfb = sf_mn.contiguous().view(torch.uint8).reshape(e, n, k // vec)
    for ex in range(e):
        for j in range(n // 128):
            for u in range(k // 256):
                unit = stream[ex, j, u]
                for r in (0, 1, 7, 8, 37, 64, 127):
                    for ci in range(8):
                        off = (r >> 3) * 1024 + (r & 7) * 128 + ((ci ^ (r & 7)) << 4)
                        assert torch.equal(unit[off:off + 16], qb[ex, 128 * j + r, u * 128 + ci * 16:u * 128 + ci * 16 + 16])
                    for pl in range(planes):
                        off = 16384 + pl * 512 + ((r & 31) * 4 + (r >> 5)) * 4
                        g = u * planes + pl
                        assert torch.equal(unit[off:off + 4], sfb[ex, 128 * j + r, 4 * g:4 * g + 4])


def test_product_quantiser_matches_oracle():
    torch.manual_seed(1)
    t = (torch.randn(8, 512) * 0.3).to(torch.bfloat16)
    for fmt in ('mxfp4', 'nvfp4'):
        p, sf, words = quant.cast_rows_to_fp4(t, fmt)
        po, sfo, sfbo = O.quant_fp4_rows(t, fmt, rounding='rne', sf_rule='div')
        assert torch.equal(p.view(torch.uint8), po) and torch.equal(sf, sfo)
        assert torch.equal(words.view(torch.uint8).reshape(8, -1), sfbo)


def test_interleave_matches_reference_rule():
    t = torch.arange(2 * 32).reshape(2, 32, 1)
    out = quant.interleave_gate_up(t)
    # [gate 0..7, up 0..7, gate 8..15, up 8..15]
    assert out[0, :, 0].tolist() == list(range(0, 8)) + list(range(16, 24)) + list(range(8, 16)) + list(range(24, 32))


def test_transform_weights_shapes():
    torch.manual_seed(2)
    w1 = (torch.randn(2, 512, 512) * 0.05).to(torch.bfloat16)
    w2 = (torch.randn(2, 512, 256) * 0.05).to(torch.bfloat16)
    l1, l2 = mm.transform_weights_for_mega_moe(quant.cast_grouped_weights_to_fp4(w1, 'mxfp4'),
                                               quant.cast_grouped_weights_to_fp4(w2, 'mxfp4'))
    assert l1[0].shape == (2, 4, 2, 17408) and l1[1].tolist() == [512, 512, 32]
    assert l2[0].shape == (2, 4, 1, 17408) and l2[1].tolist() == [512, 256, 32]


def test_ctypes_mirror_matches_the_header(tmp_path):
    """Compile a C program against include/megamoe_b200.h and compare every struct's size and field offsets with the
    ctypes mirror the Python binding uses."""
    import shutil
    import subprocess
    if shutil.which('gcc') is None:
        pytest.skip('no C compiler')
    structs = {'mm_config_t': _lib.MMConfig, 'mm_layout_t': _lib.MMLayout, 'mm_weight_geometry_t': _lib.MMWeightGeometry,
               'mm_launch_args_t': _lib.MMLaunchArgs, 'mm_frontend_args_t': _lib.MMFrontendArgs,
               'mm_static_args_t': _lib.MMStaticArgs}
    header = re.sub(r'/\*.*?\*/', '', open(os.path.join(ROOT, 'include', 'megamoe_b200.h')).read(), flags=re.S)
    lines = ['#include <stdio.h>', '#include <stddef.h>', '#include "megamoe_b200.h"', 'int main(void) {']
    fields = {}
    for cname, ct in structs.items():
        body = re.search(r'typedef struct \w+ \{([^}]*)\} ' + cname + ';', header).group(1)
        names = []
        for decl in body.split(';'):
            decl = decl.strip()
            if not decl:
                continue
            for part in decl.split(','):
                names.append(re.findall(r'[A-Za-z_][A-Za-z0-9_]*', part)[-1])
        fields[cname] = names
        lines.append(f'printf("{cname} %zu\\n", sizeof({cname}));')
        for f in names:
            lines.append(f'printf("{cname}.{f} %zu\\n", offsetof({cname}, {f}));')
    lines += ['return 0;', '}']
    src = tmp_path / 'abi.c'
    src.write_text('\n'.join(lines))
    exe = tmp_path / 'abi'
    subprocess.run(['gcc', '-I', os.path.join(ROOT, 'include'), '-o', str(exe), str(src)], check=True)
    out = dict(line.split() for line in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.splitlines())
    for cname, ct in structs.items():
        assert int(out[cname]) == ctypes.sizeof(ct), cname
        mirror = [f[0] for f in ct._fields_]
        assert mirror == fields[cname], (cname, mirror, fields[cname])
        for f in mirror:
            assert int(out[f'{cname}.{f}']) == getattr(ct, f).offset, (cname, f)


def test_frontend_rejects_fewer_experts_than_routes():
    """Eight routes per token cannot be drawn from fewer than eight experts: refused on the host, before any launch."""
    lib = _lib.load()
    cfg = _lib.MMConfig(1, 0, 4, 16, 8, 512, 256, _lib.FMT['mxfp4'], 148)
    dummy = ctypes.c_void_p(0x1000)                                  # never dereferenced: the argument check fails first
    fe = _lib.MMFrontendArgs(dummy, dummy, None, 4, 0, dummy, 1.0)
    assert lib.mm_frontend_launch(ctypes.byref(cfg), dummy, ctypes.byref(fe), None) == 1
    peers = (ctypes.c_void_p * 1)(0x1000)
    la = _lib.MMLaunchArgs(dummy, peers, dummy, dummy, dummy, 4, 0, None, -1.0, 1, 1.0, 1.0, 1.0, 1.0, 0.0, None)
    assert lib.mm_mega_moe_from_hidden_launch(ctypes.byref(cfg), ctypes.byref(la), ctypes.byref(fe), None) == 1


def test_tuning_values_round_trip():
    lib = _lib.load()
    old = lib.mm_get_tuning(_lib.TUNE['stages'])
    assert lib.mm_set_tuning(_lib.TUNE['stages'], 6) == 0 and lib.mm_get_tuning(_lib.TUNE['stages']) == 6
    assert lib.mm_set_tuning(_lib.TUNE['stages'], old) == 0
    assert lib.mm_set_tuning(99, 1) == 1 and lib.mm_set_tuning(0, -1) == 1 and lib.mm_get_tuning(99) == -1


@pytest.mark.parametrize('tw,vec', [(16, 32), (32, 32), (32, 16)])
def test_tile_image_reader_inverts_the_documented_layout(tw, vec):
    """Tile images (launches with more than 16 received rows): per 256-element K unit a record of `tw` rows x 128 B in
    the 128 B swizzle (16 B chunk c of row r at chunk c ^ (r & 7) of the row's 128 B, rows in groups of 8 x 128 B), then
    per scale word of the unit `tw` slots of 16 B with the word in the first 4 bytes. Images written with that address
    arithmetic are read back row by row by `SymmBuffer._rows_of_tile_images`."""
    from types import SimpleNamespace
    from hopper_megamoe_basedondeepgemm_b200.mega import SymmBuffer
    torch.manual_seed(tw + vec)
    row_bytes, tiles, header = 640, 3, 512
    units, planes = row_bytes // 128, 256 // (4 * vec)
    rec = tw * 128 + planes * tw * 16
    rows = torch.randint(0, 256, (tiles * tw, row_bytes), dtype=torch.uint8)
    words = torch.randint(0, 256, (tiles * tw, units * planes, 4), dtype=torch.uint8)
    img = torch.zeros((tiles, header + units * rec), dtype=torch.uint8)
    for t in range(tiles):
        for r in range(tw):
            for ci in range(row_bytes // 16):
                off = header + (ci >> 3) * rec + (r >> 3) * 1024 + (r & 7) * 128 + (((ci & 7) ^ (r & 7)) << 4)
                img[t, off:off + 16] = rows[t * tw + r, ci * 16:ci * 16 + 16]
            for g in range(units * planes):
                off = header + (g // planes) * rec + tw * 128 + (g % planes) * tw * 16 + r * 16
                img[t, off:off + 4] = words[t * tw + r, g]
    fake = SimpleNamespace(layout=SimpleNamespace(sf_vec=vec))
    got_rows, got_words = SymmBuffer._rows_of_tile_images(fake, img, row_bytes, tw, header)
    assert torch.equal(got_rows, rows) and torch.equal(got_words, words)


def _closed_form_schedule(nt, k, g):
    """The kernel's per-SM task list of one phase (`build_schedule` in csrc/mm_kernel.cuh), restated: NT weight-tile
    tasks of k units on G SMs. The first r = NT mod G tiles are split along K: tile t of them is shared by the SMs
    [ceil(t G / r), ceil((t + 1) G / r)), each taking one contiguous unit range (sizes differ by at most one); SM b
    then runs the whole tiles r + b, r + b + G, ... Returns per SM a list of (tile, first unit, end unit, parts)."""
    r = nt % g
    out = []
    for b in range(g):
        tasks = []
        if r:
            t = b * r // g
            gs, ge = -(-t * g // r), -(-(t + 1) * g // r)
            s, li = ge - gs, b - gs
            base, extra = k // s, k % s
            ub = li * base + min(li, extra)
            ue = ub + base + (1 if li < extra else 0)
            if ue > ub:
                tasks.append((t, ub, ue, min(s, k)))
        tasks += [(t, 0, k, 1) for t in range(r + b, nt, g)]
        out.append(tasks)
    return out


@pytest.mark.parametrize('g', [148, 132, 8])
def test_closed_form_schedule_covers_every_unit_once(g):
    """Every (tile, unit) of a phase is owned by exactly one SM, the parts of a split tile are contiguous ranges that
    agree on their count, and the SMs' unit totals differ by at most one tile's units (the arithmetic the kernel's
    scheduler runs per SM, for 16- and 32-row token tiles alike: only the number of tiles changes)."""
    for n_tiles, k in ((20, 12), (24, 5), (3, 7)):
        for m in list(range(1, 20)) + [48, 96, 113]:
            nt = m * n_tiles
            sched = _closed_form_schedule(nt, k, g)
            owner = {}
            parts = {}
            for b, tasks in enumerate(sched):
                assert sum(1 for t in tasks if t[3] > 1) <= 1          # at most one partial task per SM and phase
                for (t, ub, ue, np_) in tasks:
                    assert 0 <= ub < ue <= k
                    parts.setdefault(t, set()).add(np_)
                    for u in range(ub, ue):
                        assert (t, u) not in owner, (m, t, u)
                        owner[(t, u)] = b
            assert len(owner) == nt * k
            assert all(len(v) == 1 for v in parts.values())
            for t, v in parts.items():
                assert sum(1 for tasks in sched for x in tasks if x[0] == t) == next(iter(v))
            loads = [sum(ue - ub for (_, ub, ue, _) in tasks) for tasks in sched]
            assert max(loads) - min(loads) <= k


def test_global_scale_helper_refuses_host_tensors():
    """`nvfp4_global_scale` runs the library's reduction kernel: there is no CPU path, a host tensor is an error."""
    import hopper_megamoe_basedondeepgemm_b200 as mm
    with pytest.raises(RuntimeError):
        mm.nvfp4_global_scale(torch.ones(8))
    lib = _lib.load()
    assert lib.mm_tensor_absmax(None, 1, 8, None, None) == 1        # invalid argument: null pointers


class _RecordingLibrary:
    """Stands in for the C library behind the launch functions: remembers what it was called with."""
    def __init__(self):
        self.calls = []

    def mm_mega_moe_launch(self, cfg, args, stream):
        self.calls.append(('layer', args))
        return 0

    def mm_mega_moe_from_hidden_launch(self, cfg, args, fe, stream):
        self.calls.append(('hidden', args, fe))
        return 0

    def mm_fe_forward(self, *a):
        self.calls.append(('frontend', a))
        return 0


@pytest.fixture
def launches(monkeypatch):
    """A factory of small one-rank buffers in host memory, and the launches made on them (recorded, not run)."""
    from types import SimpleNamespace
    from hopper_megamoe_basedondeepgemm_b200 import mega
    lib = _RecordingLibrary()
    real_load = _lib.load
    monkeypatch.setattr(torch.Tensor, 'cuda', lambda self, *a, **k: self)
    monkeypatch.setattr(torch.cuda, 'synchronize', lambda *a, **k: None)
    monkeypatch.setattr(torch.Tensor, 'is_pinned', lambda self, *a, **k: True)
    monkeypatch.setattr(mega, '_current_stream', lambda: 0)
    real_empty = torch.empty
    monkeypatch.setattr(torch, 'empty', lambda *a, **k: real_empty(*a, **{x: v for x, v in k.items() if x != 'device'}))

    def make(fmt='mxfp4', experts=8, topk=8, hidden=512, inter=256):
        monkeypatch.setattr(_lib, 'load', real_load)
        buf = mega.SymmBuffer(None, experts, 16, topk, hidden, inter, act_format=fmt, num_sms=148)
        unit = 18432 if fmt == 'nvfp4' else 17408
        vec = 16 if fmt == 'nvfp4' else 32
        w = lambda n, k: (torch.zeros((experts, n // 128, k // 256, unit), dtype=torch.uint8), torch.tensor([n, k, vec]))      # noqa: E731
        monkeypatch.setattr(_lib, 'load', lambda check=False: lib)
        return buf, w(2 * inter, hidden), w(hidden, inter), torch.zeros((4, hidden), dtype=torch.bfloat16)
    return SimpleNamespace(make=make, calls=lib.calls)


def test_a_destroyed_buffer_is_not_launched_on(launches):
    """`destroy` gives the memory back: no call may hand its address to a kernel afterwards."""
    for fmt, call in (('mxfp4', mm.fp4_fp4_mega_moe), ('fp8', mm.fp8_fp4_mega_moe)):
        buf, l1, l2, y = launches.make(fmt)
        call(y, l1, l2, buf)
        assert launches.calls[-1][1].buffer == buf.buffer.data_ptr()
        n = len(launches.calls)
        buf.destroy()
        with pytest.raises((AttributeError, RuntimeError)):
            call(y, l1, l2, buf)
        assert len(launches.calls) == n
    buf, l1, l2, y = launches.make()
    router, ws = torch.zeros((8, 512), dtype=torch.bfloat16), torch.zeros(buf._fe_workspace_bytes, dtype=torch.uint8)
    mm.mega_moe_from_hidden(y, y.clone(), router, l1, l2, buf, ws)
    n = len(launches.calls)
    buf.destroy()
    with pytest.raises((AttributeError, RuntimeError)):
        mm.mega_moe_from_hidden(y, y.clone(), router, l1, l2, buf, ws)
    assert len(launches.calls) == n


def test_weights_are_checked_in_every_call(launches):
    """The same tensors with other contents: what a first call would refuse, a later one refuses too."""
    def changed(change):
        buf, l1, l2, y = launches.make()
        mm.fp4_fp4_mega_moe(y, l1, l2, buf)
        n = len(launches.calls)
        change(l1[0], l1[1], l2[0], l2[1])
        with pytest.raises(RuntimeError):
            mm.fp4_fp4_mega_moe(y, l1, l2, buf)
        assert len(launches.calls) == n
    changed(lambda w1, s1, w2, s2: w1.resize_(7, *w1.shape[1:]))
    changed(lambda w1, s1, w2, s2: w2.set_(w2[:4].clone()))
    changed(lambda w1, s1, w2, s2: w1.transpose_(0, 1))
    changed(lambda w1, s1, w2, s2: setattr(w1, 'data', torch.zeros(w1.shape, dtype=torch.int8)))
    changed(lambda w1, s1, w2, s2: s1.fill_(1))
    changed(lambda w1, s1, w2, s2: s2[0].add_(128))


def test_recipes_that_are_taken_and_refused(launches):
    """None stands for the format's own recipe in the W4A4 call; the A-FP8 call has a default and takes no None."""
    for fmt, call, vec in (('mxfp4', mm.fp4_fp4_mega_moe, 32), ('nvfp4', mm.fp4_fp4_mega_moe, 16), ('fp8', mm.fp8_fp4_mega_moe, 32)):
        buf, l1, l2, y = launches.make(fmt)
        call(y, l1, l2, buf)
        call(y, l1, l2, buf, recipe=[1, 1, vec])
        n = len(launches.calls)
        for wrong in ((1, 1, 64), (2, 1, vec), (1, 1)) + ((None,) if fmt == 'fp8' else ()):
            with pytest.raises((RuntimeError, AssertionError, TypeError, IndexError)):
                call(y, l1, l2, buf, recipe=wrong)
        assert len(launches.calls) == n


def test_from_hidden_states_takes_outputs_of_any_shape_with_a_row_per_token(launches):
    """The output of the from-hidden call is asked for its rows and its size, not for the shape of the hidden states; one with no room
    for every row is refused."""
    buf, l1, l2, y = launches.make()
    hidden, router, ws = y.clone(), torch.zeros((8, 512), dtype=torch.bfloat16), torch.zeros(buf._fe_workspace_bytes, dtype=torch.uint8)
    for out in (y, y.view(4, 1, 512), y.view(4, 8, 64), torch.zeros((4, 520), dtype=torch.bfloat16)):
        mm.mega_moe_from_hidden(out, hidden, router, l1, l2, buf, ws)
        assert launches.calls[-1][1].y == out.data_ptr() and launches.calls[-1][1].num_tokens == 4
    n = len(launches.calls)
    for out in (y[:3], torch.zeros((4, 256), dtype=torch.bfloat16)):
        with pytest.raises(RuntimeError):
            mm.mega_moe_from_hidden(out, hidden, router, l1, l2, buf, ws)
    assert len(launches.calls) == n


@pytest.mark.parametrize('number', [lambda v: v, str, lambda v: torch.tensor(v)])
def test_numbers_are_taken_in_every_form_that_converts(launches, number):
    """Scales, clamp and time limit in whatever float() takes; the frontend's mode and cache hint in whatever int() does."""
    buf, l1, l2, y = launches.make('nvfp4')
    scales = dict(x_global_scale=number(0.25), l1_global_scale=number(0.5), l2_global_scale=number(2.0), mid_global_scale=number(4.0))
    router, ws = torch.zeros((8, 512), dtype=torch.bfloat16), torch.zeros(buf._fe_workspace_bytes, dtype=torch.uint8)
    mm.fp4_fp4_mega_moe(y, l1, l2, buf, activation_clamp=number(8.0), timeout_ms=number(100.0), **scales)
    mm.mega_moe_from_hidden(y, y.clone(), router, l1, l2, buf, ws, activation_clamp=number(8.0), timeout_ms=number(100.0), **scales)
    for c in launches.calls:
        a = c[1]
        assert (a.x_global_scale, a.l1_global_scale, a.l2_global_scale, a.mid_global_scale) == (0.25, 0.5, 2.0, 4.0)
        assert a.activation_clamp == 8.0 and a.timeout_ms == 100.0
    assert launches.calls[1][2].x_global_scale == 0.25
    sf, idx, tw = torch.zeros((4, 8), dtype=torch.int32), torch.zeros((4, 8), dtype=torch.int64), torch.zeros((4, 8))
    mm.fe_forward(y, router, torch.zeros((4, 256), dtype=torch.int8), sf, idx, tw, ws, torch.tensor(4.0), number(1.0) if number is not str else '1')
    assert launches.calls[-1][1][12:14] == (4, 1) and all(type(v) is int for v in launches.calls[-1][1][12:14])


@pytest.mark.parametrize('fmt', ['mxfp4', 'nvfp4', 'fp8'])
@pytest.mark.parametrize('records', [[], None])
def test_intermediate_rows_of_a_batch_launch_without_rows(launches, fmt, records):
    """A launch of the one-rank batch kernel in which every slot is masked (its header line says 0 rows), or one that failed before it
    left a header line: no rows, in the shapes of the others."""
    buf = launches.make(fmt)[0]
    buf.device_status = lambda: (0, [0, 1, 16, 128] + [0] * 12)
    buf.received_records = lambda: [records]
    row = 256 if fmt == 'fp8' else 128
    assert buf.l2_acts_payload().shape == (0, row) and buf.l2_acts_payload().dtype == torch.uint8
    assert buf.l2_acts_sf_payload().shape == (0, 256 // (16 if fmt == 'nvfp4' else 32))


def test_large_buffers_hold_the_one_rank_kernels_regions_for_their_largest_launch_only():
    """The one-rank batch kernel takes at most 4096 routing entries: its expert outputs at the end of the buffer stop growing there, and
    hold every entry of a smaller buffer."""
    for tmax, rows in ((16, 128), (512, 4096), (4096, 4096), (32768, 4096)):
        st, L = _layout(ranks=1, experts=48, tmax=tmax)
        behind = L.total_bytes - (L.off_arrive + 4 * 4 * L.tile_capacity)        # (arrival counts, then other counts and the routing records)
        assert st == 0 and rows * 3072 * 2 <= behind - (2 * 64 * 4 + 256 * 8 * 16) <= rows * 3072 * 2 + 2048
    st, L = _layout(ranks=8)
    assert L.total_bytes - (L.off_arrive + 4 * 4 * L.tile_capacity) <= 2 * 64 * 4 + 256 * 8 * 16 + 2048


def test_tile_images_of_e4m3_tokens_take_the_room_their_one_user_needs():
    """Images with 256 B per E4M3 row and K unit are the one-rank batch kernel's, which takes at most 4096 rows (of 64 experts: 4096 / 16
    groups and one begun group per expert). Several ranks never write images of E4M3 tokens: their buffers keep the 128 B records."""
    rec32 = 32 * 128 + 2 * 32 * 16
    st, L = _layout(ranks=8, fmt='fp8')
    assert st == 0 and L.tile_capacity == L.mid_rows // 16
    assert L.token_tile_bytes == 32 * 16 + 12 * rec32 and L.mid_tile_bytes == 5 * rec32
    for experts, tmax in ((48, 512), (48, 4096), (64, 32768), (3, 1000), (1, 1)):
        st, L = _layout(ranks=1, experts=experts, tmax=tmax, fmt='fp8')
        rows = min(4096, tmax * min(8, experts))
        groups, tiles = rows // 16 + experts, min(128, experts + rows // 64)
        assert st == 0 and L.tile_capacity >= groups and L.tile_capacity <= 4096 // 16 + experts
        assert L.tile_capacity * L.token_tile_bytes >= 12 * (groups * 2 * 2048 + tiles * 2 * 512)
        assert L.tile_capacity * L.mid_tile_bytes >= 5 * (groups * 2 * 2048 + tiles * 2 * 512)


def _counter_bytes(L, tmax, experts):
    """What lies between the router logits and the tile images: the one-rank batch kernel's counters."""
    return L.off_token_tiles - (L.off_logits + (min(tmax, 256) * experts * 16 + 1023) // 1024 * 1024)


@pytest.mark.parametrize('fmt', ['mxfp4', 'fp8'])
@pytest.mark.parametrize('experts,tmax', [(8, 1), (48, 128), (64, 512), (64, 32768)])
def test_counters_of_the_batch_kernel_are_in_the_buffers_of_one_rank_only(fmt, experts, tmax):
    """Two sets of 128 B lines, one per column block (hidden / 128 <= 32) and two per token tile (at most 128), between the router logits
    and the token tiles. Several ranks have no such kernel: nothing lies there or behind the arrival counts."""
    st, L = _layout(ranks=1, experts=experts, tmax=tmax, fmt=fmt)
    assert st == 0 and 2 * (32 + 2 * 128) * 128 <= _counter_bytes(L, tmax, experts) <= 80 * 1024 and L.off_token_tiles % 1024 == 0
    for ranks in (2, 8):
        st, L = _layout(ranks=ranks, experts=experts * ranks, tmax=tmax, fmt=fmt)
        assert st == 0 and _counter_bytes(L, tmax, experts * ranks) == 0
        assert L.total_bytes - L.off_arrive == (16 * L.tile_capacity + 1023) // 1024 * 1024


def test_the_static_scratch_has_room_for_the_counters_beside_24_mib():
    """Configurations that need 24 MiB or less without the batch kernel's counters are served by the launch without any allocation."""
    lib, near = _lib.load(), 0
    header = open(os.path.join(ROOT, 'include', 'megamoe_b200.h')).read()
    expr = re.search(r'#define MM_STATIC_SCRATCH_BYTES (.*)', header).group(1).replace('ll', '')
    assert eval(expr) == _lib.STATIC_SCRATCH_BYTES
    shapes = [(fmt, e, h, i, k, t) for fmt in ('mxfp4', 'nvfp4', 'fp8') for e in (1, 2, 8, 20, 32, 48, 64) for h in range(512, 4097, 512)
              for i in range(256, 4097, 256) for k in (1, 2, 4, 6, 8, 16) for t in (1, 8, 16, 32, 64, 128, 256, 512)]
    for fmt, e, h, i, k, t in [('mxfp4', 8, 1536, 512, 8, 128), ('mxfp4', 32, 4096, 2048, 2, 128)] + shapes:
        cfg, L = _lib.MMConfig(1, 0, e, t, k, h, i, _lib.FMT[fmt], 148), _lib.MMLayout()
        assert lib.mm_get_layout(ctypes.byref(cfg), ctypes.byref(L)) == 0
        if L.total_bytes - _counter_bytes(L, t, e) <= 24 * 1024 * 1024:
            near += L.total_bytes > 24 * 1024 * 1024
            assert L.total_bytes <= _lib.STATIC_SCRATCH_BYTES, (fmt, e, h, i, k, t, L.total_bytes)
    assert near >= 2


_ROUTE_PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <thread>
#include <vector>
#include "mm_frontend_route.h"
#include "mm_device_attribute.h"
static int known_clusters() {                    // failures are asked again, answers kept unless not to be, by threads in any order
    mm::KnownClusters k;
    int n = -1, asked = 0;
    auto fails = [&](int*) { ++asked; return false; };
    auto seven = [&](int* out) { ++asked; *out = 7; return true; };
    if (k.get(true, &n, fails) || k.get(true, &n, fails) || asked != 2) return 1;
    if (!k.get(false, &n, seven) || n != 7 || asked != 3) return 2;
    if (k.get(true, &n, fails) || asked != 4) return 3;
    if (!k.get(true, &n, seven) || !k.get(true, &n, fails) || n != 7 || asked != 5) return 4;
    if (k.get(false, &n, fails) || asked != 6) return 5;
    mm::KnownClusters none;
    auto zero = [&](int* out) { *out = 0; return true; };
    if (!none.get(true, &n, zero) || !none.get(true, &n, seven) || n != 0 || asked != 6) return 6;
    mm::KnownClusters shared;
    static int attribute;                        // set before the answer is kept: who finds it kept sees it set
    std::atomic<int> bad{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&] {
            for (int i = 0; i < 1000; ++i) {
                int m = 0;
                if (!shared.get(true, &m, [&](int* out) { __atomic_store_n(&attribute, 1, __ATOMIC_RELAXED); *out = 7; return true; }) || m != 7) ++bad;
                if (__atomic_load_n(&attribute, __ATOMIC_RELAXED) != 1) ++bad;
            }
        });
    for (auto& t : threads) t.join();
    return bad.load() == 0 ? 0 : 7;
}
static int device_attribute() {                  // raised by threads in any order, never below what one of them needs
    mm::DeviceAttribute a;
    int sets = 0;
    auto fails = [&] { ++sets; return 7; };
    auto sets_it = [&] { ++sets; return 0; };
    if (a.raise(1, 100, fails) != 7 || a.raise(1, 100, sets_it) != 0 || a.raise(1, 90, fails) != 0 || sets != 2) return 1;
    if (a.raise(2, 90, sets_it) != 0 || a.raise(1, 101, sets_it) != 0 || sets != 4) return 2;
    if (a.raise(-1, 1, fails) != 7 || a.raise(64, 1, sets_it) != 0 || a.raise(64, 1, fails) != 7 || sets != 7) return 3;
    std::atomic<int> bad{0};
    for (int round = 0; round < 200; ++round) {
        mm::DeviceAttribute shared;
        std::atomic<int> now{0};                 // the attribute
        std::vector<std::thread> threads;
        for (int t = 1; t <= 4; ++t)
            threads.emplace_back([&, t] {
                for (int bytes = t; bytes < 40; bytes += 4) {
                    shared.raise(0, bytes, [&] { std::this_thread::yield(); now = bytes; return 0; });
                    if (now < bytes) ++bad;      // (a launch that needs `bytes` would be refused)
                }
            });
        for (auto& t : threads) t.join();
    }
    return bad.load() == 0 ? 0 : 4;
}
struct Fake {                                    // a GPU whose answers are made up; `log`: what was done
    int clusters_; bool query_ok, launch_ok, error = false; char log[64] = {}; int n = 0;
    void put(char c) { log[n++] = c; }
    bool error_pending() { return error; }
    void clear_error() { error = false; put('c'); }
    bool clusters(int* out) { put('q'); if (!query_ok) { error = true; return false; } *out = clusters_; return true; }
    bool one_launch(int per) { put(static_cast<char>('0' + per)); if (!launch_ok) error = true; return launch_ok; }
    int two_launches() { put('T'); return 42; }
};
int main(int argc, char** argv) {                // clusters query_ok launch_ok pending tokens hidden experts grid
    if (argc == 1) return known_clusters();
    if (argc == 2) return device_attribute();
    int a[8];
    for (int i = 0; i < 8; ++i) a[i] = atoi(argv[i + 1]);
    Fake f{a[0], a[1] != 0, a[2] != 0, a[3] != 0};
    const int st = mm::launch_frontend_by_size(f, a[4], a[5], a[6], a[7]);
    printf("%s %d %d\n", f.log, st, f.error ? 1 : 0);
    return 0;
}
"""


@pytest.fixture(scope='module')
def frontend_route(tmp_path_factory):
    import shutil
    import subprocess
    if shutil.which('g++') is None:
        pytest.skip('no C++ compiler')
    d = tmp_path_factory.mktemp('route')
    (d / 'route.cpp').write_text(_ROUTE_PROGRAM)
    csrc = os.path.join(ROOT, 'hopper_megamoe_basedondeepgemm_b200', 'csrc')
    cmd = ['g++', '-std=c++17', '-O1', '-pthread', '-Wall', '-Werror', '-I', csrc, '-o', str(d / 'route'), str(d / 'route.cpp')]
    for sanitizer in (['-fsanitize=thread'], []):                 # (without it where it is not installed or cannot run)
        if subprocess.run(cmd + sanitizer, capture_output=bool(sanitizer)).returncode == 0:
            if not sanitizer or 'FATAL: ThreadSanitizer' not in subprocess.run([str(d / 'route')], capture_output=True, text=True).stderr:
                break

    def run(tokens, hidden=3072, experts=48, grid=148, clusters=7, query_ok=True, launch_ok=True, pending=False):
        args = [clusters, int(query_ok), int(launch_ok), int(pending), tokens, hidden, experts, grid]
        if isinstance(tokens, list):
            return subprocess.run([str(d / 'route')] + tokens, capture_output=True, text=True)
        done, status, error = subprocess.run([str(d / 'route')] + [str(v) for v in args], check=True, capture_output=True, text=True).stdout.split()
        return done, int(status), bool(int(error))
    return run


def test_frontend_takes_two_launches_where_the_clusters_are_refused(frontend_route):
    """What the GPU refuses, a query or a launch, leaves the two launches and their status, and no error of its own; one that the
    caller had pending is not taken away."""
    assert frontend_route(1) == ('q1', 0, False)
    assert frontend_route(1, launch_ok=False) == ('q1cT', 42, False)
    assert frontend_route(9, launch_ok=False) == ('q2cT', 42, False)
    assert frontend_route(1, query_ok=False) == ('qcT', 42, False)
    assert frontend_route(1, launch_ok=False, pending=True) == ('q1T', 42, True)
    assert frontend_route(1, query_ok=False, pending=True) == ('qT', 42, True)
    assert frontend_route(1, pending=True) == ('q1', 0, True)
    assert frontend_route(1, clusters=0) == ('qT', 42, False)
    assert frontend_route(33) == frontend_route(1, hidden=4352) == frontend_route(1, experts=385) == ('T', 42, False)


def test_known_clusters_are_kept_only_when_the_query_succeeded(frontend_route):
    """Under the thread sanitizer, where there is one: the table that threads share has no data race."""
    r = frontend_route([])
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])


def test_kernel_attributes_of_a_device_are_only_raised(frontend_route):
    """Threads that launch a kernel with different shared memory sizes for the first time: none finds the attribute below its own."""
    r = frontend_route(['attribute'])
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])


@pytest.mark.parametrize('tokens,hidden,experts,grid,per', [
    (7, 256, 8, 148, 1), (7, 4096, 384, 148, 1), (14, 2048, 8, 148, 2), (15, 4096, 384, 148, 0),                  # as many tokens as clusters, twice as many
    (8, 2048, 8, 148, 2), (8, 1792, 256, 148, 0), (8, 256, 257, 148, 2),                                          # one token more
    (9, 1536, 8, 148, 2), (9, 1280, 192, 148, 0), (9, 256, 193, 148, 2),
    (1, 3072, 48, 16, 1), (1, 3072, 48, 15, 0), (7, 3072, 48, 112, 1), (7, 3072, 48, 111, 0), (9, 3072, 48, 80, 2), (9, 3072, 48, 79, 0),        # the caller's CTAs
])
def test_frontend_lines_between_one_and_two_launches(frontend_route, tokens, hidden, experts, grid, per):
    assert frontend_route(tokens, hidden, experts, grid) == (('q%d' % per, 0, False) if per else ('qT', 42, False))
