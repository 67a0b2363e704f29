"""The fused preparation entry points (sort + gather, all line ranges, layers + groups) against
the one-step entry points they stand in for, bit for bit."""

import ctypes

import numpy as np
import pytest
import torch

from pylblrtm_b200 import _lib
from pylblrtm_b200.atmosphere import COLUMN_FACTOR

pytestmark = pytest.mark.gpu
INT_MAX = 2 ** 31 - 1


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _up(a, dt=np.float64):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=dt)).cuda()


# one block, its edges, one to three merge passes with short and empty runs; random, presorted
# and heavily tied centres; masked-out, groupless and non-finite lines; all dropped
@pytest.mark.parametrize("n", [1, 2, 511, 512, 513, 1024, 4095, 4097, 33_000, 40_961, 270_001])
@pytest.mark.parametrize("kind", ["random", "sorted", "ties", "none"])
def test_sort_gather_and_ranges(cuda, n, kind):
    rng = np.random.default_rng(n)
    cols = [rng.uniform(0.0, 1.0, n) for _ in range(7)]
    cols[0] = rng.uniform(590.0, 710.0, n)
    if kind == "sorted":
        cols[0] = np.sort(cols[0])
    elif kind == "ties":
        cols[0] = np.round(cols[0] / 7.0) * 7.0
        cols[0][rng.integers(0, n, n // 9)] = rng.choice([np.nan, np.inf, -np.inf, 0.0, -0.0], n // 9)
    cols[6] = rng.uniform(-0.5, 0.5, n)
    gid = rng.integers(-1, 3, n) if kind != "none" else np.full(n, -1)
    d = [_up(c) for c in cols]
    g = _up(gid, np.int32)
    lib, lo, hi, p_max = _lib.load(), 600.0, 700.0, 0.9
    ws_n = lib.lbl_sort_workspace_bytes(n)
    ws = torch.empty(ws_n, dtype=torch.uint8, device="cuda")
    order, kept = torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty(1, dtype=torch.int32, device="cuda")
    sb = torch.empty(1, dtype=torch.float64, device="cuda")
    want = torch.empty((n, 8), dtype=torch.float64, device="cuda")
    _lib.call("lbl_sort_lines", d[0].data_ptr(), d[6].data_ptr(), g.data_ptr(), n, lo, hi, p_max, ws.data_ptr(), ws_n,
              order.data_ptr(), kept.data_ptr(), sb.data_ptr(), _stream())
    _lib.call("lbl_gather_lines", *[c.data_ptr() for c in d], g.data_ptr(), order.data_ptr(), kept.data_ptr(), n,
              want.data_ptr(), _stream())
    for n_out in sorted({n, max(1, int(kept.item())), max(1, n // 3)}):
        got = torch.full((n + 1, 8), -7.0, dtype=torch.float64, device="cuda")
        kept2 = torch.full((1,), -1, dtype=torch.int32, device="cuda")
        ws_n = lib.lbl_sort_gather_workspace_bytes(n)
        ws = torch.empty(ws_n, dtype=torch.uint8, device="cuda")
        _lib.call("lbl_sort_gather", *[c.data_ptr() for c in d], g.data_ptr(), n, lo, hi, p_max, ws.data_ptr(), ws_n,
                  n_out, got.data_ptr(), kept2.data_ptr(), _stream())
        assert kept2.item() == kept.item()
        assert torch.equal(got[:n_out].view(torch.int64), want[:n_out].view(torch.int64))
        assert torch.all(got[n_out:] == -7.0)
    with pytest.raises(RuntimeError, match="workspace"):
        _lib.call("lbl_sort_gather", *[c.data_ptr() for c in d], g.data_ptr(), n, lo, hi, p_max, ws.data_ptr(),
                  ws_n - 1, n, got.data_ptr(), kept2.data_ptr(), _stream())
    # line ranges of a ragged grid of tiles
    nu_min, step, n_nu, ts, cutoff, pad = 601.3, 0.013, 7001, 150, 4.4, 0.6
    n_tiles = -(-n_nu // ts)
    a = torch.full((3, n_tiles, 2), -1, dtype=torch.int32, device="cuda")
    b = torch.full((3, n_tiles, 2), -2, dtype=torch.int32, device="cuda")
    tail = (pad, n_tiles)
    _lib.call("lbl_tile_ranges", want.data_ptr(), kept.data_ptr(), nu_min, step, n_nu, ts, cutoff, *tail,
              a[0].data_ptr(), _stream())
    _lib.call("lbl_ml_inner_ranges", want.data_ptr(), kept.data_ptr(), nu_min, step, n_nu, ts, *tail, a[1].data_ptr(),
              _stream())
    _lib.call("lbl_jac_near_ranges", want.data_ptr(), kept.data_ptr(), nu_min, step, n_nu, ts, *tail, a[2].data_ptr(),
              _stream())
    _lib.call("lbl_line_ranges", want.data_ptr(), kept.data_ptr(), nu_min, step, n_nu, ts, cutoff, *tail,
              *[b[i].data_ptr() for i in range(3)], _stream())
    assert torch.equal(a, b)


@pytest.mark.parametrize("from_levels", [True, False])
@pytest.mark.parametrize("table", [1, 2, 33, 2931])
def test_layer_setup(cuda, from_levels, table):
    rng = np.random.default_rng(table)
    n_prof, n_lay, n_gas, n_grp = 3, 7, 2, 4
    lev_p = _up(np.sort(rng.uniform(1.0, 1000.0, (n_prof, n_lay + 1)), axis=1))
    lev_t = _up(rng.uniform(150.0, 400.0, (n_prof, n_lay + 1)))
    lev_v = _up(rng.uniform(0.0, 0.1, (n_prof, n_gas, n_lay + 1)))
    tips_t = np.linspace(160.0, 380.0, table) if table > 1 else np.array([296.0])      # clamps at both ends
    if table > 2:
        lev_t[0, :2] = float(tips_t[1])                                                  # exactly a table value
    lens = [table, 1, table, max(1, table // 2)]
    offs = np.cumsum([0] + lens[:-1])
    tt = np.concatenate([tips_t[:k] for k in lens])
    tq = np.concatenate([rng.uniform(1.0, 9.0, k) for k in lens])
    grp = [_up([0, 1, 1, 0], np.int32), _up([18.0, 44.0, 45.0, 19.0]), _up(offs, np.int32), _up(lens, np.int32),
           _up(tt), _up(tq)]
    z = lambda *s: torch.zeros(s, dtype=torch.float64, device="cuda")
    p, t, v, c = z(n_prof, n_lay), z(n_prof, n_lay), z(n_prof, n_gas, n_lay), z(n_prof, n_gas, n_lay)
    _lib.call("lbl_build_layers", lev_p.data_ptr(), lev_t.data_ptr(), lev_v.data_ptr(), n_prof, n_lay + 1, n_gas,
              COLUMN_FACTOR, p.data_ptr(), t.data_ptr(), v.data_ptr(), c.data_ptr(), _stream())
    if not from_levels:
        t[1, 2] = float("nan")
    want, got, t_out = z(n_prof * n_lay * n_grp, 6), z(n_prof * n_lay * n_grp, 6), z(n_prof, n_lay)
    _lib.call("lbl_layer_groups", t.data_ptr(), p.data_ptr(), v.data_ptr(), c.data_ptr(), n_prof, n_lay, n_gas, n_grp,
              *[x.data_ptr() for x in grp], want.data_ptr(), _stream())
    lay = [x.data_ptr() for x in ((lev_p, lev_t, lev_v) if from_levels else (p, t, v, c))]
    lay = lay + [0] * 4 if from_levels else [0] * 3 + lay
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    _lib.call("lbl_layer_setup", *lay, n_prof, n_lay, n_gas, n_grp, COLUMN_FACTOR, *[x.data_ptr() for x in grp],
              t_out.data_ptr(), got.data_ptr(), err.data_ptr(), _stream())
    bits = lambda a: a.view(torch.int64)
    assert torch.equal(bits(got), bits(want)) and torch.equal(bits(t_out), bits(t)) and err.item() == INT_MAX
