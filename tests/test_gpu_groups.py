"""Grouped launches of the surrogate network (several products, optimiser updates, row sums or
input packs per launch) against the one-at-a-time entry points, bit for bit, and the vector
gate kernel against the scalar one."""

import ctypes

import numpy as np
import pytest
import torch

from pylblrtm_b200 import _lib, surrogate

pytestmark = pytest.mark.gpu


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _close_bits(a, b):
    return torch.equal(a.view(torch.int32) if a.dtype == torch.float32 else a,
                       b.view(torch.int32) if b.dtype == torch.float32 else b)


# one and several members (8 per launch), 128- and 256-wide tiles, ragged last waves
@pytest.mark.parametrize("count,m,n,k", [(1, 128, 128, 64), (2, 256, 256, 192), (4, 256, 2048, 128),
                                         (9, 384, 384, 64), (3, 9600, 256, 128)])
def test_gemm_group_equals_single(cuda, count, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m + n)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    a = [rnd(m, k).bfloat16() for _ in range(count)]
    b = [rnd(n, k).bfloat16() for _ in range(count)]
    bias = [rnd(n) for _ in range(count)]
    maps = [(surrogate._Map(x), surrogate._Map(y)) for x, y in zip(a, b)]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for mode, dt in ((_lib.GEMM_BIAS_GELU, torch.bfloat16), (_lib.GEMM_BIAS_SIGMOID, torch.float32)):
        outs = [[torch.zeros((m, n), dtype=dt, device="cuda") for _ in range(count)] for _ in range(2)]
        eps = []
        for o in outs:
            arr = (_lib.GemmEpilogue * count)()
            for i in range(count):
                arr[i].mode, arr[i].n_valid, arr[i].bias = mode, n, bias[i].data_ptr()
                if dt == torch.float32:
                    arr[i].out_f32, arr[i].ld_f32 = o[i].data_ptr(), n
                else:
                    arr[i].y, arr[i].ld_y = o[i].data_ptr(), n
            eps.append(arr)
        for i in range(count):
            _lib.call("lbl_gemm_bf16", maps[i][0].addr, maps[i][1].addr, m, n, k, 1, ctypes.addressof(eps[0][i]),
                      err.data_ptr(), _stream())
        addr = lambda j: (ctypes.c_void_p * count)(*[p[j].addr for p in maps])
        _lib.call("lbl_gemm_bf16_group", count, addr(0), addr(1), m, n, k, ctypes.addressof(eps[1]), err.data_ptr(),
                  _stream())
        assert err.item() == 0
        for x, y in zip(*outs):
            assert torch.equal(x, y) and x.float().abs().sum() > 0
    bad = (_lib.GemmEpilogue * 1)()
    bad[0].mode, bad[0].bias, bad[0].loss = _lib.GEMM_BIAS_SIGMOID, bias[0].data_ptr(), err.data_ptr()
    with pytest.raises(RuntimeError, match="no loss"):
        _lib.call("lbl_gemm_bf16_group", 1, addr(0), addr(1), m, n, k, ctypes.addressof(bad), err.data_ptr(), _stream())


@pytest.mark.parametrize("shapes", [[(64, 64, 1, True)], [(128, 128, 2, True), (1, 128, 1, False), (132, 68, 3, True)],
                                    [(4, 4, 1, True), (1, 2048, 1, False)] * 9])
def test_adam_group_equals_single(cuda, shapes):
    g = torch.Generator(device="cuda").manual_seed(3)
    items, pairs = [], []
    for rows, cols, split, bf in shapes:
        base = [torch.randn((rows, cols), generator=g, device="cuda") for _ in range(2)]
        base.append(torch.rand((rows, cols), generator=g, device="cuda"))
        grad = torch.randn((split, rows, cols), generator=g, device="cuda")
        two = []
        for _ in range(2):
            w, m, v = (t.clone() for t in base)
            two.append((w, m, v, torch.zeros((rows, cols), dtype=torch.bfloat16, device="cuda"),
                        torch.zeros((cols, rows), dtype=torch.bfloat16, device="cuda")))
        w, m, v, wb, wt = two[0]
        _lib.call("lbl_adam_step", w.data_ptr(), m.data_ptr(), v.data_ptr(), grad.data_ptr(), split, rows * cols, rows,
                  cols, cols, 1e-3, 0.9, 0.999, 1e-8, 7, wb.data_ptr() if bf else 0, wt.data_ptr() if bf else 0, rows,
                  _stream())
        w, m, v, wb, wt = two[1]
        items.append(_lib.AdamItem(w.data_ptr(), m.data_ptr(), v.data_ptr(), grad.data_ptr(), rows * cols,
                                   wb.data_ptr() if bf else None, wt.data_ptr() if bf else None, split, rows, cols))
        pairs.append((two, grad))
    arr = (_lib.AdamItem * len(items))(*items)
    _lib.call("lbl_adam_group", ctypes.addressof(arr), len(items), 1e-3, 0.9, 0.999, 1e-8, 7, _stream())
    for two, _ in pairs:
        for x, y in zip(*two):
            assert _close_bits(x, y)
    arr[0].cols = 6
    with pytest.raises(RuntimeError, match="multiples"):
        _lib.call("lbl_adam_group", ctypes.addressof(arr), 1, 1e-3, 0.9, 0.999, 1e-8, 7, _stream())


@pytest.mark.parametrize("shapes", [[(3, 8, 8)], [(128, 128, 128), (1, 256, 264), (70, 4096, 4096)], [(5, 1032, 1032)] * 17])
def test_rowsum_group_equals_single(cuda, shapes):
    g = torch.Generator(device="cuda").manual_seed(5)
    xs = [torch.randn((r, ld), generator=g, device="cuda").bfloat16() for r, _, ld in shapes]
    a = [torch.zeros(r, device="cuda") for r, _, _ in shapes]
    b = [torch.zeros(r, device="cuda") for r, _, _ in shapes]
    for x, o, (r, c, ld) in zip(xs, a, shapes):
        _lib.call("lbl_rowsum_bf16", x.data_ptr(), r, c, ld, o.data_ptr(), _stream())
    arr = (_lib.RowsumItem * len(shapes))(*[_lib.RowsumItem(x.data_ptr(), o.data_ptr(), r, c, ld)
                                            for x, o, (r, c, ld) in zip(xs, b, shapes)])
    _lib.call("lbl_rowsum_group", ctypes.addressof(arr), len(shapes), _stream())
    for x, y in zip(a, b):
        assert _close_bits(x, y)


@pytest.mark.parametrize("members,batch,hidden", [(1, 5, 128), (2, 130, 256), (4, 128, 128), (9, 1, 128)])
def test_ensemble_equals_members(cuda, members, batch, hidden):
    """Grouped members against one network at a time; the same network twice, and members of
    different depth, take the loop and agree too."""
    nets = [surrogate.MLP(61, 300, hidden=hidden, depth=2, seed=i) for i in range(members)]
    for i, n in enumerate(nets):
        n.set_normalisation(np.full(61, 0.1 * i), np.full(61, 1.0 + 0.1 * i))
    raw = torch.randn((batch, 61), generator=torch.Generator().manual_seed(1)).cuda()
    want = torch.stack([n.predict(raw) for n in nets])
    gs = surrogate.GatedSurrogate(nets, gate=0.01)
    assert torch.equal(gs.predictions(raw), want)
    assert torch.equal(gs.predictions(raw.double()), want)              # converted as before
    mean, est, flag = gs.ensemble(raw)
    sd = (want - want.mean(0)).square().mean(0).sqrt()
    # float32 sums of at most 9 values near 0.5
    assert torch.allclose(mean, want.mean(0), rtol=1e-6, atol=0)
    assert torch.allclose(est, sd.max(1).values, rtol=1e-5, atol=1e-7)
    assert torch.equal(flag, est > 0.01)
    twice = surrogate.GatedSurrogate([nets[0], nets[0]])
    assert torch.equal(twice.predictions(raw)[1], want[0])
    other = surrogate.MLP(61, 300, hidden=hidden, depth=3, seed=50)
    mixed = surrogate.GatedSurrogate([nets[0], other])
    assert torch.equal(mixed.predictions(raw), torch.stack([want[0], other.predict(raw)]))


@pytest.mark.parametrize("n_mem,n_ch", [(2, 4), (3, 300), (4, 2000), (5, 1028), (6, 12), (8, 260), (7, 64), (4, 301)])
def test_gate_kernels_agree(cuda, n_mem, n_ch):
    """Shapes of the vector kernel, and a member count and a channel count it leaves to the
    scalar one, against the scalar kernel on a copy it has to take (odd row stride)."""
    g = torch.Generator(device="cuda").manual_seed(n_ch)
    b, ld = 37, -(-n_ch // 4) * 4 + 4
    pred = torch.rand((n_mem, b, ld), generator=g, device="cuda")
    odd = torch.zeros((n_mem, b, ld + 1), device="cuda")
    odd[..., :ld] = pred
    scale = torch.rand(n_ch, generator=g, device="cuda") + 0.5
    res = []
    for p in (pred, odd):
        mean, est = torch.zeros((b, n_ch), device="cuda"), torch.zeros(b, device="cuda")
        flag = torch.zeros(b, dtype=torch.int32, device="cuda")
        _lib.call("lbl_ensemble_gate", p.data_ptr(), n_mem, b * p.shape[2], b, p.shape[2], n_ch, scale.data_ptr(), 1.1,
                  0.3, mean.data_ptr(), est.data_ptr(), flag.data_ptr(), _stream())
        res.append((mean, est, flag))
    for x, y in zip(*res):
        assert _close_bits(x, y)


# rows that start on 16 but not on 32 bytes take two stores each; the values are the same
@pytest.mark.parametrize("m,n,k", [(128, 128, 64), (256, 512, 128)])
def test_epilogue_rows_of_any_alignment(cuda, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(n)
    a, b = (torch.randn(s, generator=g, device="cuda").bfloat16() for s in ((m, k), (n, k)))
    bias = torch.randn(n, generator=g, device="cuda")
    ma, mb = surrogate._Map(a), surrogate._Map(b)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for mode, dt, step in ((_lib.GEMM_F32, torch.float32, 4), (_lib.GEMM_BIAS_SIGMOID, torch.float32, 4),
                           (_lib.GEMM_BIAS_GELU, torch.bfloat16, 8)):
        outs = []
        for extra in (0, step, 2 * step):             # elements of 16, then 32 bytes more per row
            buf = torch.full((m * (n + extra) + step,), -7.0, dtype=dt, device="cuda")
            out = buf[step if extra else 0:][:m * (n + extra)].view(m, n + extra)
            ep = _lib.GemmEpilogue()
            ep.mode, ep.n_valid, ep.bias = mode, n, bias.data_ptr()
            if dt == torch.float32:
                ep.out_f32, ep.ld_f32 = out.data_ptr(), n + extra
            else:
                ep.y, ep.ld_y = out.data_ptr(), n + extra
            _lib.call("lbl_gemm_bf16", ma.addr, mb.addr, m, n, k, 1, ctypes.addressof(ep), err.data_ptr(), _stream())
            assert err.item() == 0
            assert (out[:, n:] == -7.0).all()
            outs.append(out[:, :n])
        assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


# two products of their own shapes: 256-wide tiles, 128-wide ones, unequal depths and split-K
@pytest.mark.parametrize("shapes", [[(4096, 1024, 1024, 1), (1024, 1024, 4096, 4)], [(128, 128, 64, 1), (128, 128, 128, 2)],
                                    [(384, 384, 256, 1), (128, 512, 1024, 8)], [(256, 256, 192, 1), (128, 128, 64, 1)]])
def test_gemm_pair_equals_single(cuda, shapes):
    g = torch.Generator(device="cuda").manual_seed(len(shapes) + shapes[0][0])
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    ab = [(rnd(m, k).bfloat16(), rnd(n, k).bfloat16()) for m, n, k, _ in shapes]
    maps = [(surrogate._Map(a), surrogate._Map(b)) for a, b in ab]
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    (m0, n0, _, _), (m1, n1, _, s1) = shapes
    z = rnd(m0, n0).bfloat16()
    outs, eps = [], []
    for _ in range(2):
        o = [torch.zeros((m0, n0), dtype=torch.bfloat16, device="cuda"),
             torch.zeros((n0, m0), dtype=torch.bfloat16, device="cuda"), torch.zeros((s1, m1, n1), device="cuda")]
        ep = (_lib.GemmEpilogue * 2)()
        ep[0].mode, ep[0].z_in, ep[0].ld_zin = _lib.GEMM_DGELU, z.data_ptr(), n0
        ep[0].y, ep[0].ld_y, ep[0].y_t, ep[0].ld_yt = o[0].data_ptr(), n0, o[1].data_ptr(), m0
        ep[1].mode, ep[1].out_f32, ep[1].ld_f32, ep[1].split_stride = _lib.GEMM_F32, o[2].data_ptr(), n1, m1 * n1
        outs.append(o)
        eps.append(ep)
    for i, (m, n, k, s) in enumerate(shapes):
        _lib.call("lbl_gemm_bf16", maps[i][0].addr, maps[i][1].addr, m, n, k, s, ctypes.addressof(eps[0][i]),
                  err.data_ptr(), _stream())
    ptrs = lambda j: (ctypes.c_void_p * 2)(*[p[j].addr for p in maps])
    ints = lambda j: (ctypes.c_int * 2)(*[s[j] for s in shapes])
    _lib.call("lbl_gemm_bf16_pair", ptrs(0), ptrs(1), ints(0), ints(1), ints(2), ints(3), ctypes.addressof(eps[1]),
              err.data_ptr(), _stream())
    assert err.item() == 0
    for x, y in zip(*outs):
        assert torch.equal(x, y) and x.float().abs().sum() > 0
    want = (ab[1][0].float() @ ab[1][1].float().T)                      # the split sums are the product
    assert torch.allclose(outs[1][2].sum(0), want, rtol=1e-4, atol=1e-4 * shapes[1][2] ** 0.5)


# remainders of the 32-row and 8-row splits, vector and scalar rows, several column blocks
@pytest.mark.parametrize("rows,n_in,ld,n_out", [(1, 1, 128, 1), (33, 61, 128, 2000), (128, 130, 256, 301), (45, 64, 64, 8)])
def test_stage_batch_equals_gather_and_pack(cuda, rows, n_in, ld, n_out):
    g = torch.Generator(device="cuda").manual_seed(rows + n_in)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    n = 2 * rows + 5
    feat, targ, mean, inv = rnd(n, n_in), rnd(n, n_out), rnd(n_in), rnd(n_in).abs() + 0.1
    idx = torch.randperm(n, generator=torch.Generator().manual_seed(1)).cuda()[:rows]
    bf = lambda *s: torch.full(s, 7.0, dtype=torch.bfloat16, device="cuda")
    x, xt, x0, xt0 = bf(rows, ld), bf(ld, rows), bf(rows, ld), bf(ld, rows)
    target = torch.full((rows, n_out), 7.0, device="cuda")
    loss = torch.ones(1, dtype=torch.float64, device="cuda")
    stage = lambda i: _lib.call("lbl_stage_batch", feat.data_ptr(), targ.data_ptr(), i.data_ptr(), n, rows, n_in, n_out,
                                mean.data_ptr(), inv.data_ptr(), x.data_ptr(), ld, xt.data_ptr(), rows,
                                target.data_ptr(), loss.data_ptr(), _stream())
    stage(idx)
    raw = feat[idx].contiguous()
    _lib.call("lbl_pack_inputs_bf16", raw.data_ptr(), rows, n_in, mean.data_ptr(), inv.data_ptr(), x0.data_ptr(), ld,
              xt0.data_ptr(), rows, _stream())
    assert torch.equal(x, x0) and torch.equal(xt, xt0) and torch.equal(target, targ[idx]) and loss.item() == 0.0
    out = idx.clone()
    out[-1] = n                                       # not a sample: read nowhere, NaN in the batch
    stage(out)
    assert target[-1].isnan().all() and x[-1, :n_in].isnan().all() and torch.equal(target[:-1], targ[idx[:-1]])
