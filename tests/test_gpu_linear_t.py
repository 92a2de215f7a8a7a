"""The tcgen05 GEMM (C = A W^T + b) against the oracle's linear_t and the on-device naive anchor."""
import ctypes

import numpy as np
import pytest
import torch

import oracle_lib as O
from gpu_util import DEV, TOL, bf16_cuda, max_rel, to_np
from logismos_b200 import ops
from logismos_b200._lib import lib

pytestmark = pytest.mark.gpu


def case(m, n, k, seed, bias=True):
    rng = np.random.default_rng(seed)
    a_t, a = bf16_cuda(rng.standard_normal((m, k)))
    w_t, w = bf16_cuda(rng.standard_normal((n, k)) * 0.05)
    b = (rng.standard_normal(n) * 0.5).astype(np.float32) if bias else None
    return a_t, a, w_t, w, b


# M ragged against the 128-row tile, N exercising every tile width (128 / 192 / 256) and a ragged last
# tile, K from one stage to the longest reduction of the model
@pytest.mark.parametrize("m,n,k", [(128, 256, 64), (1, 16, 64), (100, 1536, 1536), (333, 2048, 1536), (129, 192, 128),
                                   (2176, 1536, 1536), (257, 1536, 8960), (64, 400, 256), (700, 17920, 512)])
def test_bf16_epilogue_matches_oracle_linear_t(m, n, k):
    a_t, a, w_t, w, b = case(m, n, k, m + n + k)
    got = to_np(ops.linear_t(a_t, w_t, torch.from_numpy(b).to(DEV)))
    ref = O.linear_t(a, w, b, m, n, k).reshape(m, n)
    assert max_rel(got, ref) <= TOL
    assert np.abs(got - ref).max() <= 2 ** -8 * np.abs(ref).max() + 1e-5  # only the bf16 store rounds


@pytest.mark.parametrize("m,n,k,kind", [(64, 2048, 2048, "bf16"), (300, 1536, 1536, "resid"), (64, 12288, 2048, "swiglu"), (2, 256, 64, "bf16")])
def test_static_weight_promise_changes_nothing_but_the_fetch_order(m, n, k, kind):
    """With the static-weights flag the kernel requests its first weight stages ahead of the dependency
    wait; launched behind a kernel of this library that rewrites the ACTIVATIONS (so the early start
    really overlaps a producer), the result equals the one without the flag bit for bit."""
    from logismos_b200._lib import lib
    a_t, a, w_t, w, b = case(m, n, k, 5 * m + n + k, bias=False)
    lib.logismos_set_deterministic(1)   # no split over k: a fixed summation order
    try:
        outs = []
        for static in (False, True):
            res = torch.zeros((m, n), dtype=torch.float32, device=DEV) if kind == "resid" else None
            x = torch.zeros((m, k), dtype=torch.float32, device=DEV)
            src = a_t.float().contiguous()
            # the producer ahead of the GEMM: this library's rms_norm (unit gains) of rows pre-scaled to unit RMS
            rms = src.pow(2).mean(dim=1, keepdim=True).sqrt()
            x.copy_(src / rms)
            ones = torch.ones(k, dtype=torch.float32, device=DEV)
            torch.cuda.synchronize()
            h = ops.rms_norm_f32(x, ones, 0.0, sync=False)
            outs.append(to_np(ops.linear_t(h, w_t, residual=res, swiglu=(kind == "swiglu"), static_w=static)))
        assert np.array_equal(outs[0], outs[1])
    finally:
        lib.logismos_set_deterministic(0)


def test_matches_the_naive_anchor_on_device():
    a_t, a, w_t, w, b = case(300, 768, 1024, 5)
    bt = torch.from_numpy(b).to(DEV)
    fast = to_np(ops.linear_t(a_t, w_t, bt)); slow = to_np(ops.linear_t(a_t, w_t, bt, naive=True))
    assert np.abs(fast - slow).max() <= 2 ** -7 * np.abs(slow).max()


@pytest.mark.parametrize("m,n,k", [(200, 1536, 1536), (77, 1536, 8960), (130, 512, 64)])
def test_residual_epilogue_accumulates_into_fp32(m, n, k):
    a_t, a, w_t, w, _ = case(m, n, k, 3 * m + n, bias=False)
    rng = np.random.default_rng(1)
    x0 = rng.standard_normal((m, n)).astype(np.float32)
    x_t = torch.from_numpy(x0.copy()).to(DEV)
    ops.linear_t(a_t, w_t, residual=x_t)
    ref = x0 + O.linear_t(a, w, None, m, n, k).reshape(m, n)
    assert np.abs(to_np(x_t) - ref).max() <= 1e-4 * max(1.0, np.abs(ref).max())
    ops.linear_t(a_t, w_t, residual=x_t)  # twice: the accumulator buffers and barriers recycle cleanly
    assert np.abs(to_np(x_t) - (ref + ref - x0)).max() <= 2e-4 * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("m,inter,k", [(150, 1024, 512), (2176, 8960, 1536), (33, 96, 64)])
def test_swiglu_epilogue(m, inter, k):
    rng = np.random.default_rng(m + inter)
    a_t, a = bf16_cuda(rng.standard_normal((m, k)))
    wg_t, wg = bf16_cuda(rng.standard_normal((inter, k)) * 0.05)
    wu_t, wu = bf16_cuda(rng.standard_normal((inter, k)) * 0.05)
    # gate/up rows interleaved in blocks of 32
    inter_w = torch.stack([wg_t.view(inter // 32, 32, k), wu_t.view(inter // 32, 32, k)], dim=1).reshape(2 * inter, k).contiguous()
    got = to_np(ops.linear_t(a_t, inter_w, swiglu=True))
    g = O.linear_t(a, wg, None, m, inter, k); u = O.linear_t(a, wu, None, m, inter, k)
    ref = O.hadamard(O.silu(g), u).reshape(m, inter)
    assert max_rel(got, ref) <= TOL


def test_shape_guards_reject_before_launch():
    a = torch.zeros((8, 100), dtype=torch.bfloat16, device=DEV)  # k not a multiple of 64
    w = torch.zeros((16, 100), dtype=torch.bfloat16, device=DEV)
    with pytest.raises(Exception):
        ops.linear_t(a, w)
    with pytest.raises(ops.InvalidOp):
        ops.linear_t(a.cpu(), w)


# large outputs: rows that leave the last row tile ragged or whole, a ragged last column tile, several groups of row tiles, by pairs of CTAs
# where the rule takes them. Against fp32 products of the same bf16 values: one bf16 rounding (2^-9 of the value), fp32 sums in
# another order (1e-4 of the largest)
@pytest.mark.parametrize("m,n,k,kind", [(4161, 4112, 1024, "bf16"), (4224, 4096, 1024, "swiglu"), (2177, 1536, 8960, "resid"), (1089, 1536, 8960, "resid"), (4300, 4112, 1024, "f32"),
                                        (4097, 4096, 1024, "f32")])
def test_row_tiles_of_a_pair_of_ctas(m, n, k, kind):
    g = torch.Generator(device=DEV)
    g.manual_seed(m + n)
    a = torch.randn((m, k), generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn((n, k), generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    ref = a.float() @ w.float().T
    if kind == "swiglu":
        z = ref.reshape(m, n // 64, 2, 32)
        ref = (torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(m, n // 2)
        got = ops.linear_t(a, w, swiglu=True)
    elif kind == "resid":
        x = torch.randn((m, n), generator=g, device=DEV)
        ref = x + ref
        got = x.clone()
        ops.linear_t(a, w, residual=got)
    elif kind == "bf16":
        bias = torch.randn(n, generator=g, device=DEV)
        ref = ref + bias
        got = ops.linear_t(a, w, bias)
    else:
        got = ops.linear_act(a, w, epilogue=ops.EPI_F32)
    rounding = 0.0 if kind in ("resid", "f32") else 2 ** -8
    assert ((got.float() - ref).abs() <= rounding * ref.abs() + 1e-4 * ref.abs().max()).all()


@pytest.mark.parametrize("m", [5, 700])
def test_swiglu_divides_with_rounding(m):
    """silu(g) = g / (1 + exp(-g)) is a rounded division for every finite g. At g = -87.5 the denominator, 1.0e38, lies above 2^126, from
    where the approximate division returns zero; a large up value brings the quotient back into view. exp within 2^-21 |g| of its value."""
    k, gates = 64, torch.tensor([-87.5, -87.0, -20.0, -3.0, 0.5, 6.0, 87.5, -88.0])
    a, w = torch.zeros((m, k)), torch.zeros((128, k))
    a[:, :2] = 1.0
    z = w.view(2, 2, 32, k)
    z[:, 0, :, 0] = gates.repeat(8).view(2, 32)
    z[:, 1, :, 1] = 2.0 ** 100
    ref = (gates.double() / (1.0 + torch.exp(-gates.double())) * 2.0 ** 100).repeat(8).expand(m, 64)
    got = ops.linear_t(a.to(DEV, torch.bfloat16), w.to(DEV, torch.bfloat16), swiglu=True).cpu().double()
    assert ((got - ref).abs() <= (2 ** -8 + 2e-4) * ref.abs()).all(), (got[0, :8], ref[0, :8])


def test_swiglu_does_not_depend_on_the_tile():
    """Gates at which a quotient corrected once is not the rounded one, with up values that bring the last bit of the quotient into the bf16 result: adjacent floats around silu(g) times u
    lie on two sides of a boundary of bf16. One row (tiles of 128 columns) against 40000 (of 256), bit for bit; every sum is of up to three bf16 parts and exact."""
    f32 = np.float32

    def parts(x):  # three bf16 values that add up to a float
        out, rest = [], f32(x)
        for _ in range(3):
            out.append((np.atleast_1d(rest).view(np.uint32) & np.uint32(0xffff0000)).view(f32)[0])
            rest = f32(rest - out[-1])
        assert rest == 0
        return out

    rn = lambda v: float(torch.tensor(float(v)).to(torch.bfloat16))
    cols = []
    for bits in (0x3e609af2, 0x3e24a9bf):
        g = np.array([bits], np.uint32).view(f32)[0]
        s = f32(float(g) / (1.0 + np.exp(-float(g))))
        for step in range(-4, 4):  # the device's exponential may move the quotient some units
            lo = np.array([int(s.view(np.uint32)) + step], np.uint32).view(f32)[0]
            hi, found = np.nextafter(lo, f32(1)), 0
            for i in range(128):
                u = f32(2 * (1 + (2 * i + 1) / 256) / (float(lo) + float(hi)))  # their product with u: about half way between two values of bf16
                for v in (u, np.nextafter(u, f32(0)), np.nextafter(u, f32(99))):
                    if found < 8 and rn(f32(lo * v)) != rn(f32(hi * v)):
                        cols.append((g, v))
                        found += 1
            assert found, (bits, step)
    n, k, m = 1024, 64, 40000
    z = torch.zeros((n // 64, 2, 32, k))
    for j in range(n // 2):
        g, u = cols[j % len(cols)]
        z[j // 32, 0, j % 32, 0:3] = torch.tensor(parts(g)); z[j // 32, 1, j % 32, 3:6] = torch.tensor(parts(u))
    a = torch.zeros((m, k)); a[:, :6] = 1.0
    a, w = a.to(DEV, torch.bfloat16), z.view(n, k).to(DEV, torch.bfloat16)
    assert torch.equal(w.float().cpu(), z.view(n, k)) and tile_of(1, n, k, ops.EPI_SWIGLU)[0] == 128 and tile_of(m, n, k, ops.EPI_SWIGLU)[0] == 256
    one, many = ops.linear_t(a[:1].contiguous(), w, swiglu=True), ops.linear_t(a, w, swiglu=True)
    assert torch.equal(one.expand(m, -1), many)


def test_swiglu_of_extreme_gates_does_not_depend_on_the_tile():
    """Gates whose exponential overflows, vanishes or is near 2^100 and 2^126, zeros, the smallest and largest values, infinities, NaN: one row (tiles of 128 columns) against 40000 (of 256),
    bit for bit."""
    ln2 = float(np.log(2.0))
    gates = [0.0, -0.0, 1e-38, -1e-38, 1e-30, -1e-30, 3e38, -3e38, float("inf"), float("-inf"), float("nan"), 88.5, -88.5, 100.0, -100.0]
    gates += [-ln2 * e + d for e in (63, 64, 99, 100, 101, 125, 126, 127, 128) for d in (-0.5, 0.0, 0.5)]
    gates += np.linspace(-110.0, 110.0, 512 - len(gates)).tolist()
    n, k, m = 1024, 64, 40000
    g = torch.tensor(gates, dtype=torch.float32).to(torch.bfloat16).float()
    z = torch.zeros((n // 64, 2, 32, k))
    z[:, 0, :, 0] = g.view(16, 32); z[:, 1, :, 1] = 1.0
    a = torch.zeros((m, k)); a[:, :2] = 1.0
    a, w = a.to(DEV, torch.bfloat16), z.view(n, k).to(DEV, torch.bfloat16)
    assert tile_of(1, n, k, ops.EPI_SWIGLU)[0] == 128 and tile_of(m, n, k, ops.EPI_SWIGLU)[0] == 256
    one, many = ops.linear_t(a[:1].contiguous(), w, swiglu=True), ops.linear_t(a, w, swiglu=True)
    nan = one.isnan()
    assert torch.equal(nan.expand(m, -1), many.isnan()) and torch.equal(torch.where(nan, 0.0, one).view(torch.int16).expand(m, -1), torch.where(nan, 0.0, many).view(torch.int16))


@pytest.mark.parametrize("m,n,k", [(800, 1536, 8960), (1024, 1536, 1536), (600, 2048, 8192)])
def test_outputs_that_fill_half_the_chip_repeat(m, n, k):
    """Residual updates of middle size are one sum over k per element: the same bits every time, and those of 200 rows at a time, which
    take other tiles, under the deterministic switch."""
    g = torch.Generator(device=DEV)
    g.manual_seed(m)
    a, w = torch.randn((m, k), generator=g, device=DEV).to(torch.bfloat16), (torch.randn((n, k), generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    x = torch.randn((m, n), generator=g, device=DEV)
    outs = [ops.linear_t(a, w, residual=x.clone()) for _ in range(6)]
    assert all(torch.equal(o, outs[0]) for o in outs)
    lib.logismos_set_deterministic(1)
    try:
        parts = torch.cat([ops.linear_t(a[i:i + 200].contiguous(), w, residual=x[i:i + 200].clone()) for i in range(0, m, 200)])
    finally:
        lib.logismos_set_deterministic(0)
    assert torch.equal(parts, outs[0])


def tile_of(m, n, k, epilogue, groups=None):
    t = np.zeros(3, np.int32)
    assert lib.logismos_linear_t_tile(m, n, k, epilogue, groups, torch.cuda.get_device_properties(0).multi_processor_count, t.ctypes.data) == 0
    return t.tolist()


@pytest.mark.parametrize("m", [1283, 1409])
@pytest.mark.parametrize("kind", ["bf16", "resid", "swiglu", "glu", "relu2", "f32", "f32 direct", "groups"])
def test_every_epilogue_by_pairs_of_ctas(m, kind):
    """Tiles of 256 x 256 by a pair of CTAs, as the rule is asked to confirm: the second CTA's half of the last tile empty (3 rows) or of one row
    (129), a last column tile of 16 or 13 columns, and every way a tile leaves. Bounds as above; SiLU by an approximate division in the grouped
    and clamped units (2^-21)."""
    from logismos_b200.structs import Groups
    k, n = 1024, {"swiglu": 8192, "glu": 8192, "f32 direct": 8205}.get(kind, 8208)
    g = torch.Generator(device=DEV)
    g.manual_seed(m)
    copies = 3 if kind == "groups" else 1
    a = torch.randn((copies, m, k), generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn((n, k), generator=g, device=DEV) * 0.05).to(torch.bfloat16)
    bias = torch.randn(n, generator=g, device=DEV)
    ref = a[0].float() @ w.float().T
    epilogue = {"bf16": ops.EPI_BF16, "resid": ops.EPI_RESID_F32, "swiglu": ops.EPI_SWIGLU, "glu": ops.EPI_GLU_CLAMP, "relu2": 5, "groups": ops.EPI_BF16}.get(kind, ops.EPI_F32)
    rounding = 0.0 if epilogue in (ops.EPI_RESID_F32, ops.EPI_F32) else 2 ** -8
    if kind == "groups":
        ends, n_main = [2048, 4096, n], 8192
        out, tail = torch.empty((m, n_main), dtype=torch.bfloat16, device=DEV), torch.empty((m, n - n_main), device=DEV)
        gr = Groups(n_groups=3, n_main=n_main, tail=tail.data_ptr(), ld_tail=n - n_main, bias=bias.data_ptr(), silu_begin=2048, silu_end=4096)
        gr.end[:3] = ends
        st = torch.zeros(1, dtype=torch.int32, device=DEV)
        assert tile_of(m, n, k, epilogue, ctypes.byref(gr)) == [256, 1, 1]
        assert lib.logismos_launch_linear_groups_tc_bf16(a.data_ptr(), w.data_ptr(), out.data_ptr(), m, n, k, k, n_main, ctypes.byref(gr), st.data_ptr(), None) == 0
        torch.cuda.synchronize()
        assert int(st) == 0
        ref = torch.cat([a[i].float() @ w[b:e].float().T for i, (b, e) in enumerate(zip([0] + ends, ends))], dim=1)
        assert (tail - ref[:, n_main:]).abs().max() <= 1e-4 * ref.abs().max()
        ref = ref[:, :n_main] + bias[:n_main]
        ref[:, 2048:4096] = torch.nn.functional.silu(ref[:, 2048:4096])
        got = out
    else:
        assert tile_of(m, n, k, epilogue) == [256, 1, 1]
        if kind == "resid":
            x = torch.randn((m, n), generator=g, device=DEV)
            ref = x + ref + bias
            got = ops.linear_act(a[0], w, bias, residual=x)
        elif kind in ("swiglu", "glu"):
            z = (ref + bias).reshape(m, n // 64, 2, 32)
            gate, up = z[:, :, 0], z[:, :, 1]
            if kind == "glu":
                gate, up = gate.clamp(max=2.0), up.clamp(-2.0, 2.0) + 1.0
                ref = (gate * torch.sigmoid(1.7 * gate) * up).reshape(m, n // 2)
            else:
                ref = (torch.nn.functional.silu(gate) * up).reshape(m, n // 2)
            got = ops.linear_act(a[0], w, bias, epilogue=epilogue, p=(1.7, 2.0, 1.0))
        elif kind == "relu2":
            out, st = torch.empty((m, n), dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
            assert lib.logismos_launch_linear_t_act_bf16(a.data_ptr(), w.data_ptr(), bias.data_ptr(), out.data_ptr(), m, n, k, k, n, epilogue, 0.0, 0.0, 0.0, st.data_ptr(), None) == 0
            torch.cuda.synchronize()
            assert int(st) == 0
            got, ref = out, torch.relu(ref + bias) ** 2
        else:
            ref = ref + bias
            got = ops.linear_act(a[0], w, bias, epilogue=epilogue)
    assert ((got.float() - ref).abs() <= rounding * ref.abs() + 1e-4 * ref.abs().max()).all()
