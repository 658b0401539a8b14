"""Rounding noise floor of the FP32 scheme itself (CPU only).

Three FP32 evaluations of the same reference scheme that differ only in
rounding -- the oracle as written, the oracle with FMA contraction (as the
reference's NVRTC-compiled GPU path does), and the oracle with the C library's
logf (as the reference's CPU device does) -- are compared with each other and
with FP64.  Positions stay within 1e-5 relative of each other; velocities of
the stiff NeoHookean workload drift apart by ~1e-2 relative within a few
hundred substeps, which is the scale any FP32 implementation that is not
bit-identical operation for operation will show.
"""

import numpy as np
import pytest

import flatworld_b200 as fw
import oracle
from tests import scenes


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def test_noise_floor_neohookean():
    build = lambda: scenes.plain_large_scene(fw, n=32, hf_offset=0.17)  # noqa: E731
    loops = {p: oracle.OracleLoop(build(), 0.0, precision=p, threads=4) for p in ("f32", "f32fma", "f32libm", "f64")}
    for o in loops.values():
        o.advance(1000)
    st = {p: o.state() for p, o in loops.items()}
    x = {p: s[0] for p, s in st.items()}
    v = {p: s[1] for p, s in st.items()}
    report = {p: (rel(x[p], x["f64"]), rel(v[p], v["f64"])) for p in ("f32", "f32fma", "f32libm")}
    print("vs FP64 after 1000 substeps (x, v):", report)
    for p in ("f32fma", "f32libm"):
        assert rel(x[p], x["f32"]) < 1e-5
    # the FP32 variants are all equally far from FP64
    assert max(r[0] for r in report.values()) < 1e-5


def test_log_method_accuracy():
    """or_logf (the log of the FP32 oracle and of the kernels) against FP64
    log: < 2 ulp on a sweep of [0.5, 2) (the range of J in the workloads) and
    across the float range; exact specials."""
    from oracle.scene import log32
    rng = np.random.default_rng(0)
    xs = np.concatenate([np.linspace(0.5, 2.0, 20001), 10.0 ** rng.uniform(-37, 38, 20000)]).astype(np.float32)
    worst = 0.0
    for x in xs:
        ref = np.log(np.float64(x))
        got = log32(x)
        r32 = np.float32(ref)
        ulp = float(np.spacing(np.abs(r32)))
        worst = max(worst, abs(got - ref) / ulp)
    assert worst < 2.0, worst
    assert log32(1.0) == 0.0 and log32(0.0) == -np.inf and np.isnan(log32(-1.0)) and log32(np.inf) == np.inf


def _device_log(x, quotient=False):
    import torch

    from flatworld_b200 import _native

    t = torch.from_numpy(x).cuda()
    out, q = torch.empty_like(t), torch.empty_like(t)
    rc = _native.lib().fw_log_f32(t.data_ptr(), out.data_ptr(), q.data_ptr() if quotient else None, t.numel(),
                                  torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    return (out.cpu().numpy(), q.cpu().numpy()) if quotient else out.cpu().numpy()


def _same_bits(a, b):
    same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
    assert same.all(), (int((~same).sum()), int(np.flatnonzero(~same)[0]))


@pytest.mark.gpu
def test_device_quotient_is_the_division_on_every_mantissa():
    """The kernels form the logarithm's quotient without a division: equal to it for all 2^23 arguments."""
    m = np.arange(0x3F3504F4, 0x3FB504F4, dtype=np.uint32).view(np.float32)
    assert len(m) == 1 << 23 and m[0] ** 2.0 > 0.5 and m[-1] ** 2.0 <= 2.0
    one = np.float32(1.0)
    _same_bits(_device_log(m, quotient=True)[1], (m - one) / (m + one))


@pytest.mark.gpu
@pytest.mark.parametrize("sample", ["near one", "bit patterns", "edges"])
def test_device_log_is_the_oracles(sample):
    """The kernels' logarithm against the CPU oracle's: subnormals, zeros, negatives, infinities and NaN included."""
    from oracle.scene import log32

    if sample == "near one":  # every 64th float of [0.5, 2)
        bits = np.arange(0x3F000000, 0x40000000, 64, dtype=np.uint32)
    elif sample == "bit patterns":  # all signs and exponents
        bits = np.random.default_rng(5).integers(0, 1 << 32, 300_000, dtype=np.uint32)
    else:  # both sides of each power of two and of each change of the reduced mantissa
        exps = np.arange(0, 256, dtype=np.uint32) << np.uint32(23)
        near = np.arange(-3, 4).astype(np.int64)
        bits = np.concatenate([(exps[:, None].astype(np.int64) + near[None] + off).ravel()
                               for off in (0, 0x3504F4)]).astype(np.uint64) & np.uint64(0xFFFFFFFF)
        bits = np.concatenate([bits.astype(np.uint32), bits.astype(np.uint32) | np.uint32(0x80000000)])
    x = bits.view(np.float32)
    _same_bits(_device_log(x), np.array([log32(v) for v in x], np.float32))
