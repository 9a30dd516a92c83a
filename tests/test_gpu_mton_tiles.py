"""The M x N tensor-core kernel with in-kernel decoded code tiles
(distanceBatchMToN / distanceBatchMToNSymmetric / ...Light,
space_turbo_quant.h:588-615, 634-647)
at the edges of its tiles: row counts around its column widths (16 ... 256),
code counts around its 128-code tiles, reductions shorter than one 64-value
K block and longer than one accumulation chunk, every index width, zero rows
and rows of very different norms.  Tolerance: DIST_RTOL of the term scale
(conftest.py), the bar of every distance."""
import numpy as np
import pytest

import oracle as O
import turboquant as tq
from conftest import asym_term_scale, dist_close, sym_term_scale

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,bits", [(16, 4), (20, 8), (32, 2), (64, 3), (100, 5), (128, 4), (384, 4),
                                      (768, 8), (1000, 9), (1536, 4), (4096, 6)])
@pytest.mark.parametrize("m,n", [(9, 1), (16, 127), (17, 128), (64, 129), (65, 300), (129, 257),
                                 (256, 130), (257, 1025)])
def test_tile_edges(cuda_ok, dim, bits, m, n):
    rng = np.random.default_rng(dim * 7 + bits + 31 * m + n)
    X = (rng.standard_normal((n, dim)) * rng.uniform(1e-2, 1e2, (n, 1))).astype(np.float32)
    Q = (rng.standard_normal((m, dim)) * rng.uniform(1e-2, 1e2, (m, 1))).astype(np.float32)
    X[n // 2] = 0.0
    Q[m // 2] = 0.0
    s, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    cs = s.code_size_bytes()
    codes, rows = o.encode_batch(X), o.encode_batch(Q)
    err, ok = dist_close(s.distance_m_to_n(Q, codes), o.distance_m_to_n(Q, codes),
                         asym_term_scale(Q, codes, cs, cs - 12))
    assert ok, ("asymmetric", err.max())
    err, ok = dist_close(s.distance_m_to_n_symmetric(rows, codes),
                         o.distance_m_to_n_symmetric(rows, codes),
                         sym_term_scale(rows, codes, cs, cs - 12))
    assert ok, ("symmetric", err.max())
    err, ok = dist_close(s.distance_m_to_n_symmetric_light(rows, codes),
                         o.distance_m_to_n_symmetric_qjl(rows, codes, "light"),
                         sym_term_scale(rows, codes, cs, cs - 12))
    assert ok, ("light", err.max())


@pytest.mark.parametrize("dim,bits", [(16, 4), (20, 8), (64, 3), (128, 2), (384, 4), (768, 8), (1000, 9),
                                      (1536, 4), (4096, 6)])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 130), (17, 128), (65, 257), (129, 300)])
@pytest.mark.parametrize("variant", ["full", "full_prepared"])
def test_full_form_tile_edges(cuda_ok, dim, bits, m, n, variant):
    """The full QJL form as two passes (the correction's products, then the
    distances with them clamped in)."""
    rng = np.random.default_rng(dim * 5 + bits + 17 * m + n)
    X = (rng.standard_normal((n, dim)) * rng.uniform(1e-2, 1e2, (n, 1))).astype(np.float32)
    Q = (rng.standard_normal((m, dim)) * rng.uniform(1e-2, 1e2, (m, 1))).astype(np.float32)
    X[n // 2], Q[m // 2] = (0.0, 0.0) if n > 1 else (X[0], Q[0])
    Q[0] = X[0]  # a code against itself
    s, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    cs = s.code_size_bytes()
    codes, rows = o.encode_batch(X), o.encode_batch(Q)
    got = getattr(s, f"distance_m_to_n_symmetric_{variant}")(rows, codes)
    err, ok = dist_close(got, o.distance_m_to_n_symmetric_qjl(rows, codes, variant),
                         sym_term_scale(rows, codes, cs, cs - 12))
    assert ok, (variant, err.max())


@pytest.mark.parametrize("dim,bits", [(64, 4), (100, 8), (384, 4)])
@pytest.mark.parametrize("m,n", [(130, 6300), (257, 3801), (520, 2100)])
def test_wide_tiles_with_few_live_columns(cuda_ok, dim, bits, m, n):
    """Code counts at which 128-column tiles over CTA pairs are taken, with a
    last row tile of 2 to 8 rows: its second half of columns lies past the rows."""
    rng = np.random.default_rng(dim + bits + m + n)
    X = (rng.standard_normal((n, dim)) * rng.uniform(1e-2, 1e2, (n, 1))).astype(np.float32)
    Q = (rng.standard_normal((m, dim)) * rng.uniform(1e-2, 1e2, (m, 1))).astype(np.float32)
    s, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    cs = s.code_size_bytes()
    codes, rows = o.encode_batch(X), o.encode_batch(Q)
    scale = sym_term_scale(rows, codes, cs, cs - 12)
    err, ok = dist_close(s.distance_m_to_n_symmetric_light(rows, codes),
                         o.distance_m_to_n_symmetric_qjl(rows, codes, "light"), scale)
    assert ok, ("light", err.max())
    err, ok = dist_close(s.distance_m_to_n_symmetric(rows, codes),
                         o.distance_m_to_n_symmetric(rows, codes), scale)
    assert ok, ("symmetric", err.max())
    err, ok = dist_close(s.distance_m_to_n(Q, codes), o.distance_m_to_n(Q, codes),
                         asym_term_scale(Q, codes, cs, cs - 12))
    assert ok, ("asymmetric", err.max())


def _near(dim, m, seed, n=2048):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, dim)).astype(np.float32)
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    Q = X[:m] + (0.02 / dim ** 0.5) * rng.standard_normal((m, dim)).astype(np.float32)
    return X, np.ascontiguousarray(Q, np.float32)


def _near_errors(d, f64):
    """Errors of each row's near pair, relative to |q|^2 + |x|^2 (about 2)."""
    return (np.array([d[i, i] for i in range(len(f64))], np.float64) - f64) / 2.0


@pytest.mark.parametrize("dim,bits", [(128, 8), (384, 4), (768, 2), (1024, 3), (1536, 2), (1536, 8)])
def test_near_pairs_at_fp32_are_as_accurate_as_the_scan(cuda_ok, dim, bits):
    """Near pairs, whose terms share a sign, are where truncating sums show.  Calls
    of 16 rows (tensor cores) against calls of one row (the scan kernel's FP32
    chains): at most 1.5 times its error, and half an ulp of the sum more.  64 rows
    at once: at most the error of rounding an FP32 chain of 2 D terms, a random walk
    of 2 D half-ulps of a sum that grows to its end."""
    m = 64
    X, Q = _near(dim, m, dim + bits, n=20_000)  # enough codes that 16 rows do not run on the scan
    s, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    codes = o.encode_batch(X)
    f64 = np.array([o.distance_f64(Q[i], codes[i]) for i in range(m)])
    scan = np.concatenate([s.distance_m_to_n(Q[i:i + 1], codes) for i in range(m)])
    few = np.concatenate([s.distance_m_to_n(Q[i:i + 16], codes) for i in range(0, m, 16)])
    rms = lambda e: float(np.sqrt(np.mean(e * e)))  # noqa: E731
    es, ef, ew = (_near_errors(d, f64) for d in (scan, few, s.distance_m_to_n(Q, codes)))
    assert rms(ef) <= 1.5 * rms(es) + 2.0 ** -25, (rms(ef), rms(es))
    assert abs(ef.mean()) <= abs(es.mean()) + 2.0 ** -24, (ef.mean(), es.mean())
    D = 1 << (dim - 1).bit_length()
    assert rms(ew) <= 2.0 ** -25 * (2 * D) ** 0.5, rms(ew)


@pytest.mark.parametrize("dim", [128, 768, 1536])
@pytest.mark.parametrize("bits", [2, 3, 4, 8])
def test_near_pairs_at_split_bf16(cuda_ok, dim, bits):
    """BF16 pairs round each of a few centroid values by up to 2^-17, the same way in
    every term.  With the centroids' scale no such bias is left: near pairs are off
    by 2e-6 on average at most, the truncation of a whole chunk (1.9e-6)."""
    m = 64
    X, Q = _near(dim, m, 3 * dim + bits)
    s, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    codes, rows = o.encode_batch(X), o.encode_batch(Q)
    f64 = np.array([o.distance_f64(Q[i], codes[i]) for i in range(m)])
    e = _near_errors(s.distance_m_to_n(Q, codes, precision="split_bf16"), f64)
    assert abs(e.mean()) <= 2e-6, e.mean()
    f64 = np.array([o.distance_symmetric_f64(rows[i], codes[i]) for i in range(m)])
    e = _near_errors(s.distance_m_to_n_symmetric(rows, codes, precision="split_bf16"), f64)
    assert abs(e.mean()) <= 2e-6, e.mean()


@pytest.mark.parametrize("dim,bits", [(128, 4), (100, 8), (1536, 3)])
@pytest.mark.parametrize("m", [3, 16, 64])
def test_rows_whose_norm_overflows(cuda_ok, dim, bits, m):
    """Vectors whose squared norm overflows FP32 have the norm +inf; against them a
    distance is +inf or 0 by the sign of the inner product, also where a correction
    of the other sign is clamped in.  Rows of NaNs give 0."""
    n = 300
    rng = np.random.default_rng(dim + bits + m)
    X = rng.standard_normal((n, dim)).astype(np.float32)
    Q = rng.standard_normal((m, dim)).astype(np.float32)
    X[::7] *= np.float32(1e25)
    Q[1] *= np.float32(1e25)
    X[5], Q[2] = np.nan, np.nan
    s, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    codes, rows = o.encode_batch(X), o.encode_batch(Q)
    with np.errstate(all="ignore"):
        calls = {
            "asymmetric": (s.distance_m_to_n(Q, codes), o.distance_m_to_n(Q, codes)),
            "symmetric": (s.distance_m_to_n_symmetric(rows, codes), o.distance_m_to_n_symmetric(rows, codes)),
            "light": (s.distance_m_to_n_symmetric_light(rows, codes),
                      o.distance_m_to_n_symmetric_qjl(rows, codes, "light")),
            "full": (s.distance_m_to_n_symmetric_full(rows, codes),
                     o.distance_m_to_n_symmetric_qjl(rows, codes, "full")),
        }
    for form, (got, ref) in calls.items():
        finite = np.isfinite(ref)
        assert (~finite).any(), form
        np.testing.assert_array_equal(got[~finite], ref[~finite].astype(np.float32), err_msg=form)
        np.testing.assert_allclose(got[finite], ref[finite], rtol=1e-4, atol=1e-2, err_msg=form)


def test_a_call_that_gave_up_does_not_touch_others(cuda_ok):
    """A wait that ran out in one call on device arrays shows in the space's device
    status, and nowhere else: later calls give the same distances and no error."""
    import torch
    from turboquant import _capi

    s = tq.TurboQuantSpace(384, 4)
    X = torch.randn(4000, 384, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    codes, q = s.encode_batch(X), X[:70].contiguous()
    hq, hc = q.cpu().numpy(), codes.cpu().numpy()
    rows = codes[:70].contiguous()

    def results():
        out = [s.distance_m_to_n(q, codes), s.distance_m_to_n_symmetric(rows, codes),
               s.distance_m_to_n_symmetric_light(rows, codes), s.distance_m_to_n_symmetric_full(rows, codes)]
        torch.cuda.synchronize()
        out = [t.cpu().numpy() for t in out]
        out += [s.distance_m_to_n(hq, hc), s.distance_1_to_n(hq[0], hc),
                s.distance_m_to_n_symmetric(hc[:70], hc), s.distance_m_to_n_symmetric_full(hc[:70], hc)]
        return out

    want = results()
    s.take_device_status()
    assert _capi.lib().tq_selftest_space_wait(s._h, 50) == _capi.TQ_ERR_TIMEOUT
    for a, b in zip(results(), want):
        np.testing.assert_array_equal(a, b)
    with pytest.raises(tq.TQError) as e:
        s.take_device_status()
    assert e.value.status == _capi.TQ_ERR_TIMEOUT
    s.take_device_status()  # taken


@pytest.mark.parametrize("dim,bits", [(16, 4), (384, 4), (768, 8), (1536, 4)])
@pytest.mark.parametrize("m,pairs", [(3, 20_000), (12, 20_000), (12, 60_000), (31, 200_000), (32, 4_000)])
def test_either_side_of_the_scan_rule(cuda_ok, dim, bits, m, pairs):
    """Fewer than 32 rows run on the scan kernel or the tensor cores by a count of
    their pairs (about 40,000 at wide dims, 170,000 at narrow ones)."""
    n = pairs // m
    rng = np.random.default_rng(dim + bits + m + n)
    X, Q = (rng.standard_normal((r, dim)).astype(np.float32) for r in (n, m))
    s, o = tq.TurboQuantSpace(dim, bits), O.OracleSpace(dim, bits)
    cs = s.code_size_bytes()
    codes, rows = o.encode_batch(X), o.encode_batch(Q)
    err, ok = dist_close(s.distance_m_to_n(Q, codes), o.distance_m_to_n(Q, codes),
                         asym_term_scale(Q, codes, cs, cs - 12))
    assert ok, ("asymmetric", err.max())
    err, ok = dist_close(s.distance_m_to_n_symmetric(rows, codes), o.distance_m_to_n_symmetric(rows, codes),
                         sym_term_scale(rows, codes, cs, cs - 12))
    assert ok, ("symmetric", err.max())
