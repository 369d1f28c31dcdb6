"""Kernels and dispatch rules at the sizes where they can go wrong: host emulations of their
index logic (CPU), and the device against the oracle or the general path (GPU)."""
import math
import re
import subprocess
from pathlib import Path

import numpy as np
import pytest
import torch

import moraine_b200 as mb
from oracle import oracle as O


# ----------------------------------------------------------------------------- KS statistic
def _merge_k(a, b):
    """The reference's merge statistic (moraine/shp.py:36-44)."""
    n, j1, j2, k = len(a), 0, 0, 0
    while j1 < n and j2 < n:
        le, ge = a[j1] <= b[j2], a[j1] >= b[j2]
        j1 += le
        j2 += ge
        k = max(k, abs(j2 - j1))
    return k


def test_ks_walk_and_threshold_equal_the_merge():
    """One-sided walks and the threshold test give the merge's statistic, ties and infinities
    included, reading only inside a row of shared memory."""
    rng = np.random.default_rng(3)
    for n in (1, 2, 3, 4, 5, 7, 16, 17, 33, 50):
        row = 4 * (((n + 11) >> 2) | 1)
        for trial in range(60):
            levels = (2, 5, 1000)[trial % 3]
            a = np.sort(rng.integers(0, levels, n)).astype(np.float64)
            b = np.sort(rng.integers(0, levels, n) + (trial % 4) * levels // 4).astype(np.float64)
            if trial % 7 == 0:
                b[-1] = np.inf
            if trial % 11 == 0:
                b = a.copy()
            k = _merge_k(a, b)
            t = [0, 0]
            for s in range(n):
                assert max(t) <= s
                t = [t[0] + (not b[s] < a[t[0]]), t[1] + (not a[s] < b[t[1]])]
            assert n - min(t) == k
            assert (k == 0) == np.array_equal(a, b)
            pad = np.full(row, np.inf)  # the sentinel: nothing lies below it
            pa, pb = pad.copy(), pad.copy()
            pa[:n], pb[:n] = a, b
            for kth in range(1, n + 2):
                groups = max(0, (n - kth + 4) >> 2)
                assert 4 * ((kth - 1) >> 2) + 3 < row  # the first shifted word, read before the loop
                hit = False
                for g in range(groups):
                    assert 4 * (g + ((kth - 1) >> 2) + 1) + 3 < row
                    for i in range(4 * g, 4 * g + 4):
                        hit |= pb[i + kth - 1] < pa[i] or pa[i + kth - 1] < pb[i]
                assert hit == (k >= kth)


def _select(x, azh, rh, p_max):
    """mr_ks_test without p or dist: the chain's selection."""
    from moraine_b200 import _dev, _lib
    nl, w, n = x.shape
    win = (2 * azh + 1) * (2 * rh + 1)
    is_shp = torch.full((nl, w, win), 7, dtype=torch.uint8, device=x.device)
    num = torch.full((nl, w), -1, dtype=torch.int32, device=x.device)
    ws = _dev.workspace(_lib.load().mr_ks_workspace_bytes(nl, w, n), x.device)
    _lib.call("mr_ks_test", x.data_ptr(), nl, w, n, azh, rh, None, None, p_max, is_shp.data_ptr(), num.data_ptr(),
              ws.data_ptr(), ws.numel(), _dev.stream())
    return is_shp.cpu().numpy().reshape(nl, w, 2 * azh + 1, 2 * rh + 1), num.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("n,azh,rh", [(1, 1, 1), (2, 2, 3), (5, 5, 5), (17, 5, 5), (32, 5, 10), (41, 7, 15),
                                      (101, 5, 10), (150, 2, 15), (257, 1, 10), (512, 0, 4)])
def test_ks_selection_without_p(cuda, n, azh, rh):
    """The mask-only path equals p < p_max of the oracle's p, for every kind of threshold: the
    usual ones, none or all accepted, and tables that accept neither an interval from above."""
    rng = np.random.default_rng(n)
    nl, w = (19, 37) if n < 200 else (7, 35)
    x = rng.exponential(size=(nl, w, n)).astype(np.float32)
    x[:, w // 2:] *= 2.5
    x[3, 5] = x[3, 6]                # an identical neighbour: k = 0 off the centre
    x[4, 7] = np.round(x[4, 7], 1)   # ties
    x[4, 8] = np.round(x[4, 8], 1)
    x[5, 9, 0] = np.nan
    x[6, 3, -1] = np.inf
    p = O.ks_test(x, azh, rh)
    t = torch.from_numpy(x).to(cuda)
    for p_max in (0.05, 0.5, 1e-6, 0.0, -1.0, 1.0, 2.5):
        ref, num = O.select_shp(p, p_max)
        got, got_num = _select(t, azh, rh, p_max)
        np.testing.assert_array_equal(got.astype(bool), ref)
        np.testing.assert_array_equal(got_num, num)
        assert got.max() <= 1
    np.testing.assert_array_equal(mb.ks_test(x, azh, rh), p)


@pytest.mark.gpu
@pytest.mark.parametrize("n,azh,rh", [(5, 4, 0), (17, 0, 0), (41, 5, 0), (100, 1, 1), (200, 0, 5), (512, 1, 1)])
def test_ks_one_offset_per_thread(cuda, n, azh, rh):
    """Windows of one column, and windows so small that groups of offsets would leave threads idle."""
    rng = np.random.default_rng(n)
    x = rng.exponential(size=(11, 23, n)).astype(np.float32)
    x[:, 12:] *= 2.5
    x[3, 5] = x[3, 6]
    x[5, 9, 0] = np.nan
    p = O.ks_test(x, azh, rh)
    np.testing.assert_array_equal(mb.ks_test(x, azh, rh), p)
    for p_max in (0.05, 0.5, 1.0, 2.5):
        ref, num = O.select_shp(p, p_max)
        got, got_num = _select(torch.from_numpy(x).to(cuda), azh, rh, p_max)
        np.testing.assert_array_equal(got.astype(bool), ref)
        np.testing.assert_array_equal(got_num, num)


# ----------------------------------------------------------------------------- coherence
@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 9, 17, 31, 40, 57, 76, 77, 104, 105, 137, 200, 301, 409])
def test_coherence_block_shapes(cuda, n):
    """FP32 and FP64 Gram at the edges of their blocks, warps and rounds, SHP counts from one
    to over two staged passes, points at the border and outside the image."""
    rng = np.random.default_rng(n)
    nl, w, azw, rw = 13, 17, 9, 11
    z = (rng.normal(size=(nl, w, n)) + 1j * rng.normal(size=(nl, w, n))).astype(np.complex64)
    idx = np.array([[6, 8], [0, 0], [12, 16], [5, 3], [7, 9], [6, 7], [2, 15]], np.int32)
    mask = rng.random((len(idx), azw, rw)) < np.array([1, .7, .6, .35, .17, .02, .5])[:, None, None]
    mask[:, azw // 2, rw // 2] = True
    ref = O.emperical_co_pc(z, idx, mask)
    for precision, tol in (("fp32", 2e-6), ("fp64", 1e-7)):
        got = mb.emperical_co_pc(z, idx, mask, precision=precision)
        np.testing.assert_allclose(got, ref, atol=tol, rtol=0)
        out = mb.emperical_co_pc(z, np.array([[6, 8], [-1, 3], [6, 17]], np.int32), mask[:3], precision=precision)
        np.testing.assert_array_equal(out[0], got[0])
        assert np.isnan(out[1:].view(np.float32)).all()
    if n <= 40:
        is_shp = rng.random((nl, w, azw, rw)) < 0.4
        is_shp[..., azw // 2, rw // 2] = True
        cov_ref, coh_ref = O.emperical_co(z, is_shp)
        cov, coh = mb.emperical_co(z, is_shp)
        np.testing.assert_allclose(coh, coh_ref, atol=2e-6, rtol=0)
        np.testing.assert_allclose(cov, cov_ref, atol=2e-6 * np.abs(cov_ref).max(), rtol=0)
        np.testing.assert_array_equal(coh, np.conj(np.swapaxes(coh, -1, -2)))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 8, 9, 16, 17, 24, 25, 32, 33, 40, 41, 56, 57, 65, 72, 73, 81, 97, 104])
def test_coherence_does_not_depend_on_the_batch(cuda, n):
    """A few points (blocks of images spread over the warps) and enough of them to fill the device
    several times over: the same floats."""
    rng = np.random.default_rng(n)
    nl, w, azw, rw = 13, 17, 9, 11
    z = (rng.normal(size=(nl, w, n)) + 1j * rng.normal(size=(nl, w, n))).astype(np.complex64)
    idx = np.stack([rng.integers(0, nl, 23), rng.integers(0, w, 23)], 1).astype(np.int32)
    mask = rng.random((23, azw, rw)) < 0.6
    mask[:, azw // 2, rw // 2] = True
    few = mb.emperical_co_pc(z, idx, mask, precision="fp64")
    np.testing.assert_allclose(few, O.emperical_co_pc(z, idx, mask), atol=1e-7, rtol=0)
    many = mb.emperical_co_pc(z, np.tile(idx, (300, 1)), np.tile(mask, (300, 1, 1)), precision="fp64")
    np.testing.assert_array_equal(many, np.tile(few, (300, 1)))


# ----------------------------------------------------------------------------- streaming statistics
@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 16, 17, 32, 33, 64, 65, 129, 300])
def test_amp_disp_group_shapes(cuda, n):
    """Amplitude dispersion at the edges of the lane groups; near-constant, tiny, huge, zero,
    NaN and infinite amplitudes."""
    rng = np.random.default_rng(n)
    z = (rng.normal(size=(5, 23, n)) + 1j * rng.normal(size=(5, 23, n))).astype(np.complex64)
    z[0, 0] = 3 - 4j                       # constant: exactly 0
    z[0, 1] = (7 + 1e-4 * rng.normal(size=n)).astype(np.complex64)
    z[0, 2] *= 1e-20
    z[0, 3] *= 1e25
    z[0, 4] = 0
    z[0, 5, -1] = np.nan
    z[0, 6, 0] = np.inf
    got = mb.amp_disp(z)
    amp = np.abs(z.astype(np.complex128))
    with np.errstate(all="ignore"):
        ref = amp.std(-1) / amp.mean(-1)
    # one float32 rounding of the result, and half a float32 ulp per amplitude (5e-8 / dispersion)
    tol = 1.2e-7 * np.abs(ref) + 6e-8
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    ok = ~np.isnan(ref)
    assert np.all(np.abs(got - ref)[ok] <= tol[ok])
    assert got[0, 0] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 3, 8, 9, 17, 33, 100, 128, 129])
def test_temp_coh_all_pairs_shapes(cuda, n):
    """Both temporal coherences over all pairs, at the edges of the unrolled walk and of the pair
    table, zero and tiny coherence included."""
    rng = np.random.default_rng(n)
    q = n * (n - 1) // 2
    coh = (rng.normal(size=(37, q)) + 1j * rng.normal(size=(37, q))).astype(np.complex64)
    ph = np.exp(1j * rng.uniform(0, 7, (37, n))).astype(np.complex64)
    coh[1, 0] = 0                          # 0 / 0
    coh[2] *= 1e-15
    np.testing.assert_allclose(mb.ds_temp_coh(coh, ph), O.ds_temp_coh(coh, ph), atol=1e-6)
    np.testing.assert_allclose(mb.temp_coh(coh, ph), O.temp_coh(coh, ph), atol=1e-6)
    assert np.isnan(mb.ds_temp_coh(coh, ph)[1])


# ----------------------------------------------------------------------------- EMI
@pytest.mark.parametrize("rows", [2, 4])
def test_reduction_reads_stay_inside(rows):
    """Every read of the reduction's strips (rows above the first active one and columns past the
    edge included) lies inside the triangle and its 32 spare entries, and inside the padded
    records of the step."""
    def tri(i):
        return i * (i + 1) // 2
    for n in (*range(3, 40), 64, 100, 128, 158, 512):
        for k in range(n - 2):
            tops = range(k + 1, n) if n < 40 else {k + 1, k + 2, k + 5, min(k + 17, n - 1), n - 1}
            for top in (t for t in tops if k < t < n):
                for hi in (top, top - rows):
                    blocks = (top - (k + 1)) // 16
                    assert k + 1 + 16 * blocks + 15 < n + 16
                    for r in range(rows):
                        row = tri(hi) - (r * hi - r * (r - 1) // 2)
                        assert -8 <= hi - r < n and row == tri(hi - r)
                        assert 0 <= row + k + 1 and row + k + 16 + 16 * blocks < tri(n) + 32


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 15, 16, 17, 32, 33, 48, 49, 64, 65, 80, 97, 113, 128, 129, 144, 145, 157, 158, 159,
                               160, 161, 192, 193, 257])
def test_emi_block_shapes(cuda, n):
    """EMI at the edges of its kernels' tiles, warps and matrix placements against LAPACK FP64; a
    point whose |Gamma| is singular gives NaN and leaves its neighbours alone."""
    rng = np.random.default_rng(n)
    npts, looks = (40, 2 * n + 8) if n <= 128 else (7, n + 40)
    z = rng.normal(size=(npts, looks, n)) + 1j * rng.normal(size=(npts, looks, n))
    z += 0.8 * rng.normal(size=(npts, looks, 1)) * np.exp(1j * rng.uniform(0, 6, (npts, 1, n)))
    c = np.einsum("pli,plj->pij", z, z.conj())
    d = np.sqrt(np.einsum("pii->pi", c).real)
    r, s = np.triu_indices(n, 1)
    coh = (c / (d[:, :, None] * d[:, None, :]))[:, r, s].astype(np.complex64)
    ref = n // 2
    ph_r, q_r, gap, cond = O.emi(coh, ref=ref)
    singular = coh.copy()
    singular[3] = 1.0  # |Gamma| = ones
    for precision in ("fp64",) if n > 128 else ("fp64", "fp32"):
        ph, q = mb.emi(coh, ref=ref, precision=precision)
        eps, floor = (1e3 * 1.2e-16, 3e-7) if precision == "fp64" else (4 * 6e-8, 2e-6)
        err = np.abs(np.angle(ph * np.conj(ph_r))).max(-1)
        assert np.all(err <= O.phase_tolerance(cond, gap, eps=eps, floor=floor))
        qtol = np.maximum(1e-5, eps * cond if precision == "fp64" else 1e-5 * cond) * np.maximum(1, np.abs(q_r))
        assert np.all(np.abs(q - q_r) <= qtol)
        ph2, q2 = mb.emi(singular, ref=ref, precision=precision)
        keep = np.arange(npts) != 3
        np.testing.assert_array_equal(ph2[keep], ph[keep])
        assert n == 2 or (np.isnan(ph2[3]).all() and np.isnan(q2[3]))
    if n > 128:
        _, _, route = mb.emi(coh, ref=ref, precision="refine", return_route=True)
        assert (route == 1).all()


# ----------------------------------------------------------------------------- EMI: ownership, memory
def _emi_source():
    return (Path(mb.__file__).parent / "csrc" / "emi_fast.cu").read_text()


def test_reduction_entries_have_one_owner():
    """The reduction's walk with the constants of its source: in every step each entry of the
    trailing triangle is read and written by one lane, no lane touches another's (blocks that meet
    the diagonal included), and every record read exists."""
    src = _emi_source()
    row_pad, col_pad = (int(re.search(rf"\b{name} = (\d+)", src).group(1)) for name in ("kRowPad", "kColPad"))
    guarded = re.search(r"const bool own = left >= r;[^\n]*\n\s*C a = own \? \*e :", src) is not None
    shapes = {int(r) for r in re.findall(r"launch_reduce<double, double, \d+, (\d+), \d+", src)} | {2, 4}
    lc = np.arange(16)
    for rows in sorted(shapes):
        for n in (*range(2, 44), 63, 64, 65, 97, 108, 112, 113, 128, 157, 158, 161, 512):
            for k in range(n - 2) if n < 44 else (0, 1, 2, 15, 16, 17, n // 2, n - 20, n - 4, n - 3):
                seen = np.zeros((n, n), int)
                for top in range(n - 1, k, -2 * rows):
                    for hi in (top, top - rows):
                        assert hi - rows + 1 >= -row_pad
                        for j0 in range(k + 1, top + 1, 16):
                            assert j0 + 15 < n + col_pad
                            for i in range(hi, hi - rows, -1):
                                if j0 + 15 < top - (2 * rows - 1):
                                    assert i > j0 + 15  # all of the block left of the diagonal
                                    seen[i, j0:j0 + 16] += 1
                                    continue
                                own = j0 + lc <= i
                                touched = own if guarded else np.ones(16, bool)
                                assert not (touched & ~own).any(), "an entry of another row is read"
                                if own.any():
                                    assert i > k
                                    seen[i, (j0 + lc)[own]] += 1
                trail = np.arange(n) > k
                want = np.tril(np.ones((n, n), int)) * trail[:, None] * trail[None, :]
                assert np.array_equal(seen, want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [107, 108, 109, 110, 111, 112])
def test_emi_where_the_reduction_changes_its_warps(cuda, n):
    test_emi_block_shapes(cuda, n)


# ----------------------------------------------------------------------------- FP64 Gram: one set of floats
@pytest.mark.gpu
@pytest.mark.parametrize("n", [16, 41, 56, 57, 60, 61, 64, 72, 73, 80, 81, 88, 89, 96, 97, 104, 105, 112, 113, 120, 121, 128])
def test_fp64_gram_is_the_same_on_every_path(cuda, n):
    """A few points, enough of them for the other CTA shapes, and the same images inside a stack too
    long for the tensor instruction: the same floats."""
    rng = np.random.default_rng(n)
    nl, w, azw, rw = 13, 17, 9, 11
    z = (rng.normal(size=(nl, w, 145)) + 1j * rng.normal(size=(nl, w, 145))).astype(np.complex64)
    idx = np.stack([rng.integers(0, nl, 23), rng.integers(0, w, 23)], 1).astype(np.int32)
    mask = rng.random((23, azw, rw)) < 0.6
    mask[:, azw // 2, rw // 2] = True
    few = mb.emperical_co_pc(np.ascontiguousarray(z[..., :n]), idx, mask, precision="fp64")
    np.testing.assert_allclose(few, O.emperical_co_pc(np.ascontiguousarray(z[..., :n]), idx, mask), atol=1e-7, rtol=0)
    many = mb.emperical_co_pc(np.ascontiguousarray(z[..., :n]), np.tile(idx, (30, 1)), np.tile(mask, (30, 1, 1)),
                              precision="fp64")
    np.testing.assert_array_equal(many, np.tile(few, (30, 1)))
    m, j = np.triu_indices(145, 1)
    inside = j < n
    wide = mb.emperical_co_pc(z, idx, mask, precision="fp64")
    np.testing.assert_array_equal(wide[:, inside], few)


_PLAN_CHECK = r"""
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <new>
bool closed = false;
void* operator new(std::size_t n) { if (closed) throw std::bad_alloc(); return std::malloc(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
@SOURCE@
int main() {
  int made = 0;
  closed = true;
  for (int n = 2; n <= kDmmaImages; ++n)
    for (int64_t points : {1, 148, 149, 296, 297, 4736, 4737, 1000000}) {
      GramShape shape;
      GramPlan plan;
      try { plan = plan_gram64(n, points, 148, shape); } catch (...) { std::printf("heap at %d\n", n); return 1; }
      const int nc = (n + 7) / 8, nr = (n + 15) / 16;
      int seen[8][16] = {};
      if (plan.runs < 1 || plan.runs > kMaxRuns || plan.warps != plan.runs || plan.runs > shape.warps) return 2;
      for (int r = 0; r < plan.runs; ++r) {
        const GramRun& g = plan.run[r];
        if (g.cnt > plan.slots || plan.slots > shape.slots || g.c1 > g.cnt || !g.cnt) return 3;
        for (int q = 0; q < g.cnt; ++q) ++seen[q < g.c1 ? g.br1 : g.br2][q < g.c1 ? g.bc1 + q : g.bc2 + q - g.c1];
      }
      for (int i = 0; i < 8; ++i)
        for (int j = 0; j < 16; ++j)
          if (seen[i][j] != (i < nr && j < nc && j >= 2 * i)) { std::printf("n %d block %d %d: %d\n", n, i, j, seen[i][j]); return 4; }
      ++made;
    }
  std::printf("%d plans\n", made);
}
"""


def test_gram_plans_hold_each_block_once_without_the_heap(tmp_path):
    """Every plan of the FP64 tensor kernel deals each block of the triangle to one warp within its CTA
    shape, and is made without an allocation, which could throw through the C interface."""
    src = (Path(mb.__file__).parent / "csrc" / "coh.cu").read_text()
    head = src[src.index("constexpr int kMaxRuns"):src.index("__device__ __forceinline__ void dmma")]
    plans = src[src.index("GramPlan cut_gram64"):src.index("// Whether gram64_kernel takes n images")]
    code = tmp_path / "plans.cpp"
    code.write_text(_PLAN_CHECK.replace("@SOURCE@", "#include <vector>\n" + head + plans))
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", tmp_path / "plans", code], check=True)
    out = subprocess.run([tmp_path / "plans"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def _integers_of_square_sum(total, k, rng):
    """k integers whose squares add up to total."""
    while True:
        a = rng.integers(-900, 900, k - 4)
        rest = total - int((a * a).sum())
        for _ in range(200):
            b = rng.integers(0, int(rest ** 0.5), 2)
            left = rest - int((b * b).sum())
            for c in range(int(max(left, 0) ** 0.5), 0, -1):
                d = math.isqrt(left - c * c)
                if d * d == left - c * c:
                    return np.concatenate([a, b, [c, d]])


@pytest.mark.gpu
@pytest.mark.parametrize("n", [9, 60, 100, 128, 145])
def test_fp64_gram_rounds_like_the_quotient(cuda, n):
    """Integer samples with sums of squares 2^25: every sum is exact, and many quotients lie exactly
    between two floats, where a product with a rounded reciprocal root would fall to either side."""
    rng = np.random.default_rng(n)
    looks, total = 16, 2 ** 25
    base = _integers_of_square_sum(total, 2 * looks, rng)
    rows = []
    for _ in range(n):
        r = base.copy()
        a, b = rng.choice(2 * looks, 2, replace=False)
        r[[a, b]] = r[[b, a]]
        rows.append(r)
    x = np.array(rows).reshape(n, looks, 2)
    zi = x[..., 0] + 1j * x[..., 1]                       # (n, looks)
    num = zi @ zi.conj().T
    m, j = np.triu_indices(n, 1)
    num = num[m, j]
    f = (1.0 / np.sqrt(float(total))) ** 2
    product, quotient = (num.real * f).astype(np.float32), (num.real / total).astype(np.float32)
    assert (product != quotient).sum() > len(m) // 10     # the inputs tell the two apart
    z = np.zeros((5, 5, n), np.complex64)
    z.reshape(25, n)[:looks] = zi.T
    mask = (np.arange(25) < looks).reshape(1, 5, 5)
    got = mb.emperical_co_pc(z, np.array([[2, 2]], np.int32), mask, precision="fp64")[0]
    np.testing.assert_array_equal(got.real, quotient)
    np.testing.assert_array_equal(got.imag, (num.imag / total).astype(np.float32))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [76, 80, 88, 89, 109, 124, 136, 152, 174])
def test_gram_where_the_threads_change(cuda, n):
    """Where a CTA of more threads saves a round: against the oracle, and FP64 the same floats with
    few points and with many."""
    test_coherence_block_shapes(cuda, n)
    rng = np.random.default_rng(n)
    z = (rng.normal(size=(9, 11, n)) + 1j * rng.normal(size=(9, 11, n))).astype(np.complex64)
    idx = np.stack([rng.integers(0, 9, 13), rng.integers(0, 11, 13)], 1).astype(np.int32)
    mask = rng.random((13, 5, 7)) < 0.6
    mask[:, 2, 3] = True
    for precision in ("fp32", "fp64"):
        few = mb.emperical_co_pc(z, idx, mask, precision=precision)
        many = mb.emperical_co_pc(z, np.tile(idx, (30, 1)), np.tile(mask, (30, 1, 1)), precision=precision)
        np.testing.assert_array_equal(many, np.tile(few, (30, 1)))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [80, 109])
def test_raster_where_the_threads_change(cuda, n):
    rng = np.random.default_rng(n)
    z = (rng.normal(size=(5, 7, n)) + 1j * rng.normal(size=(5, 7, n))).astype(np.complex64)
    is_shp = rng.random((5, 7, 5, 7)) < 0.5
    is_shp[..., 2, 3] = True
    cov_ref, coh_ref = O.emperical_co(z, is_shp)
    cov, coh = mb.emperical_co(z, is_shp)
    np.testing.assert_allclose(coh, coh_ref, atol=2e-6, rtol=0)
    np.testing.assert_allclose(cov, cov_ref, atol=2e-6 * np.abs(cov_ref).max(), rtol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [22, 23, 24, 25, 26, 30, 64, 79, 80, 114])
def test_raster_written_in_pairs(cuda, n):
    """Where two values go to a store, and the same floats in buffers that allow one only."""
    from moraine_b200 import _dev, _lib
    rng = np.random.default_rng(n)
    z = (rng.normal(size=(5, 7, n)) + 1j * rng.normal(size=(5, 7, n))).astype(np.complex64)
    is_shp = rng.random((5, 7, 5, 3)) < 0.5
    is_shp[..., 2, 1] = True
    cov_ref, coh_ref = O.emperical_co(z, is_shp)
    cov, coh = mb.emperical_co(z, is_shp)
    np.testing.assert_allclose(coh, coh_ref, atol=2e-6, rtol=0)
    np.testing.assert_allclose(cov, cov_ref, atol=2e-6 * np.abs(cov_ref).max(), rtol=0)
    zt, mt = torch.from_numpy(z).to(cuda), torch.from_numpy(is_shp.astype(np.uint8)).to(cuda)
    size = coh.size
    for cov_at, coh_at in ((0, 1), (1, 0), (1, 1)):
        out = [torch.zeros(size + 2, dtype=torch.complex64, device=cuda) for _ in range(2)]
        _lib.call("mr_emperical_co", zt.data_ptr(), 5, 7, n, mt.data_ptr(), 5, 3, out[0].data_ptr() + 8 * cov_at,
                  out[1].data_ptr() + 8 * coh_at, _dev.stream())
        for buf, at, want in ((out[0], cov_at, cov), (out[1], coh_at, coh)):
            np.testing.assert_array_equal(buf[at:at + size].cpu().numpy(), want.reshape(-1))
            assert not buf[:at].any() and not buf[at + size:].any()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [128, 129, 255, 256, 257, 511, 512])
def test_amp_disp_one_pixel_at_a_time(cuda, n):
    test_amp_disp_group_shapes(cuda, n)


@pytest.mark.parametrize("n", [129, 150, 157, 158, 160, 200, 257, 400, 512])
def test_emi_workspace_of_long_stacks_is_bounded(n):
    """Above 128 images a sub-batch holds 256 MiB of points (reflectors and a few vectors each) or four
    points per SM, and a matrix per SM beside them, whatever the number of points (148 SMs)."""
    from moraine_b200 import _lib
    lib = _lib.load()
    point, matrix = 8 * n * n + 48 * n + 64, 8 * n * n + 8 * n + 16
    for points in (1, 7, 148, 296, 740, 1000, 5224, 10 ** 6):
        most = min(points * point, max(2 ** 28, 4 * 148 * point)) + min(points, 148) * matrix + 8192
        assert lib.mr_emi_workspace_bytes(points, n) <= most


@pytest.mark.gpu
@pytest.mark.parametrize("n", [129, 158, 200])
def test_emi_of_long_stacks_in_sub_batches(cuda, n):
    """More points than a sub-batch holds, and sub-batches that are no whole waves: the same floats."""
    from moraine_b200 import _lib
    rng = np.random.default_rng(n)
    r, s = np.triu_indices(n, 1)
    z = rng.normal(size=(9, n + 30, n)) + 1j * rng.normal(size=(9, n + 30, n))
    z += 0.8 * rng.normal(size=(9, n + 30, 1)) * np.exp(1j * rng.uniform(0, 6, (9, 1, n)))
    c = np.einsum("pli,plj->pij", z, z.conj())
    d = np.sqrt(np.einsum("pii->pi", c).real)
    coh = torch.from_numpy((c / (d[:, :, None] * d[:, None, :]))[:, r, s].astype(np.complex64)).to(cuda)
    ref_ph, ref_q = mb.emi(coh)
    assert np.isfinite(ref_q.cpu().numpy()).all()
    lib = _lib.load()
    try:
        for points, cap in ((2500, 0), (40, 7), (300, 148), (149, 0)):
            assert lib.mr_set_emi_sub_batch(cap) == 0
            pick = torch.arange(points, device=cuda) % 9
            ph, q = mb.emi(coh[pick].contiguous())
            assert torch.equal(ph, ref_ph[pick]) and torch.equal(q, ref_q[pick])
    finally:
        lib.mr_set_emi_sub_batch(0)


# ----------------------------------------------------------------------------- KS plans
def _ks_plan(n, azh, rh):
    import ctypes

    from moraine_b200 import _lib
    th, tw, azc = ctypes.c_int(), ctypes.c_int(), ctypes.c_int()
    rc = _lib.load().mr_ks_plan(n, azh, rh, ctypes.byref(th), ctypes.byref(tw), ctypes.byref(azc))
    return rc, (th.value, tw.value, azc.value)


@pytest.mark.parametrize("n,rh", [(512, 47), (512, 48), (511, 48), (509, 49), (5, 1280), (100, 230)])
def test_ks_plan_where_only_the_statistic_fits(n, rh):
    """A shape that mr_ks_test takes has a plan: one pixel and its row of 2 rh + 1 neighbours fit 200 KiB
    at the statistic kernel's row length."""
    assert (2 * rh + 2) * ((n + 1) | 1) * 4 <= 200 * 1024
    rc, plan = _ks_plan(n, 0, rh)
    assert rc == 0 and min(plan) >= 1


def test_ks_plan_refuses_what_fits_neither():
    assert _ks_plan(512, 0, 60)[0] == -3


@pytest.mark.gpu
def test_ks_plan_is_the_selections(cuda):
    """Tuning the statistic kernel (p asked for) leaves the reported selection plan alone."""
    n, azh, rh = 23, 3, 6
    before = _ks_plan(n, azh, rh)
    x = torch.rand((40, 50, n), device=cuda)
    mb.ks_test(x, azh, rh)
    assert _ks_plan(n, azh, rh) == before
    _select(x, azh, rh, 0.05)
    rc, plan = _ks_plan(n, azh, rh)
    assert rc == 0 and min(plan) >= 1


@pytest.mark.gpu
@pytest.mark.parametrize("n,rh", [(512, 48), (5, 1280)])
def test_ks_selection_where_only_the_statistic_fits(cuda, n, rh):
    rng = np.random.default_rng(n)
    x = rng.exponential(size=(3, 110, n)).astype(np.float32)
    x[:, 60:] *= 1.6
    ref, num = O.select_shp(O.ks_test(x, 0, rh), 0.05)
    got, got_num = _select(torch.from_numpy(x).to(cuda), 0, rh, 0.05)
    np.testing.assert_array_equal(got.astype(bool), ref)
    np.testing.assert_array_equal(got_num, num)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32", "refine", "mixed"])
@pytest.mark.parametrize("n", [2, 3, 5, 17, 33])
def test_emi_singular_point_of_a_short_stack(cuda, n, precision):
    """|Gamma| = ones meets an exact zero pivot at every size, two images included: NaN for that point,
    and nothing else changes."""
    rng = np.random.default_rng(n)
    q = n * (n - 1) // 2
    coh = (0.3 * np.exp(1j * rng.uniform(0, 6, (6, q))) * rng.uniform(0.2, 1, (6, q))).astype(np.complex64)
    ph, quality = mb.emi(coh, precision=precision)
    assert np.isfinite(quality).all()
    coh[3] = 1.0
    ph2, quality2 = mb.emi(coh, precision=precision)
    assert np.isnan(ph2[3]).all() and np.isnan(quality2[3])
    keep = np.arange(6) != 3
    np.testing.assert_array_equal(ph2[keep], ph[keep])
    np.testing.assert_array_equal(quality2[keep], quality[keep])


def _amplitudes_beside_midpoints(count, rng):
    """complex64 samples x + iy of integers with x^2 + y^2 = m^2 + 1, m odd between 2^24 and 2^25: |z| lies
    1 / 2m above the middle m between two floats. (x - 1)(x + 1) = (m - y)(m + y) with m - y = a,
    x = a t + 1, m + y = t (a t + 2)."""
    t = rng.integers(3, 1500, 4_000_000)
    a = rng.integers(2 ** 25, 2 ** 26, t.size) // t ** 2 + 1
    x, b = a * t + 1, t * (a * t + 2)
    m, y = (a + b) // 2, (b - a) // 2
    ok = ((a + b) % 2 == 0) & (m % 2 == 1) & (m > 2 ** 24) & (m < 2 ** 25) & (y > 0)
    ok &= (x == x.astype(np.float32)) & (y == y.astype(np.float32))
    x, y, m = (v[ok][:count] for v in (x, y, m))
    assert len(m) == count and (x * x + y * y == m * m + 1).all()
    return x, y, m


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 9, 30, 100, 129, 300])
def test_amp_disp_rounds_amplitudes_like_the_double_root(cuda, n):
    """One date whose |z| lies just beside the middle between two floats, the others a few ulps away: the
    dispersion shows to which float it was rounded."""
    x, y, m = _amplitudes_beside_midpoints(400, np.random.default_rng(7))
    z = (x + 1j * y).astype(np.complex64)
    a = (m + 1).astype(np.float32)  # the float above the middle
    assert np.array_equal(a, np.sqrt(x.astype(np.float64) ** 2 + y.astype(np.float64) ** 2).astype(np.float32))
    rest = (a + 3 * np.spacing(a)).astype(np.float32)
    stack = np.repeat(rest[:, None], n, axis=1).astype(np.complex64)
    stack[:, n - 1] = z
    d = a.astype(np.float64) - rest
    want = np.sqrt(d * d / n - (d / n) ** 2) / (rest + d / n)
    got = mb.amp_disp(stack.reshape(20, 20, n)).reshape(-1)
    np.testing.assert_allclose(got, want, rtol=1e-6)  # another float would be 33 or 25 % off
