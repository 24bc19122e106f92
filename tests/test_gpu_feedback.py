"""T3 -> r1, r2, W_vooo, W_vvvo feedback on the GPU against the oracle's
literal per-block restatement (distr_cc/rccsdt.py:253-366).  FP64: 1e-11
relative to the largest entry."""
import itertools

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from dcc import t3_feedback
    from oracle import feedback_ref
    return t3_feedback, feedback_ref


def _inputs(no, nv, seed):
    rng = np.random.default_rng(seed)
    nmo = no + nv
    g = rng.standard_normal((nmo,) * 4) * 0.1
    fock = rng.standard_normal((nmo, nmo)) * 0.1
    full = rng.standard_normal((no,) * 3 + (nv,) * 3)
    U = sum(full.transpose(p + tuple(3 + x for x in p)) for p in itertools.permutations(range(3))) / 6
    t3 = np.stack([U[i, j, k] for i in range(no) for j in range(i, no) for k in range(j, no)])
    ijk = np.array([(i, j, k) for i in range(no) for j in range(i, no) for k in range(j, no)], dtype=np.int32)
    return g, fock, t3, ijk, rng


@pytest.mark.parametrize("no,nv", [(3, 5), (4, 10)])
def test_r1_r2(mods, oracle, no, nv):
    fb, ref = mods
    g, fock, t3, ijk, rng = _inputs(no, nv, nv)
    r1, r2 = rng.standard_normal((no, nv)), rng.standard_normal((no, no, nv, nv))
    w1, w2 = ref.r1r2_add_t3_ref(fock, g, r1, r2, t3, no, oracle)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    d1, d2, dg, dt3 = dev(r1), dev(r2), dev(g), dev(t3)
    fb.r1_add_t3_(d1, dg, dt3, dev(ijk), no)
    X = fb.p3_201_all(dt3, no)
    fb.r2_add_t3_(d2, dev(fock), dg, X, no)
    np.testing.assert_allclose(d1.cpu().numpy(), w1, rtol=0, atol=1e-11 * np.abs(w1).max())
    np.testing.assert_allclose(d2.cpu().numpy(), w2, rtol=0, atol=1e-11 * np.abs(w2).max())


@pytest.mark.parametrize("no,nv", [(3, 5), (4, 10)])
def test_intermediates(mods, oracle, no, nv):
    fb, ref = mods
    g, fock, t3, ijk, rng = _inputs(no, nv, 3 + nv)
    Wo, Wv = rng.standard_normal((nv, no, no, no)), rng.standard_normal((nv, nv, nv, no))
    w1, w2 = ref.intermediates_t3_add_ref(g, Wo, Wv, t3, no, oracle)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    dWo, dWv, dt3 = dev(Wo), dev(Wv), dev(t3)
    X = fb.p3_201_all(dt3, no)
    fb.intermediates_t3_add_(dWo, dWv, dev(g), X, no)
    np.testing.assert_allclose(dWo.cpu().numpy(), w1, rtol=0, atol=1e-11 * np.abs(w1).max())
    np.testing.assert_allclose(dWv.cpu().numpy(), w2, rtol=0, atol=1e-11 * np.abs(w2).max())


@pytest.mark.parametrize("no,nv", [(1, 3), (2, 1), (3, 31), (3, 32), (2, 33), (2, 65), (2, 96), (2, 97), (1, 128)])
def test_r1_kernel(mods, no, nv):
    """The one-pass r1 kernel at the edges of its z tiles (32, 64, 96, 128) and of its groups of four
    first indices, against the batched GEMMs of the same sums on the CPU (1e-12 of the largest
    entry: sums of 9 nvir^2 products per block in another order)."""
    fb, _ = mods
    g = torch.Generator().manual_seed(nv)
    ijk = torch.tensor([(i, j, k) for i in range(no) for j in range(i, no) for k in range(j, no)], dtype=torch.int32)
    t3 = torch.randn(ijk.shape[0], nv, nv, nv, dtype=torch.float64, generator=g)
    E = torch.randn(no, no, nv, nv, dtype=torch.float64, generator=g)
    r1 = torch.randn(no, nv, dtype=torch.float64, generator=g)
    want = fb.r1_add_t3_(r1.clone(), None, t3, ijk, no, oovv=E)
    got = fb.r1_add_t3_(r1.cuda(), None, t3.cuda(), ijk.cuda(), no, oovv=E.cuda())
    scale = max(float((want - r1).abs().max()), float(r1.abs().max()))
    assert float((got.cpu() - want).abs().max()) <= 1e-12 * scale


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("no,nv", [(1, 1), (2, 16), (3, 17), (5, 7)])
def test_r2_fock(mods, dtype, no, nv):
    """The one-launch Fock term (fewer and more than one CTA of (b, c) per (y, z)) against the
    einsum of the same values in FP64 (1e-13: sums of nocc nvir products in another order)."""
    from dcc import _c_rccsdt
    g = torch.Generator(device="cuda").manual_seed(nv)
    X = torch.randn((no,) * 3 + (nv,) * 3, dtype=torch.float64, device="cuda", generator=g).to(dtype)
    f = torch.randn(no, nv, dtype=torch.float64, device="cuda", generator=g)
    r2 = torch.randn(no, no, nv, nv, dtype=torch.float64, device="cuda", generator=g)
    want = r2 + 0.5 * torch.einsum("xa,xyzabc->yzbc", f, X.double())
    _c_rccsdt.t3_r2_fock_(r2, X, f, no, nv, 0.5)
    assert float((r2 - want).abs().max()) <= 1e-13 * float(want.abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("no,nv", [(1, 3), (4, 9), (6, 4), (3, 17), (129, 1)])
def test_split_feedback(mods, no, nv, dtype):
    """The grouped feedback of the split precisions against the FP64 strings (1e-5 of the largest entry:
    a bf16 pair keeps an operand to 2^-18 = 4e-6, errors of random sign over the summed products): fewer and more virtual than occupied indices, and more
    values of x than a table holds; also the W strings by themselves."""
    fb, _ = mods
    g = torch.Generator(device="cuda").manual_seed(no)
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    X = r(no, no, no, nv, nv, nv).to(dtype)
    E = {"vovv": r(nv, no, nv, nv), "ooov": r(no, no, no, nv), "oovv": r(no, no, nv, nv)}
    z = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")  # noqa: E731
    want = (z(no, no, nv, nv), z(nv, no, no, no), z(nv, nv, nv, no))
    Xd = X.double()
    fb.r2_add_t3_x_(want[0], z(no, nv), E["vovv"], E["ooov"], Xd)
    fb.intermediates_t3_add_x_(want[1], want[2], E["oovv"], Xd)
    s = fb.SplitFeedback(no, nv, "bf16x3")
    got = tuple(torch.zeros_like(w) for w in want)
    s.run(X, E, {"r2": got[0], "W_vooo": got[1], "W_vvvo": got[2]})
    alone = tuple(torch.zeros_like(w) for w in want[1:])
    s.run(X, {"oovv": E["oovv"]}, {"W_vooo": alone[0], "W_vvvo": alone[1]}, names=("wvooo", "wvvvo"))
    assert int(s.status.item()) == 0
    for a, b in list(zip(got, want)) + list(zip(alone, want[1:])):
        assert float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.parametrize("no,nv", [(3, 5), (255, 1), (256, 1), (260, 2)])
def test_fock_term(no, nv):
    """The iteration's f_ov term on either side of the one-launch kernel's limit (nocc < 256) against the
    einsum in FP64 (beyond it the products are those of X's type: 1e-6 of the largest entry)."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from types import SimpleNamespace
    from dcc.t3_iteration import T3Iteration
    g = torch.Generator(device="cuda").manual_seed(no)
    X = torch.randn((no,) * 3 + (nv,) * 3, dtype=torch.float32, device="cuda", generator=g)
    f = torch.randn(no, nv, dtype=torch.float64, device="cuda", generator=g)
    r2 = torch.randn(no, no, nv, nv, dtype=torch.float64, device="cuda", generator=g)
    want = r2 + 0.5 * (f.view(no, 1, nv, 1) * X.view(no, no * no, nv, nv * nv)).sum((0, 2)).view_as(r2)
    T3Iteration._fock_term_(SimpleNamespace(no=no, nv=nv, _X=X), r2, f)
    assert float((r2 - want).abs().max()) <= 1e-6 * float(want.abs().max())
