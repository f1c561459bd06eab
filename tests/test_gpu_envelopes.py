"""The spline solve and the envelope evaluation at the sizes where their
branches change, bit for bit against the oracle: systems of 30-70 rows (the
cyclic reduction stops early from 33 on), right-hand sides whose magnitudes
span too much for that, exactly periodic traces (zero end couplings), very
uneven spacings, spacings past the reciprocal table, plateaus and nbsym 1-3
(searched segments), on both time axes, every instance and both types."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _zigzag(rng, n, knots, grow=0.0, even=False):
    """`knots` alternating extrema joined by straight lines; |value| grows by
    2^grow from first to last."""
    if even:
        step = n // (knots + 1)
        at = step * np.arange(1, knots + 1)
    else:
        at = np.sort(rng.choice(np.arange(2, n - 2, 2), size=knots, replace=False))
    v = np.where(np.arange(knots) % 2 == 0, 1.0, -1.0)
    if not even:
        v = v * rng.uniform(0.5, 2.0, size=knots)
    v = v * 2.0 ** (grow * np.arange(knots) / max(knots - 1, 1))
    return np.interp(np.arange(n), np.r_[0, at, n - 1], np.r_[0.3 * v[0], v, 0.2 * v[-1]])


def _traces():
    rng = np.random.default_rng(23)
    out = [_zigzag(rng, 900, k) for k in (5, 9, 32, 58, 59, 60, 61, 62, 63, 64, 65, 66, 70, 128, 131, 200, 400)]
    out += [_zigzag(rng, 900, k, grow=g) for k in (70, 200) for g in (20.0, 44.0, 50.0, 90.0, 400.0)]
    out += [_zigzag(rng, 900, k, even=True) for k in (8, 61, 66, 89, 149)]
    # dense noise at both ends, one smooth stretch between
    x = _zigzag(rng, 900, 160)
    x[300:600] = x[300] + (x[600] - x[300]) * np.arange(300) / 300.0
    out.append(x)
    out.append(np.where(np.arange(900) % 3 == 0, 1.0, -1.0) + 0.1 * rng.normal(size=900))
    p = _zigzag(rng, 900, 66)
    p[100:104] = p[100]                               # a plateau: searched segments
    out.append(p)
    return np.stack(out)


def _envelopes(O, x, T, nbsym):
    e = O.find_extrema(x)
    if e.ind_max.size < 1 or e.ind_min.size < 1 or e.ind_max.size + e.ind_min.size <= 2:
        return np.zeros_like(x), np.zeros_like(x)
    (pu, vu), (pd, vd), _ = O.mirror_knots(T, x, e.ind_max, e.ind_min, nbsym)
    return O.envelope(T, pu, vu)[0], O.envelope(T, pd, vd)[0]


@pytest.mark.parametrize("real", ["double", "float"])
@pytest.mark.parametrize("nbsym", [1, 2, 3])
@pytest.mark.parametrize("axis", ["arange", "given"])
def test_envelopes_equal_the_oracle(real, nbsym, axis):
    import torch
    from cuda_emd import EMDKernelConfig
    from oracle import emd_oracle as O
    dt = np.float64 if real == "double" else np.float32
    with np.errstate(over="ignore"):
        X = _traces().astype(dt)
    if real == "float":
        X = X[np.isfinite(X).all(1) & (np.abs(X).max(1) < 2.0 ** 60)]
    n = X.shape[1]
    T = np.arange(n, dtype=dt) if axis == "arange" else np.cumsum(
        np.random.default_rng(3).uniform(1.0, 3.0, size=n)).astype(dt)
    L = EMDKernelConfig(nbsym=nbsym, real_t=real).build()
    got = L.run_envelope_only(torch.from_numpy(X).cuda(),
                              None if axis == "arange" else torch.from_numpy(T).cuda())
    upper, lower = got[0].cpu().numpy(), got[1].cpu().numpy()
    for i in range(X.shape[0]):
        u, d = _envelopes(O, X[i], T, nbsym)
        assert upper[i].tobytes() == u.astype(dt).tobytes(), i
        assert lower[i].tobytes() == d.astype(dt).tobytes(), i


@pytest.mark.parametrize("variant", [4, 2, 1])
@pytest.mark.parametrize("axis", ["arange", "given"])
def test_sift_passes_equal_the_oracle(variant, axis):
    import torch
    from cuda_emd import EMDKernelConfig
    from oracle import emd_oracle as O
    X = _traces()
    n = X.shape[1]
    T = np.arange(n, dtype=np.float64) if axis == "arange" else np.cumsum(
        np.random.default_rng(3).uniform(1.0, 3.0, size=n))
    cfg = EMDKernelConfig(max_iteration=12, max_imfs=6)
    L = cfg.build()
    L._plan.set_variant(variant)
    got = [o.cpu().numpy() for o in L.run(torch.from_numpy(X).cuda(), None if axis == "arange"
                                          else torch.from_numpy(T).cuda())]
    for i in range(X.shape[0]):
        r = O.emd_signal(X[i], T, O.OracleConfig(max_iteration=12, max_imfs=6))
        assert int(got[1][i]) == r.n_imfs, i
        assert got[0][i].tobytes() == r.imfs.tobytes(), i


def test_spacing_past_the_reciprocal_table():
    import torch
    from cuda_emd import EMDKernelConfig
    from oracle import emd_oracle as O
    n = 40000
    t = np.arange(n, dtype=np.float64)
    x = np.sin(t / 40.0) * np.exp(-t / 400.0) + 1e-3 * np.cos(2 * np.pi * t / 21000.0)
    x += np.sin((n - t) / 30.0) * np.exp(-(n - t) / 300.0)
    e = O.find_extrema(x)
    assert max(np.diff(e.ind_max).max(), np.diff(e.ind_min).max()) > 16384
    cfg = dict(max_iteration=4, max_imfs=4)
    got = EMDKernelConfig(**cfg).build().run(torch.from_numpy(x[None]).cuda(), None)
    r = O.emd_signal(x, t, O.OracleConfig(**cfg))
    assert got[0][0].cpu().numpy().tobytes() == r.imfs.tobytes()


@pytest.mark.parametrize("nbsym", [1, 2, 3, 7, 8])
@pytest.mark.parametrize("n", [7, 12, 33, 40])
def test_mirroring_of_few_extrema_equals_the_oracle(n, nbsym):
    """A handful of extrema per side, fewer and more than nbsym, every order of
    first and last kind and both sides of the end-sample tests."""
    import torch
    from cuda_emd import EMDKernelConfig
    from oracle import emd_oracle as O
    rng = np.random.default_rng(100 * n + nbsym)
    X = rng.normal(size=(120, n))
    X[::2] = np.cumsum(X[::2], axis=1)               # smoother: fewer extrema
    X[::5, [0, -1]] *= 8.0                            # end samples beyond their neighbours
    T = np.arange(n, dtype=np.float64)
    got = EMDKernelConfig(nbsym=nbsym).build().run_envelope_only(torch.from_numpy(X).cuda(), None)
    upper, lower = got[0].cpu().numpy(), got[1].cpu().numpy()
    for i in range(X.shape[0]):
        u, d = _envelopes(O, X[i], T, nbsym)
        assert upper[i].tobytes() == u.tobytes() and lower[i].tobytes() == d.tobytes(), i


@pytest.mark.parametrize("scale", [1.0, 1e-170, 1e150])
def test_spacings_and_values_of_any_magnitude(scale):
    """Operands that the quotients without range tests do not cover: spacings
    over a range of 2^40, axes far from 1, moments far from 1, knots of -0 and
    +0 side by side."""
    import torch
    from cuda_emd import EMDKernelConfig
    from oracle import emd_oracle as O
    rng = np.random.default_rng(31)
    n = 700
    X = [_zigzag(rng, n, k) * v for k in (9, 62, 66, 150) for v in (1.0, 1e-120, 1e120)]
    z = _zigzag(rng, n, 150)
    z[z > 0.0] = np.where(rng.random(int((z > 0.0).sum())) < 0.5, 0.0, -0.0)
    X = np.stack(X + [z])
    step = np.ones(n - 1)
    step[300:320] = 2.0 ** rng.uniform(0, 40, size=20)
    T = np.concatenate([[0.0], np.cumsum(step)]) * scale
    L = EMDKernelConfig().build()
    got = L.run_envelope_only(torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda())
    run = [o.cpu().numpy() for o in EMDKernelConfig(max_iteration=4, max_imfs=4).build().run(
        torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda())]
    for i in range(X.shape[0]):
        with np.errstate(all="ignore"):
            u, d = _envelopes(O, X[i], T, 2)
            r = O.emd_signal(X[i], T, O.OracleConfig(max_iteration=4, max_imfs=4))
        for a, b in ((got[0][i].cpu().numpy(), u), (got[1][i].cpu().numpy(), d), (run[0][i], r.imfs)):
            same = (a.view(np.int64) == b.view(np.int64)) | (np.isnan(a) & np.isnan(b))
            assert same.all(), (i, int((~same).sum()))
