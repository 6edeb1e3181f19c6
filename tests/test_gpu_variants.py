"""GPU tests of the kernels chosen by size, at the edges of their ranges."""
import numpy as np
import pytest

from oracle import oracle as O
from projects_b200 import gridrec as G
from projects_b200 import phantom as ph

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n,a,C_,S", [(9, 5, 6.0, 16), (16, 7, 4.0, 5), (64, 48, 6.0, 7),
                                      (90, 45, 7.0, 15), (130, 33, 5.0, 11), (257, 60, 6.0, 13),
                                      (256, 300, 6.0, 16), (250, 310, 6.0, 6),
                                      (9, 5, 6.0, 1), (64, 48, 6.0, 2), (90, 45, 7.0, 3),
                                      (130, 33, 5.0, 4), (256, 300, 6.0, 1), (257, 310, 6.0, 4)])
def test_group_gridding_same_bits(n, a, C_, S):
    """Chunks of 1 to 8 pairs (whole and partly filled groups of 1, 2, 4 and 8, an odd slice at the
    end, split centre sub-tiles at 256 x 300): the bits of the kernel whose work list the
    groups follow, tiles up to 6 pairs and 16 pairs above (the oracle's tests hold those)."""
    th = ph.angles_deg(a)
    rng = np.random.default_rng(n + a)
    centers = (n / 2 + rng.uniform(-1.5, 1.5, S)).astype(np.float32)
    sinos = np.stack([ph.random_ellipse_sinogram(n + a + s, n, a, center=float(c))[0]
                      for s, c in enumerate(centers)])
    outs = []
    for mode in (0, -1 if (S + 1) // 2 < 7 else 1):
        with G.Plan(n, a, th, filter=G.FILTER_HANN, pswf_c=C_, max_pairs=8, wide_grid=mode) as plan:
            M0 = plan.M0
            o = torch.full((S, M0, max(M0, n)), float("nan"), device="cuda")
            plan.reconstruct_batch(_dev(sinos), o, centers=_dev(centers))
            torch.cuda.synchronize()
            plan.device_status()
            outs.append(o.cpu().numpy()[:, :, :M0])
    np.testing.assert_array_equal(outs[0], outs[1])


@pytest.mark.parametrize("n,a,S,group", [(16, 5, 1, 4), (32, 40, 3, 4), (64, 45, 7, 4),
                                         (128, 33, 5, 3), (256, 21, 2, 1)])
def test_fbp_groups_same_bits_and_oracle(n, a, S, group):
    """Slices backprojected in groups of 4, 2 and 1 (every remainder of the call and of the
    plan's slice count): the bits of one slice at a time, whose row filter packs the same
    rows, and the oracle's image."""
    th = np.linspace(0.0, 179.0, a).astype(np.float32)
    rng = np.random.default_rng(n + S)
    sinos = rng.uniform(-1.0, 6.0, (S, a, n)).astype(np.float32)  # values beyond 5 are gated
    f = G.FBP(n, a, th, max_slices=group)
    got = f.reconstruct(_dev(sinos)).cpu().numpy()
    f.close()
    one = G.FBP(n, a, th, max_slices=1)
    for s in range(S):
        alone = one.reconstruct(_dev(sinos[s:s + 1])).cpu().numpy()[0]
        np.testing.assert_array_equal(got[s], alone)
        ref = O.port_optimized_fbp(sinos[s], th)
        assert ph.rel_l2(got[s], ref) < 1e-5
    one.close()


@pytest.mark.parametrize("n,a,S", [(4, 3, 1), (12, 40, 2), (512, 37, 3), (516, 5, 2), (1024, 130, 2),
                                   (1028, 33, 1), (2048, 70, 3), (2052, 9, 2), (4096, 21, 2),
                                   (4100, 11, 1)])
def test_ring_removal_widths_and_row_values(n, a, S):
    """Widths at the edges of the vector kernels (and one beyond them), with rows that
    leave the one-reciprocal division: all zero, mean 0 but not zero, samples near the
    smallest normal float, a row mean above 2^40.  Against the float64 oracle, and the
    scalar kernels on the same data off its 16-byte alignment."""
    rng = np.random.default_rng(n + a)
    x = rng.uniform(0.1, 2.0, (S, a, n)).astype(np.float32)
    x[rng.uniform(size=x.shape) < 0.04] = 0.0
    x[0, 0] = 0.0
    x[-1, 1, ::2], x[-1, 1, 1::2] = 0.5, -0.5  # mean 0
    x[0, 2, : n // 2] = 2e-38
    ref = np.stack([O.port_ring_removal(s, 1.0, 5) for s in x])
    got = G.ring_removal(_dev(x), 1.0, 5)
    buf = torch.empty(x.size + 1, device="cuda")
    off = buf[1:].view(x.shape)
    off.copy_(_dev(x))
    G.ring_removal(off, 1.0, 5)
    # FP32 rounds against float64: the bound of the other ring tests
    assert ph.rel_l2(got.cpu().numpy(), ref) < 2e-5
    assert ph.rel_l2(off.cpu().numpy(), ref) < 2e-5
    y = x.copy()
    y[0, 0] = 2.0 ** 50
    ref = np.stack([O.port_ring_removal(s, 1.0, 5) for s in y])
    assert ph.rel_l2(G.ring_removal(_dev(y), 1.0, 5).cpu().numpy(), ref) < 2e-5


@pytest.mark.parametrize("shape", [(1, 4, 5), (1, 1, 70), (1, 3, 65), (3, 9, 64), (2, 70, 127),
                                   (1, 130, 63), (2, 200, 130)])
def test_network_gradients_ragged_shapes(shape):
    """Loss and weight gradients at image sizes around the strip kernels' 64 columns and 16
    pixels, one row, one segment per row and several rows per segment: the float64 oracle
    with BF16 activations, the bound of the other gradient test."""
    from oracle import cnn_oracle as CO
    from projects_b200 import learned as L
    rng = np.random.default_rng(sum(shape))
    p = L.init_params(4)
    p[144:160] = rng.normal(0, 0.1, 16)
    p[2464:2480] = rng.normal(0, 0.1, 16)
    p[2480:] = rng.normal(0, 0.05, 145)
    x = rng.normal(0, 1, shape).astype(np.float32)
    t = (x + rng.normal(0, 0.3, shape)).astype(np.float32)
    net = L.CorrectionNet(p)
    loss = net.loss_and_grads(_dev(x), _dev(t))
    g = net.grads.cpu().numpy().astype(np.float64)
    q = p.astype(np.float64).copy()
    q[160:2464] = CO._bf16(p[160:2464])
    ref_loss, ref = CO.loss_and_grads(q, x, t, bf16=True)
    assert abs(loss - ref_loss) <= 2e-3 * ref_loss
    for a, b in ((0, 144), (144, 160), (160, 2464), (2464, 2480), (2480, 2624), (2624, 2625)):
        err = np.linalg.norm(g[a:b] - ref[a:b]) / max(np.linalg.norm(ref[a:b]), 1e-30)
        assert err < 2e-2, (a, err)


@pytest.mark.parametrize("n,a,S,pairs", [(8, 5, 1, 1), (33, 20, 3, 1), (64, 45, 5, 2), (100, 60, 4, 4),
                                           (600, 9, 3, 2), (1030, 6, 3, 1)])
def test_padded_window_same_bits(n, a, S, pairs):
    """The padded reconstruction shifts and pads as it forms the spectra and transforms and
    writes its centre window only: the bits of the whole image reconstructed from the
    padded rows, then cropped (rows aligned and not, odd widths, an odd last slice, several
    chunks)."""
    th = ph.angles_deg(a)
    rng = np.random.default_rng(n + S)
    sinos = _dev(rng.uniform(0.0, 2.0, (S, a, n)).astype(np.float32))
    shift = 0.75 if S != 3 else -1.5 - 2 * n  # taps inside the row, all beyond its end
    with G.Plan(2 * n, a, th, filter=G.FILTER_HANN, max_pairs=pairs) as plan:
        got = G.reconstruct_padded(plan, sinos, shift)
        whole = torch.empty((S, plan.M0, max(plan.M0, 2 * n)), device="cuda")
        padded = G.shift_pad(sinos, torch.full((S,), shift), out_width=2 * n)
        plan.reconstruct_batch(padded, whole)
        want = G.crop_center(whole, n, n // 2)
        torch.cuda.synchronize()
        plan.device_status()
    np.testing.assert_array_equal(got.cpu().numpy()[..., :n], want.cpu().numpy())


@pytest.mark.parametrize("lo,hi,nbins", [(-0.5, 1.5, 7), (0.0, 1.0, 1023), (-1e-3, 3e-3, 10000),
                                         (0.0, 1e-30, 5), (-1e35, 1e35, 11)])
def test_entropy_bins_at_their_edges(lo, hi, nbins):
    """Pixels on and next to every bin edge, zeros of both signs, denormals, infinities, NaN and
    the largest values: the counts of the float32 quotient truncated as a host cast does."""
    inv = np.float32(np.float32(hi) - np.float32(lo)) / np.float32(nbins)
    edges = (np.float32(lo) + np.arange(-2, nbins + 3, dtype=np.float32) * inv).astype(np.float32)
    x = np.concatenate([edges, np.nextafter(edges, np.float32(np.inf)),
                        np.nextafter(edges, np.float32(-np.inf)),
                        np.float32([0.0, -0.0, 1e-45, -1e-45, np.inf, -np.inf, np.nan, 3e38, -3e38])])
    x = np.resize(x, (2, 9, (x.size + 17) // 18)).astype(np.float32)
    with np.errstate(all="ignore"):
        f = ((x - np.float32(lo)) / inv).astype(np.float32)
    f = f[np.isfinite(f) & (np.abs(f) < 2.0 ** 31)]
    k = np.trunc(f).astype(np.int64)
    counts = np.bincount(k[(k >= 0) & (k <= nbins)], minlength=nbins + 1)
    p = counts[counts > 0] / x.size
    want = -(p * np.log2(p)).sum()
    got = G.entropy(_dev(x), lo, hi, nbins, group=2).cpu().numpy()
    assert abs(float(got[0]) - want) <= 1e-6 * max(1.0, want)  # a float32 result


@pytest.mark.parametrize("n,ring_group", [(200, 8), (512, 8), (600, 8), (1100, 4), (2100, 4), (4100, 2)])
def test_persistent_columns_same_bits(n, ring_group):
    """The persistent column FFT at M = 256 .. 8192 (widest strips of each) against one strip
    per block on the same input."""
    a, S = 7, 3
    rng = np.random.default_rng(n)
    sinos = _dev(rng.uniform(0.0, 2.0, (S, a, n)).astype(np.float32))
    outs = []
    with G.Plan(n, a, ph.angles_deg(a), filter=G.FILTER_HANN, max_pairs=1) as plan:
        for g, ring in ((0, None), (2, False), (ring_group, True)):
            plan.set_tuning(cols_group=g, cols_ring=ring)
            o = torch.full((S, plan.M0, max(plan.M0, n)), float("nan"), device="cuda")
            plan.reconstruct_batch(sinos, o)
            torch.cuda.synchronize()
            plan.device_status()
            outs.append(o.cpu().numpy()[:, :, :plan.M0])
    np.testing.assert_array_equal(outs[0], outs[1])
    np.testing.assert_array_equal(outs[2], outs[1])


@pytest.mark.parametrize("n,a,S", [(8, 5, 9), (512, 37, 40), (1024, 97, 12), (2048, 61, 50), (4096, 35, 24),
                                   (1021, 50, 3)])
def test_ring_slice_bits_do_not_depend_on_the_stack(n, a, S):
    """A slice alone, in a pair and in the whole stack (blocks of 4 rows up to many) gives the
    same bits, with a row of mean 0 that is not all zero in one slice."""
    rng = np.random.default_rng(n + S)
    x = rng.uniform(0.0, 2.0, (S, a, n)).astype(np.float32)
    x[rng.uniform(size=x.shape) < 0.04] = 0.0
    x[1, 1, ::2], x[1, 1, 1::2] = 0.5, -0.5 if n % 2 == 0 else 0.0
    whole = G.ring_removal(_dev(x), 1.0, 4).cpu().numpy()
    for s in (0, 1, S - 2, S - 1):
        np.testing.assert_array_equal(G.ring_removal(_dev(x[s:s + 1]), 1.0, 4).cpu().numpy()[0], whole[s])
    np.testing.assert_array_equal(G.ring_removal(_dev(x[:2]), 1.0, 4).cpu().numpy(), whole[:2])


@pytest.mark.parametrize("n", [12, 516, 1020, 2044, 4092])
def test_ring_quotients_correctly_rounded(n):
    """Rounds without column correction (coefficient 0) on rows of two samples, whose sum has
    one rounding in any order: every value is RN(RN(x g) / r), bit for bit, whether the row
    divides by its reciprocal or not (means beyond 2^40, products below 2^-60)."""
    rng = np.random.default_rng(n)
    S, a = 2, 700
    x = np.zeros((S, a, n), np.float32)
    for s in range(S):
        for i in range(a):
            j = rng.choice(n, 2, replace=False)
            x[s, i, j] = (2.0 ** rng.uniform(-20, 20, 2)).astype(np.float32)
            if i % 50 == 0:
                x[s, i, j[0]] = np.float32(2.0 ** rng.uniform(-100, -55))
            if s == 1 and i % 50 == 1:
                x[s, i, j] = (2.0 ** rng.uniform(52, 60, 2)).astype(np.float32)
    got = G.ring_removal(_dev(x), 0.0, 3).cpu().numpy()
    for _ in range(3):
        r = np.float32(x.sum(axis=2, dtype=np.float64)) / np.float32(n)
        g = np.float32(r.astype(np.float64).mean(axis=1))
        x = (x * g[:, None, None]) / r[:, :, None]
    assert x.dtype == np.float32
    np.testing.assert_array_equal(got, x)


def test_plan_holds_spectra_for_its_own_groups():
    """A plan's spectra hold the group that its largest chunk grids as (1, 2, 4, 4, 8, 8 pairs
    for plans of 1 to 6), no more and no less: its bytes against those of a plan of the same
    pairs without groups, whose spectra hold exactly its pairs."""
    n, a = 256, 30
    th = ph.angles_deg(a)
    pair = a * 2 * 128 * 8  # one pair's spectra: two half lines of 128 complex values per angle
    records = set()
    for pairs, group in ((1, 1), (2, 2), (3, 4), (4, 4), (5, 8), (6, 8)):
        size = {}
        for mode in (0, -1):
            with G.Plan(n, a, th, max_pairs=pairs, wide_grid=mode) as plan:
                size[mode] = plan.device_bytes()
        # (the list's scratch: 32 complex cells of a group)
        records.add(size[0] - size[-1] - (group - pairs) * pair - group * 32 * 8)
    assert len(records) == 1, records


@pytest.mark.parametrize("pairs,chunk", [(3, 3), (6, 6), (12, 8)])
def test_plan_where_the_group_records_do_not_fit(pairs, chunk):
    """On a GPU with room for a plan's buffers but not for its optional group records, the plan
    is made without them and gives the same bits; records that come with a later change of the
    tuning, when there is room, grid the same chunks by groups within the plan's buffers."""
    n, a = 512, 2000
    th = ph.angles_deg(a)
    S = 2 * chunk - 1
    rng = np.random.default_rng(pairs)
    sinos = _dev(rng.uniform(0.0, 2.0, (S, a, n)).astype(np.float32))

    def images(plan):
        o = torch.full((S, plan.M0, n), float("nan"), device="cuda")
        plan.reconstruct_batch(sinos, o)
        torch.cuda.synchronize()
        plan.device_status()
        return o.cpu().numpy()[:, :, :plan.M0]

    def make():
        return G.Plan(n, a, th, filter=G.FILTER_HANN, max_pairs=pairs)

    with make() as plan:
        want, whole = images(plan), plan.device_bytes()
        cap = plan.set_tuning("tiles" if pairs < 7 else "wide", 600)["item_cap"]
        tuned = images(plan)
    with G.Plan(n, a, th, filter=G.FILTER_HANN, max_pairs=pairs, wide_grid=-1) as plan:
        bare = plan.device_bytes()
    torch.cuda.empty_cache()
    list_bytes = 30 << 20  # well under one list of records (32 bytes each, more than 2 a sample)
    assert whole - bare > list_bytes and 2 * n * a * 32 > list_bytes
    # room for everything but the last list of records, less half of that
    room = whole - list_bytes // 2
    filler = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    try:
        plan = make()
        short = plan.device_bytes()
    finally:
        del filler
        torch.cuda.empty_cache()
    with plan:
        assert short < whole - list_bytes, (short, whole)
        np.testing.assert_array_equal(images(plan), want)
        assert plan.set_tuning("tiles" if pairs < 7 else "wide", 600)["item_cap"] == cap
        np.testing.assert_array_equal(images(plan), tuned)


@pytest.mark.parametrize("S", [2, 3, 8])
def test_more_angles_than_a_grid_has_rows(S):
    """Chunks of 1 to 4 pairs of 65,600 angles: the tile kernel, whose spectra take the angle as
    the grid's x, as with wide_grid = -1."""
    n, a = 16, 65600
    th = ph.angles_deg(a)
    sinos = _dev(np.random.default_rng(S).uniform(0.0, 2.0, (S, a, n)).astype(np.float32))
    outs = []
    for mode in (0, -1):
        with G.Plan(n, a, th, filter=G.FILTER_HANN, max_pairs=4, wide_grid=mode) as plan:
            o = torch.full((S, plan.M0, n), float("nan"), device="cuda")
            plan.reconstruct_batch(sinos, o)
            torch.cuda.synchronize()
            plan.device_status()
            outs.append(o.cpu().numpy()[:, :, :plan.M0])
    np.testing.assert_array_equal(outs[0], outs[1])


def test_center_search_leaves_the_sinograms_to_the_caller():
    """The images of the best shift are those of the sinograms as they were passed, also where
    the caller overwrites them on another stream as soon as the call has returned."""
    n, a = 1000, 2400
    rng = np.random.default_rng(4)
    x = rng.uniform(0.0, 2.0, (2, a, n)).astype(np.float32)
    shifts = np.float32([-0.5, 0.5])
    side = torch.cuda.Stream()
    with G.Plan(2 * n, a, ph.angles_deg(a), filter=G.FILTER_HANN) as plan:
        s = _dev(x)
        scores, best, want = G.center_search(plan, s[0], s[1], shifts, -1.0, 3.0, 500, want_images=True)
        torch.cuda.synchronize()
        other = torch.full_like(s, 7.0)
        for _ in range(3):
            s.copy_(torch.from_numpy(x))
            torch.cuda.synchronize()
            with torch.cuda.stream(side):
                again = G.center_search(plan, s[0], s[1], shifts, -1.0, 3.0, 500, want_images=True, stream=side)
            s.copy_(other)  # on the current stream, not ordered after `side`
            torch.cuda.synchronize()
            assert again[1] == best
            np.testing.assert_array_equal(again[0], scores)
            assert torch.equal(again[2], want)


def test_fbp_too_many_angles_refused_and_nothing_left_behind():
    """More angles than the shared-memory table holds: refused as unsupported before anything
    runs, and the next call is not told of it; more than the default table limit: run."""
    n = 16
    x = _dev(np.random.default_rng(0).uniform(0.0, 2.0, (1, 30000, n)).astype(np.float32))
    many = G.FBP(n, 30000, ph.angles_deg(30000), max_slices=1)
    some = G.FBP(n, 7000, ph.angles_deg(7000), max_slices=1)
    for _ in range(2):
        with pytest.raises(G.GrError, match="UNSUPPORTED"):
            many.reconstruct(x)
        got = some.reconstruct(x[:, :7000].contiguous()).cpu().numpy()[0]
        assert ph.rel_l2(got, O.port_optimized_fbp(x[0, :7000].cpu().numpy(), ph.angles_deg(7000))) < 1e-5
    many.close()
    some.close()


@pytest.mark.parametrize("n,pairs,group,ring", [(2048, 1, 4, False), (2048, 2, 4, False), (2048, 3, 8, True),
                                                (1024, 4, 8, False), (4096, 1, 4, True), (8192, 1, 2, False)])
def test_column_form_reported_and_pinned(n, pairs, group, ring):
    """The tuning names the column FFT that a full chunk runs by default (persistent from
    four strips per SM at M = 2048 and 4096), and keeps what is pinned, also a persistent
    form without a width for a chunk of few strips: the same bits."""
    a = 3
    S = 2 * pairs
    sinos = _dev(np.random.default_rng(n).uniform(0.0, 2.0, (S, a, n)).astype(np.float32))
    with G.Plan(n, a, ph.angles_deg(a), filter=G.FILTER_HANN, max_pairs=pairs) as plan:
        def images():
            o = torch.full((S, plan.M0, max(plan.M0, n)), float("nan"), device="cuda")
            plan.reconstruct_batch(sinos, o)
            torch.cuda.synchronize()
            plan.device_status()
            return o[:, :, :plan.M0]

        t = plan.tuning()
        assert (t["cols_group"], t["cols_ring"]) == (group, ring)
        want = images()
        t = plan.set_tuning(cols_ring=True)
        assert (t["cols_group"], t["cols_ring"]) == (min(8, 16384 // n), True)
        assert torch.equal(images(), want)
        t = plan.set_tuning(cols_ring=False)
        assert (t["cols_group"], t["cols_ring"]) == (2 if n == 8192 else min(8, 8192 // n), False)
        assert torch.equal(images(), want)


def test_network_refuses_an_empty_minibatch():
    from projects_b200 import learned as L
    net = L.CorrectionNet(L.init_params(1))
    for shape in ((0, 8, 8), (2, 0, 8), (2, 8, 0)):
        x = torch.empty(shape, device="cuda")
        with pytest.raises(G.GrError, match="GR_ERR_ARG"):
            net.loss_and_grads(x, x)


@pytest.mark.parametrize("shape", [(223, 200, 60), (1, 900, 130), (2, 33, 64), (3, 65, 17)])
@pytest.mark.parametrize("signs", ["one", "mixed"])
def test_network_weight_gradients_exact_contraction(shape, signs):
    """The weight gradients against the float64 contraction of the activations and gradients
    that the backward pass itself stored (BF16, FP32 for x and the output's gradient), in units
    of the sum of the terms' magnitudes.  One image's whole height per block, several segments, all
    terms of one sign (where errors of one sign add up) and of both.  Bound 3e-7: the result's
    own rounding (2^-24), what an MMA of 16 pixels cuts off (2^-23) and 128 rounded FP32 additions
    on a growing sum (0.6 sqrt(128 / 3) 2^-25 = 1.2e-7)."""
    from projects_b200 import learned as L
    n, h, w = shape
    rng = np.random.default_rng(h)
    p = rng.normal(0, 0.2, 2625).astype(np.float32)
    x = rng.uniform(0.5, 1.5, shape).astype(np.float32)
    if signs == "one":
        p = np.abs(p)
        target = np.zeros_like(x)
    else:
        x -= 1.0
        target = (x + rng.normal(0, 0.3, shape)).astype(np.float32)
    net = L.CorrectionNet(p)
    x = _dev(x)
    net.loss_and_grads(x, _dev(target))
    px = n * h * w  # the workspace: h1, h2, gz1, gz2 (BF16 x 16), the output's gradient
    h1, h2, g1, g2 = (net._ws[k * px * 32:(k + 1) * px * 32].view(torch.bfloat16).view(n, h, w, 16).double()
                      for k in range(4))
    gy = net._ws[4 * px * 32:4 * px * 32 + 4 * px].view(torch.float32).view(n, h, w).double()

    def grads(x, h1, h2, g1, g2, gy):
        out = torch.zeros(2625, dtype=torch.float64, device="cuda")
        pad = torch.nn.functional.pad
        X, H, Y = pad(x, (1, 1, 1, 1)), pad(h1, (0, 0, 1, 1, 1, 1)), pad(gy, (1, 1, 1, 1))
        f1, f2, fh = g1.reshape(-1, 16), g2.reshape(-1, 16), h2.reshape(-1, 16)
        for tap in range(9):
            r, c = tap // 3, tap % 3
            out[tap * 16:tap * 16 + 16] = f1.T @ X[:, r:r + h, c:c + w].reshape(-1)
            out[160 + tap * 256:416 + tap * 256] = (f2.T @ H[:, r:r + h, c:c + w].reshape(-1, 16)).reshape(-1)
            out[2480 + tap * 16:2496 + tap * 16] = fh.T @ Y[:, 2 - r:2 - r + h, 2 - c:2 - c + w].reshape(-1)
        out[144:160], out[2464:2480], out[2624] = f1.sum(0), f2.sum(0), gy.sum()
        return out

    args = (x.double(), h1, h2, g1, g2, gy)
    want, size = grads(*args), grads(*(t.abs() for t in args))
    err = ((net.grads.double() - want).abs() / size.clamp_min(1e-300)).max()
    assert float(err) < 3e-7
