"""The occupied-orbital build on the INT8 tensor cores (rijk_i8.cu) against the
oracle's formulas, at the edges of its tiles: 128-row and 64-column blocks of K,
16-column digit groups, 32-column steps of k, the tensor's digits made in the tile
(up to two blocks of 64 orbitals) or through memory."""
import numpy as np
import pytest

from rest_b200.synth import host_case

pytestmark = pytest.mark.gpu


def _full(packed, n):
    out = np.zeros((packed.shape[1], n, n))
    jj, ii = np.tril_indices(n)
    out[:, ii, jj] = packed.T
    out[:, jj, ii] = packed.T
    return out


def _k(ctx, n, c, occ, spin=1):
    vk = ctx.vk_upper_with_ri_v(c, [x.shape[1] - 1 for x in c], occ, spin, 1.0)
    jj, ii = np.tril_indices(n)
    out = []
    for s in range(spin):
        m = np.zeros((n, n))
        m[ii, jj] = vk[s]
        m[jj, ii] = vk[s]
        out.append(m)
    return out


def _ctx(rimatr, n):
    from rest_b200 import RIJK

    ctx = RIJK(0)
    ctx.set_rimatr(rimatr, n)
    return ctx


@pytest.mark.parametrize("n,naux,o", [(64, 31, 5), (65, 40, 1), (96, 33, 16), (127, 30, 17), (129, 21, 64),
                                      (201, 50, 15), (256, 64, 33), (257, 37, 65), (300, 29, 128), (310, 9, 129),
                                      (385, 20, 180)])
def test_k_within_the_operands_rounding(n, naux, o):
    case = host_case(n, naux, o, seed=n)
    occ = np.linspace(0.5, 2.0, o)
    x = np.einsum("pmn,ni->mpi", _full(case.rimatr, n), case.c_occ * np.sqrt(occ)).reshape(n, -1)
    with _ctx(case.rimatr, n) as ctx:
        k = _k(ctx, n, [case.c_occ], [occ])[0]
    # an element of X is a sum of n products of 55-bit operands (2^-55 of the row's
    # and column's maxima each), and its digits are off by 2^-55 of the row's maximum;
    # a K element sums naux o products of two of them, and so does the reference
    m = np.abs(x).max(axis=1)
    bscale = np.abs(_full(case.rimatr, n)).max(axis=(0, 2)) * np.abs(case.c_occ).max() * np.sqrt(2.0)
    tol = 2 * naux * o * (np.outer(m, m) * 2.0**-53 + n * 2.0**-53 * np.outer(m, bscale)) + 1e-300
    assert np.all(np.abs(k - x @ x.T) <= np.maximum(tol, tol.T))


@pytest.mark.parametrize("n,naux,o,spin", [(70, 60, 9, 1), (140, 90, 150, 1), (161, 75, 70, 2), (300, 60, 20, 2)])
def test_j_and_k_in_chunks(n, naux, o, spin, monkeypatch):
    """J's scalars and K over several chunks of X and sub-chunks of tensor digits
    give what one chunk gives, to FP64 rounding."""
    case = host_case(n, naux, min(o, n), seed=n + o)
    rng = np.random.default_rng(o)
    cs = [case.c_occ] + [np.asfortranarray(np.linalg.qr(rng.standard_normal((n, min(o, n))))[0])][:spin - 1]
    occ = [np.linspace(0.1, 1.0, c.shape[1]) for c in cs]
    homo = [c.shape[1] - 1 for c in cs]
    got = []
    for budget in (None, 12 << 20):
        if budget:
            monkeypatch.setenv("RIJK_SCRATCH_BYTES", str(budget))
        with _ctx(case.rimatr, n) as ctx:
            vj, vk = ctx.vjk_upper_with_ri_v(cs, homo, occ, spin, 1.0, 1.0)
            dms = [np.asfortranarray((c * w) @ c.T) for c, w in zip(cs, occ)]
            ref = ctx.vj_upper_with_rimatr_v(dms, spin, 1.0)  # J by two FP64 passes
        for s in range(spin):
            assert np.abs(vj[s] - ref[s]).max() <= 1e-13 * np.abs(ref[s]).max() * np.sqrt(n)
        got.append((vj, vk))
    for s in range(spin):
        assert np.abs(got[0][0][s] - got[1][0][s]).max() <= 1e-13 * np.abs(got[0][0][s]).max()
        assert np.abs(got[0][1][s] - got[1][1][s]).max() <= 1e-13 * np.abs(got[0][1][s]).max()


@pytest.mark.parametrize("n,naux,o", [(64, 5, 3), (263, 7, 31), (320, 3, 200)])
def test_integers_are_exact(n, naux, o):
    rng = np.random.default_rng(n)
    r = np.asfortranarray(rng.integers(-9, 10, (n * (n + 1) // 2, naux)).astype(float))
    c = np.asfortranarray(rng.integers(-3, 4, (n, o)).astype(float))
    x = np.einsum("pmn,ni->mpi", _full(r, n), c).reshape(n, -1)
    with _ctx(r, n) as ctx:
        k = _k(ctx, n, [c], [np.ones(o)])[0]
    assert np.array_equal(k, x @ x.T)


def test_two_spins_and_scaled_rows():
    """Rows many orders of magnitude apart: each is held relative to its own maximum."""
    n, naux, o = 230, 40, 21
    case = host_case(n, naux, o, seed=3)
    rng = np.random.default_rng(4)
    d = 2.0 ** rng.integers(-120, 120, n)
    jj, ii = np.tril_indices(n)
    r = np.asfortranarray(case.rimatr * (d[ii] * d[jj])[:, None])
    cs = [np.asfortranarray(rng.standard_normal((n, o))) for _ in range(2)]
    with _ctx(r, n) as ctx:
        ks = _k(ctx, n, cs, [np.ones(o), np.ones(o)], spin=2)
    b = _full(case.rimatr, n) * d
    for c, k in zip(cs, ks):
        x = np.einsum("pmn,ni->mpi", b, c).reshape(n, -1)
        ref = x @ x.T
        # 55 bits below the row maxima, sums of naux o products of sums of n
        assert np.abs(k / np.outer(d, d) - ref).max() <= naux * o * n * 2.0**-53 * np.abs(x).max() ** 2


def test_zero_and_nonfinite_tensor_rows():
    n, naux, o = 210, 12, 9
    case = host_case(n, naux, o, seed=8)
    full = _full(case.rimatr, n)
    full[:, 7, :] = full[:, :, 7] = 0.0  # a basis function without any element
    full[3, 11, 20] = full[3, 20, 11] = np.nan
    jj, ii = np.tril_indices(n)
    r = np.asfortranarray(full[:, ii, jj].T)
    with _ctx(r, n) as ctx:
        k = _k(ctx, n, [case.c_occ], [np.ones(o)])[0]
    bad = np.zeros((n, n), bool)
    bad[[11, 20], :] = bad[:, [11, 20]] = True
    assert np.isnan(k[bad]).all() and np.isfinite(k[~bad]).all()
    keep = [i for i in range(n) if i not in (7, 11, 20)]
    assert not k[7, keep].any()


@pytest.mark.parametrize("n,naux", [(128, 40), (129, 33), (160, 21), (257, 9)])
def test_density_form(n, naux):
    """K from a density: packed for two symmetric ones, full for one that is not;
    digits in the tile (n = 128) and through memory."""
    case = host_case(n, naux, n // 5, seed=n)
    b = _full(case.rimatr, n)
    rng = np.random.default_rng(n)
    sym = [case.dm, np.asfortranarray(case.dm @ case.dm + np.eye(n))]
    d = np.asfortranarray(rng.standard_normal((n, n)))
    jj, ii = np.tril_indices(n)
    with _ctx(case.rimatr, n) as ctx:
        up = ctx.vk_upper_with_ri_v_use_dm_only(sym, 2, 1.0)
        full = ctx.vk_full_fromdm_with_ri_v([d], 1, 1.0)[0]
    for got, dm in [(up[0], sym[0]), (up[1], sym[1]), (full, d)]:
        t = b @ dm
        ref = np.einsum("pmk,pkn->mn", t, b)
        # T off by n 2^-53 of its operands' maxima, T's and B's digits by 2^-55 of the
        # rows' maxima, over naux n products, twice (the reference's own rounding)
        tol = 2 * naux * n * 2.0**-53 * (np.abs(t).max() + n * np.abs(b).max() * np.abs(dm).max()) * np.abs(b).max()
        assert np.abs(got - (ref[ii, jj] if got.ndim == 1 else ref)).max() <= tol


def test_density_form_in_chunks(monkeypatch):
    n, naux = 140, 70
    case = host_case(n, naux, 20, seed=1)
    got = []
    for budget in (None, 24 << 20):
        if budget:
            monkeypatch.setenv("RIJK_SCRATCH_BYTES", str(budget))
        with _ctx(case.rimatr, n) as ctx:
            got.append(ctx.vk_upper_with_rimatr_use_dm_only([case.dm], 1, 1.0)[0])
    assert np.abs(got[0] - got[1]).max() <= 1e-13 * np.abs(got[0]).max()


def test_group_of_both_forms():
    """A group whose larger molecules take the INT8 form and the others DMMA: each
    equals its own build, and a molecule that is switched off is left alone."""
    import torch

    from rest_b200 import RIJKGroup

    shapes = [(24, 60, 5), (120, 40, 25), (96, 70, 20), (187, 33, 64), (200, 17, 80), (130, 90, 129)]
    nm = max(n for n, _, _ in shapes)
    ctxs, cs, ref = [], [], []
    for i, (n, naux, o) in enumerate(shapes):
        case = host_case(n, naux, o, seed=20 + i)
        ctxs.append(_ctx(case.rimatr, n))
        cs.append(case.c_occ)
        vj, vk = ctxs[-1].vjk_upper_with_ri_v([case.c_occ], [o - 1], [np.full(o, 2.0)], 1, 1.0, -0.5)
        jj, ii = np.tril_indices(n)
        m = np.zeros((n, n))
        m[ii, jj] = m[jj, ii] = vj[0] + vk[0]
        ref.append(m)
    C = torch.zeros(len(shapes), nm, nm, dtype=torch.float64, device="cuda")
    for i, c in enumerate(cs):
        C[i, :c.shape[0], :c.shape[1]] = torch.as_tensor(c, device="cuda")
    out = torch.full_like(C, 7.0)
    g = RIJKGroup(ctxs, [o for _, _, o in shapes])
    for off in (None, 1, 4, 5):
        active = torch.tensor([0 if i == off else 1 for i in range(len(shapes))], dtype=torch.int32, device="cuda")
        out.fill_(7.0)
        torch.cuda.synchronize()
        g.jk_occ_dev(C.data_ptr(), nm * nm, nm, 1, -0.5, active.data_ptr(), out.data_ptr(), nm * nm, nm)
        g.synchronize()
        got = out.cpu().numpy()
        for i, (n, _, _) in enumerate(shapes):
            if i == off:
                assert (got[i] == 7.0).all()
            else:  # both sum naux o products and naux rows in FP64, in other orders
                assert np.abs(got[i, :n, :n] - ref[i]).max() <= 1e-12 * np.abs(ref[i]).max()
    g.close()
    for c in ctxs:
        c.close()


@pytest.mark.parametrize("n,naux,o", [(130, 37, 21), (260, 21, 140)])
def test_captured_build_follows_the_tensor(n, naux, o):
    """A build captured on a pinned context and replayed after other rows were loaded
    into the tensor: some a thousand times larger than the ones it was captured with,
    some zero before."""
    import torch

    old, new = host_case(n, naux, o, seed=1), host_case(n, naux, o, seed=2)
    r0 = old.rimatr.copy(order="F")
    r0[:, naux // 2:] = 0.0
    r1 = np.asfortranarray(1000.0 * new.rimatr)
    c = torch.as_tensor(old.c_occ.T.copy(), device="cuda")
    occ = torch.full((o,), 2.0, dtype=torch.float64, device="cuda")
    dm = 2.0 * c.T @ c
    rows = torch.as_tensor(r1.T.copy(), device="cuda")
    npair = n * (n + 1) // 2

    def build(ctx, out):
        st = torch.cuda.current_stream().cuda_stream
        ctx.vjk_upper_occ_dev(c.data_ptr(), o, [o - 1], occ.data_ptr(), 1, 1.0, 1.0, out[0].data_ptr(),
                              out[1].data_ptr(), st)
        ctx.vk_upper_dm_dev(dm.data_ptr(), 1, 1.0, out[2].data_ptr(), st)

    want, got = (torch.zeros(3, npair, dtype=torch.float64, device="cuda") for _ in range(2))
    with _ctx(r1, n) as fresh:
        build(fresh, want)
        fresh.synchronize(torch.cuda.current_stream().cuda_stream)
    with _ctx(r0, n) as ctx:
        build(ctx, got)
        torch.cuda.synchronize()
        ctx.pin_buffers(True)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            build(ctx, got)
        st = torch.cuda.current_stream().cuda_stream
        ctx.tensor_load_rows_dev(rows.data_ptr(), 0, naux, 0, st)
        graph.replay()
        ctx.synchronize(st)
        # the same kernels on the same operands, their K partials and J shares added in one order
        assert torch.equal(got, want)
        del graph
        ctx.pin_buffers(False)


def test_every_producer_of_the_tensor():
    """Each way a tensor gets into a context, after one of much smaller elements, gives
    the same K: what the INT8 form keeps of the rows is the new tensor's."""
    import torch

    n, naux, o = 72, 40, 9
    case = host_case(n, naux, o, seed=6)
    full = np.asfortranarray(_full(case.rimatr, n).transpose(1, 2, 0))
    rows = torch.as_tensor(np.ascontiguousarray(case.rimatr.T), device="cuda")
    blocks = torch.as_tensor(np.ascontiguousarray(full.transpose(2, 1, 0)), device="cuda")
    torch.cuda.synchronize()
    eye = np.eye(naux, order="F")

    def by_rows(ctx):
        ctx.tensor_alloc(n, naux)
        ctx.tensor_load_rows_dev(rows.data_ptr(), 0, 17, 0)
        ctx.tensor_load_rows_dev(blocks[17:].data_ptr(), 17, naux - 17, 1)

    producers = [lambda ctx: ctx.set_rimatr(case.rimatr, n), lambda ctx: ctx.set_ri3fn(full), by_rows,
                 lambda ctx: ctx.fit_rimatr(eye, case.rimatr, n),
                 lambda ctx: ctx.build_rimatr_cholesky(eye, case.rimatr, n)]
    got = []
    for produce in producers:
        with _ctx(np.asfortranarray(1e-6 * case.rimatr), n) as ctx:
            produce(ctx)
            got.append(_k(ctx, n, [case.c_occ], [np.ones(o)])[0])
    for k in got[1:]:
        assert np.array_equal(k, got[0])

    from rest_b200.geometry import water_cluster

    mol = water_cluster(3, seed=1)
    bas, aux = mol.shells("def2-SVP"), mol.shells("def2-SVP-JKFIT")
    with _ctx(np.asfortranarray(1e-6 * case.rimatr), n) as ctx:
        ctx.build_rimatr_from_shells(bas, aux)
        k = _k(ctx, n, [case.c_occ], [np.ones(o)])[0]
        r = ctx.get_rimatr()
    with _ctx(r, n) as ctx:
        assert np.array_equal(k, _k(ctx, n, [case.c_occ], [np.ones(o)])[0])


def test_group_created_behind_loads_in_flight():
    """Rows are loaded, a group made of their context and a build enqueued, all on one
    non-blocking stream that is still busy: stream order alone has to be enough."""
    import torch

    from rest_b200 import RIJK, RIJKGroup

    n, naux, o = 150, 60, 20
    case = host_case(n, naux, o, seed=9)
    with _ctx(case.rimatr, n) as ctx:
        vj, vk = ctx.vjk_upper_with_ri_v([case.c_occ], [o - 1], [np.full(o, 2.0)], 1, 1.0, -0.5)
    rows = torch.as_tensor(np.ascontiguousarray(case.rimatr.T), device="cuda")
    C = torch.as_tensor(np.ascontiguousarray(case.c_occ), device="cuda")
    active = torch.ones(1, dtype=torch.int32, device="cuda")
    out = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    busy = torch.randn(4096, 4096, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    with RIJK(0) as ctx:
        ctx.tensor_alloc(n, naux)
        with torch.cuda.stream(st):
            x = busy
            for _ in range(40):  # some tens of milliseconds
                x = (x @ busy) * 1e-2
        ctx.tensor_load_rows_dev(rows.data_ptr(), 0, naux, 0, st.cuda_stream)
        g = RIJKGroup([ctx], [o])
        g.jk_occ_dev(C.data_ptr(), n * o, o, 1, -0.5, active.data_ptr(), out.data_ptr(), n * n, n, st.cuda_stream)
        g.synchronize(st.cuda_stream)
        g.close()
    jj, ii = np.tril_indices(n)
    ref = vj[0] + vk[0]
    # both sum naux o products and naux rows in FP64, in other orders
    assert np.abs(out.cpu().numpy()[ii, jj] - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("n", [16384, 27000])
def test_largest_sums_of_the_half_transform(n):
    """Every digit of both operands at the end of its range, over the most functions the
    INT8 form takes and over more than 32-bit sums of such products hold (18808 for
    digits 0 and 6 together with 1 and 5, 2 and 4, 3 and 3; what overflows at 27000 is
    of weight 2^-29 of the sum, far above the tolerance)."""
    import torch

    from rest_b200 import RIJK

    b = -(126 * 256**6 + 128 * (256**6 - 1) // 255) / 2.0**55
    npair = n * (n + 1) // 2
    rows = torch.full((npair,), b, dtype=torch.float64, device="cuda")
    c = torch.full((n,), b, dtype=torch.float64, device="cuda")
    occ = torch.ones(1, dtype=torch.float64, device="cuda")
    vj, vk = (torch.empty(npair, dtype=torch.float64, device="cuda") for _ in range(2))
    st = torch.cuda.current_stream().cuda_stream
    with RIJK(0) as ctx:
        ctx.tensor_alloc(n, 1)
        ctx.tensor_load_rows_dev(rows.data_ptr(), 0, 1, 0, st)
        ctx.vjk_upper_occ_dev(c.data_ptr(), 1, [0], occ.data_ptr(), 1, 1.0, 1.0, vj.data_ptr(), vk.data_ptr(), st)
        ctx.synchronize(st)
    for out, ref in ((vk, (n * b * b) ** 2), (vj, n * n * b**4)):  # X = n b c; w = sum of n x c, J = w B
        # sums of n equal terms, then products: n + 3 roundings
        assert float((out - ref).abs().max()) <= (n + 3) * 2.0**-53 * abs(ref)


def test_threads_of_different_sizes():
    """Contexts of several host threads load rows at once: what one of them sets up
    for its kernels does not depend on another's size."""
    import threading

    import torch

    from rest_b200 import RIJK

    errors = []
    sizes = (64, 1200, 130, 1000)
    rows = torch.zeros(1200 * 1201 // 2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ready = threading.Barrier(len(sizes))

    def work(n):
        try:
            with RIJK(0) as ctx:
                ctx.tensor_alloc(n, 1)
                ready.wait()
                for _ in range(3000):
                    ctx.tensor_load_rows_dev(rows.data_ptr(), 0, 1, 0, 0)
                ctx.synchronize()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            errors.append((n, repr(e)))

    threads = [threading.Thread(target=work, args=(n,)) for n in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors


@pytest.mark.parametrize("up", [980, -980])
def test_operands_at_the_ends_of_the_range(up):
    """Tensor and orbitals scaled against each other: X is the unscaled problem's."""
    n, naux, o = 140, 9, 11
    case = host_case(n, naux, o, seed=5)
    x = np.einsum("pmn,ni->mpi", _full(case.rimatr, n), case.c_occ).reshape(n, -1)
    r = np.asfortranarray(np.ldexp(case.rimatr, up))
    c = np.asfortranarray(np.ldexp(case.c_occ, -up))
    with _ctx(r, n) as ctx:
        k = _k(ctx, n, [c], [np.ones(o)])[0]
    # as test_k_within_the_operands_rounding
    m = np.abs(x).max(axis=1)
    bscale = np.abs(case.rimatr).max() * np.abs(case.c_occ).max()
    assert np.abs(k - x @ x.T).max() <= 2 * naux * o * (m.max() ** 2 + n * m.max() * bscale) * 2.0**-53


def _local_case(n, naux, seed):
    """A tensor whose elements fall off with the functions' distance, to 1e-50."""
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0, 20, (n, 3))
    env = np.exp(-0.1 * ((pos[:, None] - pos[None]) ** 2).sum(-1))
    s = np.exp(np.log(1e-3) * rng.uniform(size=naux))
    jj, ii = np.tril_indices(n)
    return np.asfortranarray((rng.standard_normal((naux, ii.size)) * s[:, None] * env[ii, jj]).T), rng


def test_exchange_form_is_the_callers_choice():
    """Orbitals on one function each, so that many elements of K have only terms far
    below the rows' largest: DMMA's error is relative to those terms, the INT8 form's to
    the rows' maxima."""
    import torch

    from rest_b200 import RIJKGroup

    n, naux, o = 200, 60, 33
    r, rng = _local_case(n, naux, 0)
    b = _full(r, n)
    c = np.zeros((n, o), order="F")
    c[rng.choice(n, o, replace=False), np.arange(o)] = 1.0
    d = np.asfortranarray(np.diag(rng.uniform(0.5, 1.0, n)))
    x = np.einsum("pmn,ni->mpi", b, c).reshape(n, -1)
    t = (b @ d).transpose(1, 0, 2).reshape(n, -1)
    y = b.transpose(1, 0, 2).reshape(n, -1)
    jj, ii = np.tril_indices(n)
    with _ctx(r, n) as ctx:
        with pytest.raises(ValueError):
            ctx.set_exchange("fp32")
        for form in ("int8", "dmma"):
            ctx.set_exchange(form)
            k = _k(ctx, n, [c], [np.ones(o)])[0]
            kd = ctx.vk_full_fromdm_with_ri_v([d], 1, 1.0)[0]
            # X is exact (one term an element), K sums naux o products, twice (the
            # reference's own rounding); T one product, K naux n
            for got, p, q, terms in ((k, x, x, naux * o), (kd, t, y, naux * n)):
                err = np.abs(got - p @ q.T)
                own = 2 * (terms + 1) * 2.0**-53 * (np.abs(p) @ np.abs(q).T)
                if form == "dmma":
                    assert np.all(err <= own)
                else:
                    # digits: 2^-54 of the rows' maxima for B, X (or T) and B each,
                    # through naux o (naux n) products
                    top = np.abs(y).max(axis=1)
                    assert np.all(err <= own + 8 * terms * 2.0**-53 * np.outer(top, top))
                    assert np.any(err > 1e3 * own)  # what the other form is there for
        # a group takes each member's choice at creation
        C = torch.as_tensor(np.ascontiguousarray(c), device="cuda")
        active = torch.ones(1, dtype=torch.int32, device="cuda")
        out = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        vj = ctx.vj_upper_with_rimatr_v([np.asfortranarray(2.0 * c @ c.T)], 1, 1.0)[0]
        g = RIJKGroup([ctx], [o])
        ctx.set_exchange("int8")
        g.jk_occ_dev(C.data_ptr(), n * o, o, 1, 1.0, active.data_ptr(), out.data_ptr(), n * n, n)
        g.synchronize()
        g.close()
        ref = 2 * x @ x.T
        jf = np.zeros((n, n))
        jf[ii, jj] = jf[jj, ii] = vj
        own = (np.abs(ref) + np.abs(jf)) + 2 * np.abs(x) @ np.abs(x).T
        # J's terms: naux scalars of o n products each, times the tensor's elements
        w = 2 * np.einsum("pmn,mi,ni->p", np.abs(b), np.abs(c), np.abs(c))
        own = own + np.einsum("p,pmn->mn", w, np.abs(b))
        assert np.all(np.abs(out.cpu().numpy() - ref - jf) <= 2 * naux * n * 2.0**-53 * own)


def test_digits_of_the_update():
    """K_ij = o x_i x_j of operands with all seven digits in use, against whole numbers:
    the update from X (orbitals on one function each, so that X is the tensor's columns)
    and from T and the tensor's rows (the density form with D = 1)."""
    import i8_cases as I

    n, o = 170, 8
    pat = I.patterns(n - o, 3)
    v = [I.value(d) for d in pat]
    b = np.zeros((1, n, n))
    b[0, o:, :o] = np.array(v, dtype=float)[:, None]
    b[0, :o, o:] = b[0, o:, :o].T
    jj, ii = np.tril_indices(n)
    c = np.asfortranarray(np.eye(n)[:, :o])
    with _ctx(np.asfortranarray(b[:, ii, jj].T), n) as ctx:
        k = _k(ctx, n, [c], [np.ones(o)])[0]
        kd = ctx.vk_full_fromdm_with_ri_v([np.asfortranarray(np.eye(n))], 1, 1.0)[0]
    for got in (k, kd):  # all nonzero terms in one step of one split: a single rounding
        for i in range(n - o):
            for j in range(0, n - o, 7):
                assert I.relative_error(got[o + i, o + j], o * v[i] * v[j]) <= I.PRODUCT_TOL


@pytest.mark.parametrize("n,o", [(70, 1), (130, 17), (130, 130), (260, 200)])
def test_digits_of_the_half_transform(n, o):
    """X = n b c with all digits of b and c in use, seen through K = X X^T: digits made in
    the tile and through memory, in the first and the last column of the orbitals."""
    import i8_cases as I

    pat = I.patterns(4, n)
    jj, ii = np.tril_indices(n)
    for db in pat:
        b = I.value(db)
        with _ctx(np.full((ii.size, 1), float(b), order="F"), n) as ctx:
            for dc in pat[:3]:
                for col in {0, o - 1}:
                    c = np.zeros((n, o), order="F")
                    c[:, col] = float(I.value(dc))
                    k = _k(ctx, n, [c], [np.ones(o)])[0]
                    x = int(float(n * b * I.value(dc)))  # rounded to nearest, as the levels' sum is
                    # X one rounding off at most (the dropped levels turn a tie), twice in K
                    err = max(I.relative_error(k[i, j], x * x) for i in (0, 31, 32, n // 2, n - 1) for j in (0, n - 1))
                    assert err <= 2 * 2.0**-53 + I.PRODUCT_TOL


def _leave_free(nbytes):
    """Device memory held so that about ``nbytes`` stay free."""
    import torch
    from cuda.bindings import runtime

    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    # what the stream-ordered pool keeps would come back to an allocation that fails
    err, pool = runtime.cudaDeviceGetDefaultMemPool(torch.cuda.current_device())
    assert int(err) == 0 and int(runtime.cudaMemPoolTrimTo(pool, 0)[0]) == 0
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(free - nbytes, dtype=torch.uint8, device="cuda")


def test_builds_without_room_for_the_digits():
    """With room for the DMMA form's scratch only, a build and a group take that form
    (half-transformed orbitals or density 1.2, 0.5 and 2.6 GB; the digits' form 1.6, 1.3
    and 4.9)."""
    import torch

    from rest_b200 import RIJK, RIJKGroup

    for n, naux, o, free, kind in ((300, 2000, 200, 1400 << 20, "occ"), (300, 390, 200, 800 << 20, "dm"),
                                   (130, 20000, 64, 3500 << 20, "group")):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(n)
        rows = torch.randn(naux // 10, n * (n + 1) // 2, generator=gen, dtype=torch.float64, device="cuda")
        C = torch.linalg.qr(torch.randn(n, o, generator=gen, dtype=torch.float64, device="cuda"))[0].contiguous()
        c = C.T.contiguous()
        dm = C @ c
        occ = torch.full((o,), 2.0, dtype=torch.float64, device="cuda")
        vj, vk = (torch.empty(n * (n + 1) // 2, dtype=torch.float64, device="cuda") for _ in range(2))
        active = torch.ones(1, dtype=torch.int32, device="cuda")
        out = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        got = []
        for short in (False, True):
            with RIJK(0) as ctx:
                ctx.tensor_alloc(n, naux)
                for p in range(10):
                    ctx.tensor_load_rows_dev(rows.data_ptr(), p * (naux // 10), naux // 10, 0)
                ctx.synchronize()
                launches = RIJK.kernel_launches()
                hold = _leave_free(free) if short else None
                if kind == "group":
                    g = RIJKGroup([ctx], [o])
                    g.jk_occ_dev(C.data_ptr(), n * o, o, 1, -0.5, active.data_ptr(), out.data_ptr(), n * n, n)
                    g.synchronize()
                    g.close()
                    res = out.clone()
                elif kind == "dm":
                    ctx.vk_upper_dm_dev(dm.data_ptr(), 1, -0.5, vk.data_ptr())
                    ctx.synchronize()
                    res = vk.clone()
                else:
                    ctx.vjk_upper_occ_dev(c.data_ptr(), o, [o - 1], occ.data_ptr(), 1, 1.0, -0.5, vj.data_ptr(),
                                          vk.data_ptr())
                    ctx.synchronize()
                    res = torch.stack([vj, vk])
                del hold
                torch.cuda.empty_cache()
                got.append((res, RIJK.kernel_launches() - launches))
        assert got[0][1] != got[1][1]  # the other form's launches
        # both sum naux o products of sums of n, in other orders
        assert float((got[1][0] - got[0][0]).abs().max()) <= 1e-12 * float(got[0][0].abs().max())
