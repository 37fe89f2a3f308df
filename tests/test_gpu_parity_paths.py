"""GPU parity tests of the paths the benchmark measures: the slab-pipelined host
loader, the loader without the kept input-order CSR, several tail column blocks,
the workload configuration 1 at its stated size with the loss curve, full runs at
the wide ranks, the host twin of the synthetic generator, and the bounded waits of
the warp-specialised tensor-core kernel.  Everything goes through the C ABI."""
import numpy as np
import pytest

from oracle import oracle as O
from helpers import rel_fro, make_problem, oracle_preprocess, baseline_scale

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    assert torch.cuda.is_available()
    torch.cuda.set_device(0)
    return torch


def _engine(params, options=(), **kw):
    from npeff_ref_b200 import MuNmf
    eng = MuNmf(params, **kw)
    for name, value in options:
        eng.set_option(name, value)
    return eng


def _ragged(rng, n, m, lens):
    ptr = np.zeros(n + 1, dtype=np.int64)
    ptr[1:] = np.cumsum(lens)
    ind = np.concatenate([rng.choice(m, size=l, replace=False) for l in lens] +
                         [np.zeros(0, dtype=np.int64)]).astype(np.int32)
    vals = (rng.random(int(ptr[-1]), dtype=np.float32) + 0.01).astype(np.float32)
    return vals, ind, ptr


# ---------------------------------------------------------------------------
@pytest.mark.parametrize("slabs", [2, 4, 8])
@pytest.mark.parametrize("n_shards", [1, 2])
def test_loader_in_slabs_bit_exact(torch_cuda, slabs, n_shards):
    """dnpeff_set_csr with the values uploaded in several row slabs on a second stream
    (the path the end-to-end benchmark takes from 64 Mi entries on), forced here on a
    small ragged matrix whose rows 20..39 are empty, so that some slabs hold no entry:
    CSR, CSC, pruning map and |A|^2 against the oracle, bit for bit."""
    from npeff_ref_b200 import MuNmfParams
    rng = np.random.default_rng(100 + slabs)
    n, m = 67, 900
    lens = rng.integers(0, 60, size=n)
    lens[20:40] = 0
    lens[[0, 66]] = [0, 59]
    vals, ind, ptr = _ragged(rng, n, m, lens)
    norms = (rng.random(n, dtype=np.float32) + 0.5).astype(np.float32)
    v = O.normalize_rows(vals, ptr, norms)
    v, c, rp, n2o = O.prune_columns(v, ind, ptr, m, 2)
    mk = len(n2o)
    for s in range(n_shards):
        with _engine(MuNmfParams(rank=8), [("loader_slabs", slabs), ("keep_canonical_csr", 1)],
                     shard_index=s, n_shards=n_shards) as eng:
            eng.set_csr(n, m, vals, ind, ptr, 0, norms, 2)
            nn, mkept, c0, ms, nnz = eng.shape
            assert (nn, mkept) == (n, mk) and (c0, ms) == O.split_range(mk, n_shards, s)
            assert np.array_equal(eng.new_to_og(), n2o)
            sv, sc, srp = O.split_columns(v, c, rp, c0, ms)
            gv, gc, grp = eng.export_shard_csr()
            assert np.array_equal(grp, srp) and np.array_equal(gc, sc) and np.array_equal(gv, sv)
            cv, cr, cp = O.csr_to_csc(sv, sc, srp, ms)
            hv, hr, hp = eng.export_shard_csc()
            assert np.array_equal(hp, cp) and np.array_equal(hr, cr) and np.array_equal(hv, cv)
            assert abs(eng.a_sq_norm() - float((sv.astype(np.float64) ** 2).sum())) < 1e-9 * max(nnz, 1)


def test_loader_in_slabs_fixed_k_with_dense_block(torch_cuda):
    """The same with the D-PEF file's implicit offsets (k entries per row), a rank that
    keeps the popular columns as a dense block and narrow tail column blocks: the
    slab-wise extraction, bucketing and dense fill must give the factors of the
    one-slab load bit for bit, with and without the kept input-order CSR."""
    from npeff_ref_b200 import MuNmfParams
    n, m, k, r = 300, 9000, 1200, 32
    vals, idx, norms = make_problem(n, m, k, seed=41)
    v, c, rp, n2o = oracle_preprocess(vals, idx, norms, m)
    mk = len(n2o)
    scale = baseline_scale(v, n, mk, r)
    outs = []
    for slabs, keep in [(1, 1), (4, 1), (4, 0), (8, 0)]:
        with _engine(MuNmfParams(rank=r, eps=1e-12, seed=3, init_scale=scale),
                     [("loader_slabs", slabs), ("keep_canonical_csr", keep), ("tail_block_bytes", 64 * 1024)]) as eng:
            eng.set_csr(n, m, vals, idx, None, k, norms, 1)
            n_pop, pop_nnz, n_blocks, tile_rows = eng.layout()
            assert n_pop >= 8 and tile_rows == 0 and n_blocks >= 4
            if keep:
                gv, gc, grp = eng.export_shard_csr()
                assert np.array_equal(grp, rp) and np.array_equal(gc, c) and np.array_equal(gv, v)
            else:
                from npeff_ref_b200 import DnpeffError
                with pytest.raises(DnpeffError) as ei:
                    eng.export_shard_csr()
                assert ei.value.code == -1 and "keep_canonical_csr" in str(ei.value)
            eng.init_factors()
            W0, H0 = eng.load_w_to_host(), eng.load_h_to_host()
            eng.run(3, log_every=0)
            outs.append((eng.load_w_to_host(), eng.load_h_to_host(), eng.compute_uncached_loss()))
            cv, cr, cp = O.csr_to_csc(v, c, rp, mk)
            hv, hr, hp = eng.export_shard_csc()   # rebuilt at full size on demand
            assert np.array_equal(hp, cp) and np.array_equal(hr, cr) and np.array_equal(hv, cv)
            eng.step_h()                          # and the engine still iterates afterwards
    for W, H, l in outs[1:]:
        assert np.array_equal(W, outs[0][0]) and np.array_equal(H, outs[0][1]) and l == outs[0][2]
    Wo, Ho = O.run(v, c, rp, mk, W0, H0, 3, 1e-12)
    assert rel_fro(outs[0][0], Wo) < 1e-5 and rel_fro(outs[0][1], Ho) < 1e-5


def test_device_loader_in_internal_slabs(torch_cuda):
    """dnpeff_set_csr_device cuts large inputs into row slabs of its own; the slab
    boundaries must not show in the result (a matrix of 40 rows is one slab, so the
    check runs the slab loop through the host entry point with 8 slabs and compares
    it with the device entry point)."""
    from npeff_ref_b200 import MuNmfParams
    torch = torch_cuda
    n, m, k, r = 40, 700, 90, 8
    vals, idx, norms = make_problem(n, m, k, seed=9)
    res = []
    for device_input in (False, True):
        with _engine(MuNmfParams(rank=r, seed=1, init_scale=0.1), [("loader_slabs", 8), ("keep_canonical_csr", 1)]) as eng:
            if device_input:
                dv, di, dn = (torch.from_numpy(a).cuda() for a in (vals, idx, norms))
                eng.set_csr_device(n, m, dv.data_ptr(), di.data_ptr(), 0, k, dn.data_ptr(), 1)
            else:
                eng.set_csr(n, m, vals, idx, None, k, norms, 1)
            res.append(eng.export_shard_csr() + eng.export_shard_csc())
    for a, b in zip(*res):
        assert np.array_equal(a, b)


# ---------------------------------------------------------------------------
def test_configuration_1_at_stated_size_with_loss_curve(torch_cuda):
    """Workload configuration 1 as stated: n = 2048 examples, m = 65 536 features, 4096
    stored values per row, Zipf(1.1) columns, rank 32, factors Uniform(0,1) *
    sqrt(mean(A)/r), eps = 1e-12, seed 0, 50 iterations.  Targets: W and H within 1e-4
    relative Frobenius of the float64-accumulating oracle from identical initial
    factors, the loss within 1e-5 relative at every 10th step."""
    from npeff_ref_b200 import MuNmfParams
    n, m, k, r, iters, eps = 2048, 65536, 4096, 32, 50, 1e-12
    vals, idx, norms = O.synth_pef_hashed(n, m, k, alpha=1.1, sigma=1.0, seed=0)
    v, c, rp, n2o = oracle_preprocess(vals, idx, norms, m)
    mk = len(n2o)
    scale = baseline_scale(v, n, mk, r)
    Wo0, Ho0 = O.init_factors(n, mk, r, 0, scale)
    Wo, Ho, ls = O.run(v, c, rp, mk, Wo0, Ho0, iters, eps, acc64=True, losses=True)
    with _engine(MuNmfParams(rank=r, eps=eps, seed=0, init_scale=scale)) as eng:
        eng.set_csr(n, m, vals, idx, None, k, norms, 1)
        assert eng.shape[1] == mk
        eng.init_factors()
        assert np.array_equal(eng.load_w_to_host(), Wo0) and np.array_equal(eng.load_h_to_host(), Ho0)
        for step in range(10, iters + 1, 10):
            eng.run(10, log_every=0)
            l = eng.compute_uncached_loss()
            assert abs(l - ls[step - 1]) < 1e-5 * ls[step - 1], (step, l, ls[step - 1])   # stated target
        W, H = eng.load_w_to_host(), eng.load_h_to_host()
    assert rel_fro(W, Wo) < 1e-4, rel_fro(W, Wo)      # stated target
    assert rel_fro(H, Ho) < 1e-4, rel_fro(H, Ho)


@pytest.mark.parametrize("n,m,k,r,iters,tail_bytes", [
    (400, 7000, 900, 384, 20, 2 << 20), (560, 7000, 900, 512, 20, 2 << 20),
    (1100, 60000, 6000, 128, 50, 8 << 20), (700, 30000, 1500, 256, 30, 4 << 20)])
def test_full_run_wide_and_headline_ranks(torch_cuda, n, m, k, r, iters, tail_bytes):
    """Full runs at ranks 384 and 512 (panelled tensor-core kernels) and, at ranks 128
    and 256, on matrices whose dense popular block spans several row tiles and K
    splits with several tail column blocks and rows long enough for the block-per-row
    gather kernel; loss compared every 10th step."""
    from npeff_ref_b200 import MuNmfParams
    eps = 1e-12
    vals, idx, norms = make_problem(n, m, k, seed=n + r)
    v, c, rp, n2o = oracle_preprocess(vals, idx, norms, m)
    mk = len(n2o)
    scale = baseline_scale(v, n, mk, r)
    W0, H0 = O.init_factors(n, mk, r, 5, scale)
    Wo, Ho, ls = O.run(v, c, rp, mk, W0, H0, iters, eps, acc64=True, losses=True)
    a2 = float((v.astype(np.float64) ** 2).sum())
    with _engine(MuNmfParams(rank=r, eps=eps, seed=5, init_scale=scale), [("tail_block_bytes", tail_bytes)]) as eng:
        eng.set_csr(n, m, vals, idx, None, k, norms, 1)
        n_pop, _, n_blocks, tile_rows = eng.layout()
        assert n_pop > 128 and tile_rows == 0 and n_blocks >= 2
        eng.init_factors()
        for step in range(10, iters + 1, 10):
            eng.run(10, log_every=0)
            l = eng.compute_uncached_loss()
            # squared form: accurate to 3e-6 of |A|^2 (see test_full_run_matches_oracle);
            # the 1e-5 relative target applies where the fit is not near-exact
            assert abs(l * l - ls[step - 1] ** 2) < 3e-6 * a2
            if ls[step - 1] ** 2 > 0.05 * a2:
                assert abs(l - ls[step - 1]) < 1e-5 * ls[step - 1], (step, l, ls[step - 1])
        W, H = eng.load_w_to_host(), eng.load_h_to_host()
    assert rel_fro(W, Wo) < 1e-4, rel_fro(W, Wo)
    assert rel_fro(H, Ho) < 1e-4, rel_fro(H, Ho)


# ---------------------------------------------------------------------------
def test_host_generator_twin_matches_device_generator(torch_cuda):
    """The timed CPU arm generates its input with the host twin of the device
    generator: the column indices must be identical, the values equal to rounding."""
    from npeff_ref_b200._lib import lib, check
    torch = torch_cuda
    for (n, m, k, alpha, sigma, seed) in [(48, 50000, 2048, 1.1, 1.0, 7), (33, 4096, 1024, 1.4, 2.0, 4),
                                         (5, 300, 300, 1.1, 1.0, 1)]:
        vals = torch.empty((n, k), dtype=torch.float32, device="cuda")
        idx = torch.empty((n, k), dtype=torch.int32, device="cuda")
        norms = torch.empty((n,), dtype=torch.float32, device="cuda")
        st = torch.cuda.current_stream().cuda_stream
        check(lib().dnpeff_synth_pef_device(n, m, k, alpha, sigma, seed, vals.data_ptr(), idx.data_ptr(),
                                            norms.data_ptr(), st))
        hv, hi, hn = O.synth_pef_hashed(n, m, k, alpha=alpha, sigma=sigma, seed=seed)
        assert np.array_equal(idx.cpu().numpy(), hi)
        assert np.allclose(vals.cpu().numpy(), hv, rtol=2e-6, atol=0)
        assert np.allclose(norms.cpu().numpy(), hn, rtol=2e-6)


def test_streamed_file_loader_matches_array_loader(torch_cuda, tmp_path):
    """dnpeff_load_pef_hdf5 reads the engine's rows in 64 MB chunks through two pinned
    staging buffers; a file of 2 600 x 16 384 values (170 MB per dataset) takes three
    chunks, so both buffers are reused.  The loaded matrix must equal, bit for bit, the
    one dnpeff_set_csr builds from the same arrays; the leading-hyperslab arguments
    (--n_examples, --n_fisher_values) are covered too."""
    import ctypes as C
    from npeff_ref_b200 import MuNmfParams
    from npeff_ref_b200._lib import lib, check
    n, m, k = 2600, 300000, 16384
    vals, idx, norms = O.synth_pef_hashed(n, m, k, seed=12)
    path = str(tmp_path / "pef.h5")
    check(lib().dnpeff_write_pef_hdf5(path.encode(), n, k, C.c_void_p(vals.ctypes.data), C.c_void_p(idx.ctypes.data),
                                      C.c_void_p(norms.ctypes.data), m))
    for (ne, nk) in [(0, 0), (1500, 9000)]:
        rows, cols = (ne or n), (nk or k)
        with _engine(MuNmfParams(rank=8), [("keep_canonical_csr", 1)]) as a, \
                _engine(MuNmfParams(rank=8), [("keep_canonical_csr", 1)]) as b:
            check(lib().dnpeff_load_pef_hdf5(a._h, path.encode(), ne, nk, 2))
            b.set_csr(rows, m, np.ascontiguousarray(vals[:rows, :cols]), np.ascontiguousarray(idx[:rows, :cols]),
                      None, cols, norms[:rows], 2)
            assert a.shape == b.shape and np.array_equal(a.new_to_og(), b.new_to_og())
            for x, y in zip(a.export_shard_csr(), b.export_shard_csr()):
                assert np.array_equal(x, y)


def test_device_generator_row_ranges_are_slices_of_the_matrix(torch_cuda):
    """dnpeff_synth_pef_device_rows: a row's content depends on its index and the seed
    only, so a rank of a row-split job generates exactly its slice of the matrix."""
    from npeff_ref_b200._lib import lib, check
    torch = torch_cuda
    n, m, k = 37, 9000, 512
    st = torch.cuda.current_stream().cuda_stream

    def gen(first, rows):
        v = torch.empty((rows, k), dtype=torch.float32, device="cuda")
        i = torch.empty((rows, k), dtype=torch.int32, device="cuda")
        nr = torch.empty((rows,), dtype=torch.float32, device="cuda")
        check(lib().dnpeff_synth_pef_device_rows(first, rows, m, k, 1.1, 1.0, 3, v.data_ptr(), i.data_ptr(),
                                                 nr.data_ptr(), st))
        return v.cpu().numpy(), i.cpu().numpy(), nr.cpu().numpy()

    fv, fi, fn = gen(0, n)
    for first, rows in [(0, 10), (10, 20), (30, 7)]:
        v, i, nr = gen(first, rows)
        assert np.array_equal(v, fv[first:first + rows]) and np.array_equal(i, fi[first:first + rows])
        assert np.array_equal(nr, fn[first:first + rows])


# ---------------------------------------------------------------------------
def test_bounded_wait_runs_out_and_engine_recovers(torch_cuda):
    """The only device-side failure detection in the product: every wait between the
    roles of the warp-specialised tensor-core kernel is bounded.  With the limit set
    to a single poll the first wait for a bulk copy runs out, the kernel leaves
    cleanly (copies and MMAs already issued are waited for with the full limit, its
    TMEM is freed), and the next status read reports DNPEFF_ERR_CUDA.  With the limit
    restored the same engine computes correct results.  No fault, trap or hang is
    involved: the kernel returns by itself."""
    from npeff_ref_b200 import MuNmfParams, DnpeffError
    n, m, k, r, eps = 700, 20000, 2000, 64, 1e-12
    vals, idx, norms = make_problem(n, m, k, seed=123)
    v, c, rp, n2o = oracle_preprocess(vals, idx, norms, m)
    mk = len(n2o)
    scale = baseline_scale(v, n, mk, r)
    with _engine(MuNmfParams(rank=r, eps=eps, seed=2, init_scale=scale)) as eng:
        eng.set_csr(n, m, vals, idx, None, k, norms, 1)
        assert eng.layout()[3] == 0            # dense popular block: k_block_tc is on the path
        eng.init_factors()
        W0, H0 = eng.load_w_to_host(), eng.load_h_to_host()
        eng.set_option("wait_limit", 1)
        eng.step_w()
        with pytest.raises(DnpeffError) as ei:
            eng.synchronize()
        assert ei.value.code == -2 and "ran out" in str(ei.value)
        eng.set_option("wait_limit", 0)        # back to the default
        eng.synchronize()                      # the status was reported once and cleared
        eng.init_factors(W0, H0)
        eng.step_w()
        W1 = eng.load_w_to_host()
        assert rel_fro(W1, O.step_w(v, c, rp, mk, W0, H0, eps)) < 2e-6


# ---------------------------------------------------------------------------
@pytest.mark.parametrize("n,m,lens,r", [
    (1, 40, (7, 8), 32), (3, 60, (1, 2), 5), (64, 2048, (96, 97), 32), (149, 5000, (0, 40), 64), (149, 5000, (0, 40), 52),
    (700, 9001, (1, 900), 96), (300, 9000, (1500, 1501), 128), (2000, 400, (150, 250), 20)])
def test_small_problems_in_one_launch(torch_cuda, n, m, lens, r):
    """Runs of more than one iteration of a small problem are one cooperative launch: fewer rows
    than blocks and more, rows without entries, rows of one entry and rows cut over many
    units of entries, against single steps (the large path) and the oracle; twice the same bits."""
    from npeff_ref_b200 import MuNmfParams
    rng = np.random.default_rng(n + r)
    vals, ind, ptr = _ragged(rng, n, m, rng.integers(lens[0], lens[1], size=n))
    iters, eps = 7, 1e-8
    got = []
    with _engine(MuNmfParams(rank=r, eps=eps, seed=6, init_scale=0.3)) as eng:
        eng.set_csr(n, m, vals, ind, ptr, 0, None, 1)
        mk = eng.shape[1]
        W0, H0 = O.init_factors(n, mk, r, 6, 0.3)
        for _ in range(2):
            eng.init_factors()
            launches = eng.launch_count()
            eng.run(iters, log_every=0)
            launches = eng.launch_count() - launches
            got.append((eng.load_w_to_host(), eng.load_h_to_host()))
        assert launches == 1  # (the first run makes the CSC as well)
        eng.init_factors()
        for _ in range(iters):
            eng.step_w()
            eng.step_h()
        Ws, Hs = eng.load_w_to_host(), eng.load_h_to_host()
    v, c, rp, n2o = O.prune_columns(vals, ind, ptr, m, 1)
    Wo, Ho, ls = O.run(v, c, rp, mk, W0, H0, iters, eps, acc64=True, losses=True)
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert rel_fro(got[0][0], Wo) < 1e-5 and rel_fro(got[0][1], Ho) < 1e-5
    assert rel_fro(got[0][0], Ws) < 1e-5 and rel_fro(got[0][1], Hs) < 1e-5


@pytest.mark.parametrize("n,m,lens,r", [
    (65, 3000, (40, 41), 96), (129, 2600, (1, 60), 128),      # a row more than a tile, or a half, of the wide strides
    (600, 900, (300, 301), 100), (2400, 70, (30, 60), 96),    # rows cut over many workers; more rows than tiles on W's side
    (40, 50000, (2000, 2100), 64), (16, 20000, (6000, 6001), 128),   # several tiles a worker on H's
    (24, 20000, (3000, 3001), 96), (24, 26000, (3000, 3001), 90)])
def test_small_problem_tiles_and_tiny_values(torch_cuda, n, m, lens, r):
    """The one-launch kernel around its tiles and cuts, and with components so small that numerators fall below 2^-100
    and below the normal range: against single steps and the oracle."""
    from npeff_ref_b200 import MuNmfParams
    rng = np.random.default_rng(n + m + r)
    vals, ind, ptr = _ragged(rng, n, m, rng.integers(lens[0], lens[1], size=n))
    iters, eps = 3, 1e-8
    with _engine(MuNmfParams(rank=r, eps=eps, seed=6, init_scale=0.3)) as eng:
        eng.set_csr(n, m, vals, ind, ptr, 0, None, 1)
        mk = eng.shape[1]
        W0, H0 = O.init_factors(n, mk, r, 6, 0.3)
        H0[::5] *= np.float32(1e-33)
        H0[1::7] *= np.float32(1e-38)
        for _ in range(2):
            eng.init_factors(W0, H0)
            launches = eng.launch_count()
            eng.run(iters, log_every=0)
            launches = eng.launch_count() - launches
        assert launches == 1  # (the first run makes the CSC as well)
        got = eng.load_w_to_host(), eng.load_h_to_host()
        eng.init_factors(W0, H0)
        for _ in range(iters):
            eng.step_w()
            eng.step_h()
        Ws, Hs = eng.load_w_to_host(), eng.load_h_to_host()
    v, c, rp, n2o = O.prune_columns(vals, ind, ptr, m, 1)
    Wo, Ho, _ = O.run(v, c, rp, mk, W0, H0, iters, eps, acc64=True, losses=True)
    for g, s, o in ((got[0], Ws, Wo), (got[1], Hs, Ho)):
        assert rel_fro(g, o) < 1e-5 and rel_fro(g, s) < 1e-5
        assert np.isfinite(g).all()
    # Entry by entry: an update is good to a few 1e-6 (numerator and denominator are sums of positive terms: 2^-24 times the
    # square root of their number and more, and the tensor core's 6e-7), three updates of either factor to 4e-5; the last place of
    # the subnormal range, 2^-149, once an update and factor
    assert np.allclose(got[1], Ho, rtol=4e-5, atol=1e-44), np.abs(got[1] - Ho).max()


@pytest.mark.parametrize("n,m,k,r", [(8000, 1200000, 4000, 32), (17000, 200000, 1800, 20)])
def test_small_problem_long_sums_against_float64(torch_cuda, n, m, k, r):
    """The one-launch kernel with some 3e7 entries: tens of tiles a worker on H's side, rows of thousands of entries on W's, and
    units of one and a half to two thousand entries a row or less.  Two iterations against float64: a numerator is a
    sum of chains of 64 and then of at most some 60 positive terms, off by 2^-24 * 0.5 * sqrt(124 / 3) = 2e-7 at one standard
    deviation of the roundings (half of it measured), and two numerators of either factor go into the result; one
    chain of two thousand alone would be off by 7e-7."""
    from npeff_ref_b200 import MuNmfParams
    from npeff_ref_b200._lib import lib, check
    torch = torch_cuda
    vals = torch.empty((n, k), dtype=torch.float32, device="cuda")
    idx = torch.empty((n, k), dtype=torch.int32, device="cuda")
    norms = torch.empty((n,), dtype=torch.float32, device="cuda")
    check(lib().dnpeff_synth_pef_device(n, m, k, 1.1, 1.0, 5, vals.data_ptr(), idx.data_ptr(), norms.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream))
    vals /= norms[:, None]
    torch.cuda.synchronize()
    eps = 1e-12
    with _engine(MuNmfParams(rank=r, eps=eps, seed=3)) as eng:
        eng.set_csr_device(n, m, vals.data_ptr(), idx.data_ptr(), 0, k, 0, 1)
        mk = eng.shape[1]
        eng.set_init_scale((eng.a_sum() / (n * mk) / r) ** 0.5)
        for _ in range(2):
            eng.init_factors()
            W0, H0 = eng.load_w_to_host(), eng.load_h_to_host()
            launches = eng.launch_count()
            eng.run(2, log_every=0)
            launches = eng.launch_count() - launches
        assert launches == 1
        got = [torch.from_numpy(x).cuda() for x in (eng.load_w_to_host(), eng.load_h_to_host().T.copy())]
        to_kept = torch.zeros(m, dtype=torch.int64, device="cuda")
        to_kept[torch.from_numpy(eng.new_to_og()).cuda().long()] = torch.arange(mk, device="cuda")
    W, H = (torch.from_numpy(x).cuda().double() for x in (W0, H0.T.copy()))
    parts = [(to_kept[idx[a:a + 1000].long()], vals[a:a + 1000].double()) for a in range(0, n, 1000)]
    for _ in range(2):
        num = torch.cat([torch.bmm(v.unsqueeze(1), H[c.reshape(-1)].reshape(*c.shape, r))[:, 0] for c, v in parts])
        W = W * (num / (W @ (H.T @ H) + eps))
        num = torch.zeros_like(H)
        for (c, v), w in zip(parts, W.split(1000)):
            num.index_add_(0, c.reshape(-1), (v.unsqueeze(2) * w.unsqueeze(1)).reshape(-1, r))
        H = H * (num / (H @ (W.T @ W) + eps))
    for g, want in zip(got, (W, H)):
        assert float((g.double() - want).norm() / want.norm()) < 3e-7


def test_small_problem_barrier_wait_runs_out(torch_cuda):
    """With a wait limit of one poll the grid barrier of the small-problem kernel gives up, every
    block leaves, the status says so, and the engine works again with the default limit."""
    from npeff_ref_b200 import MuNmfParams, DnpeffError
    n, m, k, r = 200, 4000, 120, 32
    vals, idx, norms = make_problem(n, m, k, seed=9)
    with _engine(MuNmfParams(rank=r, eps=1e-8, seed=2, init_scale=0.1)) as eng:
        eng.set_csr(n, m, vals, idx, None, k, norms, 1)
        eng.init_factors()
        eng.run(5, log_every=0)
        want = eng.load_w_to_host()
        eng.set_option("wait_limit", 1)
        eng.init_factors()
        eng.run(5, log_every=0)
        with pytest.raises(DnpeffError) as ei:
            eng.synchronize()
        assert ei.value.code == -2 and "ran out" in str(ei.value)
        eng.set_option("wait_limit", 0)
        eng.init_factors()
        eng.run(5, log_every=0)
        assert np.array_equal(eng.load_w_to_host(), want)


def test_small_problems_of_two_engines_at_once(torch_cuda):
    """Two threads with an engine and a stream each, at the strides whose blocks hold all of an SM's TMEM: launches of the
    one-launch kernel queue up behind one another (a block takes more than half of an SM's shared memory) and give
    the same bits as one engine after the other."""
    import threading
    from npeff_ref_b200 import MuNmfParams
    torch = torch_cuda
    problems = [(300, 9000, 1500, 128), (200, 20000, 600, 96)]
    inputs = [make_problem(n, m, k, seed=n + r) for n, m, k, r in problems]
    got = [[], []]

    def job(i, runs, out):
        n, m, k, r = problems[i]
        vals, idx, norms = inputs[i]
        stream = torch.cuda.Stream()
        with _engine(MuNmfParams(rank=r, eps=1e-8, seed=6, init_scale=0.05), stream=stream.cuda_stream) as eng:
            eng.set_csr(n, m, vals, idx, None, k, norms, 1)
            for _ in range(runs):
                eng.init_factors()
                eng.run(100, log_every=0)
                out.append((eng.load_w_to_host(), eng.load_h_to_host()))

    for i in range(2):
        job(i, 1, got[i])
    threads = [threading.Thread(target=job, args=(i, 10, got[i])) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for outs in got:
        assert len(outs) == 11
        for W, H in outs[1:]:
            assert np.array_equal(W, outs[0][0]) and np.array_equal(H, outs[0][1])


@pytest.mark.parametrize("popular", [8, 0])
def test_small_problem_with_more_rows_than_a_long_column_can_have(torch_cuda, popular):
    """Rank 32 with 820 000 rows of two entries, just past the rows up to which a column of more than 512 entries can be put in row
    order: with popular columns (102 500 entries each) the one-launch kernel, which needs them in the CSC, would be refused what
    the large path does; without them it runs.  Against the oracle and single steps, and by the number of launches."""
    from npeff_ref_b200 import MuNmfParams
    rng = np.random.default_rng(popular)
    n, m, r, iters, eps = 820000, 4000, 32, 2, 1e-8
    rows = np.arange(n)
    ind = np.stack([rng.permutation(rows) % (popular or m // 2), m // 2 + rng.permutation(rows) % (m // 2)], axis=1).astype(np.int32)
    vals = rng.random((n, 2), dtype=np.float32) + np.float32(0.1)
    with _engine(MuNmfParams(rank=r, eps=eps, seed=6, init_scale=0.3)) as eng:
        eng.set_csr(n, m, vals, ind, None, 2, None, 1)
        mk = eng.shape[1]
        assert eng.layout()[0] == popular
        W0, H0 = O.init_factors(n, mk, r, 6, 0.3)
        for _ in range(2):
            eng.init_factors()
            launches = eng.launch_count()
            eng.run(iters, log_every=0)
            launches = eng.launch_count() - launches
        assert (launches == 1) == (popular == 0)
        got = eng.load_w_to_host(), eng.load_h_to_host()
        eng.init_factors()
        for _ in range(iters):
            eng.step_w()
            eng.step_h()
        steps = eng.load_w_to_host(), eng.load_h_to_host()
    v, c, rp, n2o = O.prune_columns(vals.ravel(), ind.ravel(), np.arange(0, 2 * n + 1, 2, dtype=np.int64), m, 1)
    want = O.run(v, c, rp, mk, W0, H0, iters, eps, acc64=True, losses=True)
    for g, s, o in zip(got, steps, want):
        assert rel_fro(g, o) < 1e-5 and rel_fro(g, s) < 1e-5


@pytest.mark.parametrize("iters,log_every", [(7, 0), (5, 2)])
def test_small_problem_without_room_for_its_launch(torch_cuda, capfd, iters, log_every):
    """Where the runtime refuses the cooperative launch of the small-problem kernel (the process may use
    only some of the SMs), the run is made by the large path: the same bits as step by step, and
    every log line is there."""
    from npeff_ref_b200 import MuNmfParams
    n, m, k, r = 200, 4000, 120, 32
    vals, idx, norms = make_problem(n, m, k, seed=9)
    with _engine(MuNmfParams(rank=r, eps=1e-8, seed=2, init_scale=0.1), [("refuse_cooperative", 1)]) as eng:
        eng.set_csr(n, m, vals, idx, None, k, norms, 1)
        eng.init_factors()
        for _ in range(iters):
            eng.step_w()
            eng.step_h()
        want = eng.load_w_to_host(), eng.load_h_to_host()
        eng.init_factors()
        eng.run(iters, log_every=log_every)
        got = eng.load_w_to_host(), eng.load_h_to_host()
        eng.set_option("refuse_cooperative", 0)
        eng.init_factors()
        eng.run(iters, log_every=0)
        small = eng.load_w_to_host()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    assert rel_fro(small, want[0]) < 1e-5
    assert capfd.readouterr().out.count("step ") == (iters // log_every if log_every else 0)


def test_small_problem_after_memory_ran_out(torch_cuda):
    """A run that finds no memory for the one-launch kernel's buffers says so, and the next one, with memory again,
    makes them all.  The engine's 64 MB slab is filled to different degrees by H, so that in some of the sizes the partials
    (19 MB) do not fit behind the smaller buffers, and the device has no room for another slab."""
    from npeff_ref_b200 import MuNmfParams, DnpeffError, release_memory
    torch = torch_cuda
    n, r, failed = 40, 128, 0
    for m in range(60000, 120001, 10000):
        rng = np.random.default_rng(m)
        idx = rng.permutation(m).astype(np.int32).reshape(n, m // n)   # every column once
        vals = rng.random((n, m // n), dtype=np.float32)

        def engine():
            eng = _engine(MuNmfParams(rank=r, eps=1e-8, seed=2, init_scale=0.1), keep_memory=False)
            eng.set_csr(n, m, vals, idx, None, m // n, None, 1)
            eng.export_shard_csc()                                     # (built in full)
            eng.init_factors()
            return eng

        with engine() as eng:
            eng.run(3, log_every=0)
            want = eng.load_w_to_host(), eng.load_h_to_host()
        with engine() as eng:
            release_memory()
            torch.cuda.empty_cache()
            filler = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
            try:
                eng.run(3, log_every=0)
            except DnpeffError as e:
                assert e.code == -2 and "cudaMalloc" in str(e)
                failed += 1
            del filler
            torch.cuda.empty_cache()
            eng.init_factors()
            eng.run(3, log_every=0)
            assert np.array_equal(eng.load_w_to_host(), want[0]) and np.array_equal(eng.load_h_to_host(), want[1])
    assert failed > 0


def test_failed_csc_builds_hold_no_memory(torch_cuda):
    """A matrix with a column twice in a row is refused when the CSC is built, and every time anew: the arrays of
    the builds that failed (80 MB each) do not add up."""
    from npeff_ref_b200 import MuNmfParams, DnpeffError
    n, k = 2000, 5000
    idx = np.tile(np.arange(k, dtype=np.int32), (n, 1))
    idx[7, 5] = idx[7, 6]
    vals = np.ones((n, k), np.float32)
    free = []
    with _engine(MuNmfParams(rank=20), keep_memory=False) as eng:
        eng.set_csr(n, k, vals, idx, None, k, None, 1)
        for _ in range(6):
            with pytest.raises(DnpeffError, match="twice"):
                eng.export_shard_csc()
            free.append(torch_cuda.cuda.mem_get_info()[0])
    assert free[0] - free[-1] < (100 << 20), free


@pytest.mark.parametrize("keep", [False, True])
def test_device_memory_after_destroy(torch_cuda, keep):
    """dnpeff_destroy gives the device memory back; with keep_memory it stays for the next engine, which
    uses it, and dnpeff_release_memory gives it back.  Free memory as the device reports it, to 32 MB
    (modules that load on first use are loaded by a first engine)."""
    from npeff_ref_b200 import MuNmfParams, release_memory
    torch = torch_cuda
    n, m, k, r = 64, 1 << 20, 8, 128
    rng = np.random.default_rng(0)
    idx = np.stack([rng.choice(m, k, replace=False) for _ in range(n)]).astype(np.int32)
    vals = rng.random((n, k), dtype=np.float32)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def job(keep):
        # a list of kept columns makes H large with few entries: 524288 x 128 floats
        eng = _engine(MuNmfParams(rank=r, eps=1e-8), keep_memory=keep)
        eng.set_csr_retain(n, m, vals, idx, np.arange(1 << 19, dtype=np.int32), None, k)
        eng.init_factors()
        eng.step_w()
        eng.step_h()
        inside = free()
        eng.close()
        return inside

    job(False)
    release_memory()
    before = free()
    inside = job(keep)
    after = free()
    assert before - inside > (400 << 20)       # H and A^T W, 256 MB each
    if keep:
        assert before - after > (400 << 20)
        assert abs(job(True) - inside) < (32 << 20)
        release_memory(0)
        after = free()
    assert before - after < (32 << 20)


def test_layout_near_the_memory_cap_does_not_depend_on_earlier_engines(torch_cuda):
    """Where the dense block is capped by the free memory, what earlier engines left for the next one, and
    what the engine itself holds from an earlier load, counts as free: the same popular columns and the same
    bits of W from a fresh process's engine, from one that comes after others, and from one loaded again."""
    from npeff_ref_b200 import MuNmfParams, release_memory
    from npeff_ref_b200._lib import lib, check
    torch = torch_cuda
    n, m, k, r = 8192, 40000, 2048, 32
    vals = torch.empty((n, k), dtype=torch.float32, device="cuda")
    idx = torch.empty((n, k), dtype=torch.int32, device="cuda")
    norms = torch.empty(n, dtype=torch.float32, device="cuda")
    check(lib().dnpeff_synth_pef_device(n, m, k, 0.05, 1.0, 3, vals.data_ptr(), idx.data_ptr(), norms.data_ptr(),
                                        torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()

    def load(eng):
        eng.set_csr_device(n, m, vals.data_ptr(), idx.data_ptr(), 0, k, norms.data_ptr(), 1)
        eng.init_factors()
        eng.step_w()
        eng.step_h()
        eng.step_w()
        return eng.layout()[0], eng.load_w_to_host()

    params = MuNmfParams(rank=r, eps=1e-8, seed=1, init_scale=0.1)
    with _engine(params) as eng:               # modules that load on first use
        load(eng)
    release_memory()
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (11 << 29), dtype=torch.uint8, device="cuda")  # 5.5 GB are left
    try:
        with _engine(params) as eng:
            first = load(eng)
            again = load(eng)
        with _engine(MuNmfParams(rank=128, eps=1e-8, seed=1, init_scale=0.1)) as eng:
            load(eng)                          # leaves slabs of other sizes
        with _engine(params) as eng:
            later = load(eng)
    finally:
        del filler
        torch.cuda.empty_cache()
        release_memory()
    assert 128 <= first[0] < 30000             # capped: 40000 columns are held by a 32nd of the rows
    for got in (again, later):
        assert got[0] == first[0] and np.array_equal(got[1], first[1])


@pytest.mark.parametrize("n_shards,m_kept,padded", [(2, 1 << 20, True), (2, 31_000_000, False), (1, 1 << 20, True)])
def test_padding_of_a_sharded_rank_is_bounded(torch_cuda, n_shards, m_kept, padded):
    """Rank 130 is stored with a stride of 256 while that costs an engine of a job at most 22.5 GB, by sizes
    that all engines know, and as it is beyond.  The stride shows in the memory that H takes."""
    from npeff_ref_b200 import MuNmfParams, release_memory
    n, k, r = 40, 4, 130
    rng = np.random.default_rng(1)
    idx = np.stack([rng.choice(m_kept, k, replace=False) for _ in range(n)]).astype(np.int32)
    vals = rng.random((n, k), dtype=np.float32)
    free = torch_cuda.cuda.mem_get_info
    with _engine(MuNmfParams(rank=r), keep_memory=False, n_shards=n_shards) as eng:
        release_memory()
        before = free()[0]
        eng.set_csr_retain(n, m_kept, vals, idx, np.arange(m_kept, dtype=np.int32), None, k)
        columns = eng.shape[3]
        used = before - free()[0]
    assert columns == m_kept // n_shards
    assert (used > 4 * columns * 220) == padded      # H: 520 bytes a column, or 1024


# ---------------------------------------------------------------------------
def test_one_engine_loaded_again_with_other_sizes(torch_cuda):
    """One engine takes matrices of growing and shrinking size (its memory comes from slabs that
    stay), with host arrays on both sides of the size from which they go through page-locked
    chunks (1 MB a thread, and chunks that do not divide it): the shard bit-exact, factors given
    and read back unchanged, and a second engine in use at the same time not disturbed."""
    from npeff_ref_b200 import MuNmfParams
    r = 24
    with _engine(MuNmfParams(rank=r, eps=1e-8, seed=1), [("keep_canonical_csr", 1)]) as eng, \
            _engine(MuNmfParams(rank=r, eps=1e-8, seed=1)) as other:
        vals0, idx0, norms0 = make_problem(60, 1500, 90, seed=7)
        other.set_csr(60, 1500, vals0, idx0, None, 90, norms0, 1)
        other.init_factors()
        before = other.load_h_to_host()
        for n, m, k in [(50, 3000, 111), (900, 40001, 1531), (300, 9000, 1500), (1, 500, 37), (1301, 60007, 2111)]:
            vals, idx, norms = make_problem(n, m, k, seed=n)
            v, c, rp, n2o = oracle_preprocess(vals, idx, norms, m)
            eng.set_csr(n, m, vals, idx, None, k, norms, 1)
            gv, gc, gp = eng.export_shard_csr()
            assert np.array_equal(gp, rp) and np.array_equal(gc, c) and np.array_equal(gv, v)
            assert np.array_equal(eng.new_to_og(), n2o)
            rng = np.random.default_rng(n)
            W0 = rng.random((n, r), dtype=np.float32)
            H0 = rng.random((r, len(n2o)), dtype=np.float32)
            eng.init_factors(W0, H0)
            assert np.array_equal(eng.load_w_to_host(), W0) and np.array_equal(eng.load_h_to_host(), H0)
            eng.step_w()
            assert rel_fro(eng.load_w_to_host(), O.step_w(v, c, rp, len(n2o), W0, H0, 1e-8)) < 2e-6
        assert np.array_equal(other.load_h_to_host(), before)


# ---------------------------------------------------------------------------
_NO_TC_SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/tests")
from npeff_ref_b200 import MuNmf, MuNmfParams
from helpers import make_problem
n, m, k, r = 300, 9000, 1500, 128
vals, idx, norms = make_problem(n, m, k, seed=428)
with MuNmf(MuNmfParams(rank=r, eps=1e-12, seed=0, init_scale=float(sys.argv[3]))) as eng:
    eng.set_csr(n, m, vals, idx, None, k, norms, 1)
    layout = eng.layout()
    eng.init_factors()
    eng.run(20, log_every=0)
    np.savez(sys.argv[2], W=eng.load_w_to_host(), H=eng.load_h_to_host(), loss=eng.compute_uncached_loss(),
             tile_rows=layout[3])
"""


def test_cuda_core_path_at_a_tensor_core_rank(torch_cuda, tmp_path):
    """DNPEFF_NO_TC=1 keeps every contraction on the CUDA-core kernels and the popular
    columns on the shared-memory tiled sparse kernel (the path other ranks take, and the
    A/B comparison for the tensor-core kernels).  At rank 128 it must match the oracle
    like the tensor-core path does."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    n, m, k, r, iters = 300, 9000, 1500, 128, 20
    vals, idx, norms = make_problem(n, m, k, seed=428)
    v, c, rp, n2o = oracle_preprocess(vals, idx, norms, m)
    mk = len(n2o)
    scale = baseline_scale(v, n, mk, r)
    W0, H0 = O.init_factors(n, mk, r, 0, scale)
    Wo, Ho, ls = O.run(v, c, rp, mk, W0, H0, iters, 1e-12, acc64=True, losses=True)
    outs = {}
    for name, env in (("tc", {}), ("no_tc", {"DNPEFF_NO_TC": "1"})):
        out = str(tmp_path / (name + ".npz"))
        res = subprocess.run([sys.executable, "-c", _NO_TC_SCRIPT, root, out, repr(scale)],
                             env=dict(os.environ, **env), capture_output=True, text=True, timeout=600)
        assert res.returncode == 0, res.stderr[-2000:]
        outs[name] = np.load(out)
    assert int(outs["tc"]["tile_rows"]) == 0 and int(outs["no_tc"]["tile_rows"]) > 0   # dense block / tiled sparse kernel
    for name in outs:
        assert rel_fro(outs[name]["W"], Wo) < 1e-4 and rel_fro(outs[name]["H"], Ho) < 1e-4, name
        assert abs(float(outs[name]["loss"]) - ls[-1]) < 1e-5 * ls[-1], name


@pytest.mark.parametrize("n,r", [(1, 32), (1184, 32), (1185, 30), (2369, 32), (593, 64), (1190, 50), (296, 96), (601, 96),
                                 (148, 128), (299, 128), (597, 100), (9001, 128)])
def test_w_only_steps_match_single_steps(torch_cuda, n, r):
    """fit_w_only's steps in one launch against as many single updates (tensor cores): the row counts where the
    rows per thread change, a ragged last block, padded ranks, and the rows from which on rank 128 leaves the CUDA cores."""
    from npeff_ref_b200 import MuNmfParams
    m, k, steps = 600, 40, 7
    vals, idx, norms = make_problem(n, m, k, seed=n + r)
    with _engine(MuNmfParams(rank=r, eps=1e-7, seed=4, init_scale=0.05)) as eng:
        eng.set_csr(n, m, vals, idx, None, k, norms, 1)
        eng.init_factors()
        for _ in range(steps):
            eng.step_w()
        want = eng.load_w_to_host()
        eng.init_factors()
        eng.fit_w_only(steps, want_loss=False)
        assert rel_fro(eng.load_w_to_host(), want) < 1e-5


@pytest.mark.parametrize("n,r", [(12000, 96), (12001, 96), (18944, 90), (18945, 96), (24001, 96)])
def test_w_only_steps_where_rank_96_changes_kernels(torch_cuda, n, r):
    """Rank 96 leaves the CUDA cores at 12000 rows a wave of the tensor-core kernel: either side of it, the
    last row of the first wave and the first of the second (the bound of the test above)."""
    test_w_only_steps_match_single_steps(torch_cuda, n, r)


@pytest.mark.parametrize("r", [64, 100, 128])
def test_large_h_into_page_locked_memory(torch_cuda, r):
    """A large H read back in parts (page-locked destination) against the one copy into pageable memory; 100: a ragged last part."""
    from npeff_ref_b200 import MuNmfParams
    from npeff_ref_b200._lib import lib, check
    n, m = 44, 268400
    rng = np.random.default_rng(r)
    idx = rng.permutation(m).astype(np.int32).reshape(n, m // n)   # every column once
    vals = rng.random((n, m // n), dtype=np.float32)
    with _engine(MuNmfParams(rank=r, eps=1e-8, seed=2, init_scale=0.1)) as eng:
        eng.set_csr(n, m, vals, idx, None, m // n, np.ones(n, np.float32), 1)
        eng.init_factors()
        want = eng.load_h_to_host()
        got = torch_cuda.zeros((r, m), pin_memory=True)
        check(lib().dnpeff_get_h(eng._h, got.data_ptr()))
        assert np.array_equal(got.numpy(), want)
