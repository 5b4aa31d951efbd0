"""Kernel paths at the sizes where they can go wrong, against the oracle (tolerance 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch as t
    assert t.cuda.is_available(), "GPU tests need a CUDA device"
    return t


def device_product(fpc, torch, q, a, b, **options):
    """One product through the device entry point, with the plan's status word checked."""
    n, limbs = a.shape
    with fpc.Plan(n, 32 * limbs, limbs, q, **options) as plan:
        da, db = (torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b))
        dc = torch.full_like(da, -1)
        plan.run_device(da.data_ptr(), db.data_ptr(), dc.data_ptr(), torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        assert plan.status() == 0
        return dc.cpu().numpy().view(np.uint32)


# rows around the chunks of 16 and 64 words that the reduction reads, with its switch between them
# (L + 2 = 64), and fewer rows than a warp has lanes
@pytest.mark.parametrize("limbs", [1, 2, 3, 13, 14, 15, 30, 31, 46, 61, 62, 63, 64, 125, 126, 127, 190])
@pytest.mark.parametrize("n", [1, 16, 64])
def test_reduction_row_ends(n, limbs, fpc, inputs, oracle, torch):
    full = inputs.random_modulus(limbs, 7 * limbs + n)
    narrow_top = full.copy()
    narrow_top[-1] = 1                  # results whose top word equals q's are common
    ones = np.full(limbs, 0xFFFFFFFF, np.uint32)   # q = 2^(32 L) - 1
    moduli = [full, ones] + ([narrow_top] if limbs > 1 else [])
    if limbs > 2:
        short = full.copy()
        short[limbs // 2:] = 0          # q shorter than its limbs
        short[limbs // 2 - 1] |= 1
        moduli.append(short)
    for q in moduli:
        rng = np.random.Generator(np.random.PCG64(limbs))
        words = np.flatnonzero(q)[-1] + 1
        pairs = [tuple(np.pad(inputs.random_operand(rng, n, q[:words]), ((0, 0), (0, limbs - words)))
                       for _ in range(2))]
        pairs += [(inputs.edge_operand(n, q, x), inputs.edge_operand(n, q, y)) for x, y in inputs.EDGE_PAIRS[1:]]
        for a, b in pairs:
            assert np.array_equal(device_product(fpc, torch, q, a, b), oracle.kronecker(q, a, b))


# byte GEMMs of one partial column tile (from 8192 rows on they go to the tensor cores), of a few
# tiles with a partial last one, and of K steps with zero-filled tails
@pytest.mark.parametrize("n,limbs", [(4096, 1), (4096, 5), (8192, 1), (8192, 2), (8192, 27), (8192, 29), (8192, 47),
                                     (8192, 60), (4096, 65)])
def test_partial_column_tiles(n, limbs, fpc, inputs, oracle, torch):
    q, a, b = inputs.instance(n, limbs, 900 + limbs, 0)
    assert np.array_equal(device_product(fpc, torch, q, a, b), oracle.kronecker(q, a, b))


# the gathering GEMMs: rows of one and two K steps with and without 16-byte rows, the switch between
# the fused reduction (L + 5 <= 64 words) and word sums, and the largest gathered CRT GEMM (L = 123)
@pytest.mark.parametrize("n,split", [(128, 1), (2048, 1), (2048, 4), (4096, 2)])
@pytest.mark.parametrize("limbs", [1, 4, 27, 28, 31, 32, 33, 56, 59, 60, 64, 65, 100, 123, 124])
def test_gathered_tiles(n, split, limbs, fpc, inputs, oracle, torch):
    q, a, b = inputs.instance(n, limbs, 70 + limbs, 0)
    want = oracle.kronecker(q, a, b)
    assert np.array_equal(device_product(fpc, torch, q, a, b, split=split), want)
    with fpc.Plan(n, 32 * limbs, limbs, q, split=split) as plan:
        assert np.array_equal(plan.run(a, b), want)


@pytest.mark.parametrize("limbs", [4, 28, 55])
def test_operands_on_any_word_boundary(limbs, fpc, inputs, oracle, torch):
    n = 1024
    q, a, b = inputs.instance(n, limbs, 5, 0)
    want = oracle.kronecker(q, a, b)
    stream = torch.cuda.current_stream().cuda_stream
    with fpc.Plan(n, 32 * limbs, limbs, q) as plan:
        for shift in ((0, 0, 0), (1, 0, 0), (0, 3, 1), (2, 2, 2)):
            buffers = [torch.zeros(n * limbs + 4, dtype=torch.int32, device="cuda") for _ in range(3)]
            views = [t[k:k + n * limbs] for t, k in zip(buffers, shift)]
            views[0].copy_(torch.from_numpy(a.view(np.int32).ravel()))
            views[1].copy_(torch.from_numpy(b.view(np.int32).ravel()))
            plan.run_device(*(v.data_ptr() for v in views), stream)
            torch.cuda.synchronize()
            assert np.array_equal(views[2].cpu().numpy().view(np.uint32).reshape(n, limbs), want)


def test_host_chunks_below_a_gathered_tile(fpc, inputs, oracle):
    """N=16384 in 16 transforms: the host path's output chunks are 64 positions of each transform."""
    n, limbs = 16384, 20
    q, a, b = inputs.instance(n, limbs, 8, 0)
    with fpc.Plan(n, 32 * limbs, limbs, q, split=16) as plan:
        assert np.array_equal(plan.run(a, b), oracle.kronecker(q, a, b))


# rows in 2 to 16 segments of a reduction, with carries that run through whole segments: with
# q = 2^(32 L) - 1 and its neighbours, products of q - 1 and of limbs of ones leave long runs of equal words
@pytest.mark.parametrize("limbs", [31, 32, 33, 63, 64, 127, 128, 254, 255, 256, 270, 300, 511, 520])
@pytest.mark.parametrize("n", [1, 4, 128])
def test_segmented_reduction(n, limbs, fpc, inputs, oracle, torch):
    top = 1 << (32 * limbs)
    for qv in (top - 1, top // 2 + 1, (top >> 33) - 1, top - (top >> 40) + 1):
        q = inputs.from_int(qv, limbs)
        rng = np.random.Generator(np.random.PCG64(limbs))
        words = np.flatnonzero(q)[-1] + 1
        pairs = [tuple(np.pad(inputs.random_operand(rng, n, q[:words]), ((0, 0), (0, limbs - words)))
                       for _ in range(2))]
        pairs += [(inputs.edge_operand(n, q, x), inputs.edge_operand(n, q, y)) for x, y in inputs.EDGE_PAIRS]
        for a, b in pairs:
            assert np.array_equal(device_product(fpc, torch, q, a, b), oracle.kronecker(q, a, b))


# every length of the fused transforms, with as few primes as possible and with more than one per SM
@pytest.mark.parametrize("n", [256, 512, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("limbs", [1, 75, 150])
def test_fused_transforms(n, limbs, fpc, inputs, oracle, torch):
    q, a, b = inputs.instance(n, limbs, 60 + limbs, 0)
    want = oracle.kronecker(q, a, b)
    assert np.array_equal(device_product(fpc, torch, q, a, b), want)
    with fpc.Plan(n, 32 * limbs, limbs, q) as plan:
        assert np.array_equal(plan.run(a, b), want)


# rings that run as one kernel (N r L up to 5000, 12288 at N = 64) and their neighbours that do not
@pytest.mark.parametrize("n,limbs", [(64, 1), (64, 2), (64, 8), (64, 9), (64, 10), (128, 1), (128, 3), (128, 4),
                                     (128, 5), (256, 1), (256, 2), (256, 3), (512, 1), (32, 2), (2048, 1)])
def test_small_products(n, limbs, fpc, inputs, oracle, torch):
    top = 1 << (32 * limbs)
    for qv in (inputs.to_int(inputs.random_modulus(limbs, n)), top - 1, top // 2 + 1, 3, (top >> 31) + 1):
        q = inputs.from_int(qv, limbs)
        rng = np.random.Generator(np.random.PCG64(limbs))
        words = np.flatnonzero(q)[-1] + 1
        pairs = [tuple(np.pad(inputs.random_operand(rng, n, q[:words]), ((0, 0), (0, limbs - words)))
                       for _ in range(2))]
        pairs += [(inputs.edge_operand(n, q, x), inputs.edge_operand(n, q, y)) for x, y in inputs.EDGE_PAIRS]
        for a, b in pairs:
            want = oracle.kronecker(q, a, b)
            assert np.array_equal(device_product(fpc, torch, q, a, b), want)
        with fpc.Plan(n, 32 * limbs, limbs, q) as plan:  # the last pair once more through the host path
            assert np.array_equal(plan.run(a, b), want)


def test_small_product_stages_match_the_general_path(fpc, inputs):
    """The stage buffers of a one-kernel product are those of the same product in stages."""
    n, limbs = 256, 3
    q, a, b = inputs.instance(n, limbs, 6, 0)
    dumps = []
    for gemm in (fpc.GEMM_AUTO, fpc.GEMM_SIMT):
        with fpc.Plan(n, 32 * limbs, limbs, q, gemm=gemm) as plan:
            c = plan.run(a, b)
            r = plan.info()["primes"]
            dumps.append((c.tobytes(), plan.debug_read(0)[:r * n * 4], plan.debug_read(1), plan.debug_read(2)))
    assert dumps[0] == dumps[1]


# the reduction over two column tiles, at one to four row tiles per CTA: L = 60..62 (the second tile
# holds words of the quotient only), the ends of the second tile, and word sums again past it
@pytest.mark.parametrize("n,limbs", [(8192, 60), (16384, 60), (16384, 61), (16384, 62), (16384, 63), (16384, 75),
                                     (16384, 123), (16384, 124), (32768, 62), (32768, 91), (65536, 60), (65536, 63), (65536, 123)])
def test_reduction_over_two_column_tiles(n, limbs, fpc, inputs, torch):
    q, a, b = inputs.instance(n, limbs, 300 + limbs, 0)
    top = inputs.edge_operand(n, q, "max")
    for x, y in ((a, b), (top, a), (top, top)):
        assert np.array_equal(device_product(fpc, torch, q, x, y),
                              device_product(fpc, torch, q, x, y, gemm=fpc.GEMM_SIMT))


def test_residues_past_four_gigabytes(fpc, inputs, oracle, torch):
    """2 r N residues of 4 bytes at N=131072, L=2048 are 4.5 GB: the conversions of both tensor kernels
    address operand b's last primes past 32 bits."""
    n, limbs = 131072, 2048
    q, a, b = inputs.instance(n, limbs, 41, 0)
    want = {i: oracle.schoolbook_at(q, a, b, i)[0] for i in (15, n - 1)}
    da, db = (torch.from_numpy(x.view(np.int32)).cuda() for x in (a, b))
    for gemm in (fpc.GEMM_AUTO, fpc.GEMM_TENSOR_SINGLE):
        with fpc.Plan(n, 32 * limbs, limbs, q, gemm=gemm) as plan:
            info = plan.info()
            assert info["gemm"] == 3 and 8 * info["primes"] * n > 1 << 32
            dc = torch.full_like(da, -1)
            plan.run_device(da.data_ptr(), db.data_ptr(), dc.data_ptr(), torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert plan.status() == 0
        for i, row in want.items():
            assert np.array_equal(row, dc[i].cpu().numpy().view(np.uint32)), (gemm, i)


# few primes and many zero limbs above q: the last one-kernel products (L = 48), and around 48 KB of their
# shared memory
@pytest.mark.parametrize("limbs", [47, 48, 49, *range(85, 94)])
@pytest.mark.parametrize("qv", [2001, (1 << 24) - 3, (1 << 27) - 39])
def test_small_products_with_zero_limbs(limbs, qv, fpc, inputs, oracle, torch):
    n, q = 64, inputs.from_int(qv, limbs)
    rng = np.random.Generator(np.random.PCG64(limbs))
    a, b = (np.pad(inputs.random_operand(rng, n, q[:1]), ((0, 0), (0, limbs - 1))) for _ in range(2))
    want = oracle.kronecker(q, a, b)
    assert np.array_equal(device_product(fpc, torch, q, a, b), want)
    with fpc.Plan(n, 32 * limbs, limbs, q) as plan:
        assert np.array_equal(plan.run(a, b), want)


def test_small_products_of_several_sizes_on_threads(fpc, inputs, oracle):
    """Launches of one-kernel products that need different amounts of shared memory."""
    import threading
    n, qv, failed = 64, 2001, []

    def worker(limbs):
        q = inputs.from_int(qv, limbs)
        a = np.pad(inputs.random_operand(np.random.Generator(np.random.PCG64(1)), n, q[:1]), ((0, 0), (0, limbs - 1)))
        want = oracle.kronecker(q, a, a)
        try:
            with fpc.Plan(n, 32 * limbs, limbs, q) as plan:
                for _ in range(2000):
                    assert np.array_equal(plan.run(a, a), want)
        except Exception as e:
            failed.append((limbs, repr(e)))

    threads = [threading.Thread(target=worker, args=(limbs,)) for limbs in (20, 48, 100, 192)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


# the word sums that the gathering CRT GEMM leaves (L = 60 up, below N = 16384), from exact products
@pytest.mark.parametrize("n,limbs,split", [(256, 60, 2), (512, 64, 1), (1024, 100, 4), (512, 123, 2)])
def test_word_sums_of_gathered_tiles(n, limbs, split, fpc, inputs):
    import model
    q, a, b = inputs.instance(n, limbs, 77, 0)
    setup = model.make_plan(n, limbs, inputs.to_int(q), split)
    product, weights, _, _ = model.crt_constants(setup)
    bits = 2 * 32 * limbs + n.bit_length()
    x, y = (sum(v << (bits * i) for i, v in enumerate(inputs.poly_to_ints(p))) for p in (a, b))
    z = x * y
    at = [(z >> (bits * i)) & ((1 << bits) - 1) for i in range(2 * n)]
    z = [at[i] - at[i + n] for i in range(n)]
    v = np.array([[zi * pow(product // p, -1, p) % p for p in setup.primes] for zi in z], dtype=np.uint32)
    words, r = limbs + 5, len(setup.primes)
    w_bytes = np.frombuffer(b"".join(w.to_bytes(4 * words, "little") for w in weights), np.uint8).reshape(r, 4 * words)
    columns = np.zeros((n, 4 * words), np.int64)
    v_bytes = v.view(np.uint8).reshape(n, r, 4).astype(np.int64)
    for d in range(4):  # column c takes byte c - d of W_k
        columns[:, d:] += v_bytes[:, :, d] @ w_bytes[:, :4 * words - d].astype(np.int64)
    sums = (columns.reshape(n, words, 4) << (8 * np.arange(4))).sum(axis=2)
    with fpc.Plan(n, 32 * limbs, limbs, q, split=split) as plan:
        assert inputs.poly_to_ints(plan.run(a, b)) == [zi % inputs.to_int(q) for zi in z]
        # the sums first: reading the CRT inputs may make them from the residues
        assert np.array_equal(np.frombuffer(plan.debug_read(2), np.int64).reshape(n, words), sums)
        crt_in = np.frombuffer(plan.debug_read(1), np.uint32).reshape(n, plan.info()["padded_primes"])
        assert np.array_equal(crt_in[:, :r], v) and not crt_in[:, r:].any()


def test_reading_a_stage_buffer_leaves_it_as_it_is(fpc, inputs, torch):
    """Word sums that the product keeps are read, not made again from the residues."""
    n, limbs = 512, 64
    q, a, b = inputs.instance(n, limbs, 77, 0)
    with fpc.Plan(n, 32 * limbs, limbs, q, external_work=True) as plan:
        work = torch.empty(plan.work_bytes(), dtype=torch.uint8, device="cuda")
        plan.bind_work(work.data_ptr(), work.numel())
        plan.run(a, b)
        work.fill_(0xA5)
        torch.cuda.synchronize()
        assert set(plan.debug_read(2)) == {0xA5}


def test_device_bytes_of_a_one_kernel_product(fpc, inputs):
    """A one-kernel product keeps its CRT weights as words, [r][L+5], beside the general path's tables."""
    n, limbs = 256, 2
    q, _, _ = inputs.instance(n, limbs, 6, 0)
    infos = []
    for gemm in (fpc.GEMM_AUTO, fpc.GEMM_SIMT):
        with fpc.Plan(n, 32 * limbs, limbs, q, gemm=gemm) as plan:
            infos.append(plan.info())
    small, general = infos
    assert small["kernels_per_product"] == 1 < general["kernels_per_product"]
    kept = 4 * small["primes"] * small["words"]
    assert small["table_bytes"] - general["table_bytes"] == kept
    assert small["device_bytes"] - general["device_bytes"] == kept


# the reduction over two column tiles against exact products: L = 60 and 62 (the second tile holds words of
# the quotient only), 63, and the last L that fits
@pytest.mark.parametrize("n,limbs", [(16384, 60), (16384, 62), (16384, 63), (16384, 123), (32768, 91)])
def test_reduction_over_two_column_tiles_matches_the_oracle(n, limbs, fpc, inputs, oracle, torch):
    q, a, b = inputs.instance(n, limbs, 300 + limbs, 0)
    top = inputs.edge_operand(n, q, "max")
    for x, y in ((a, b), (top, a), (top, top)):
        assert np.array_equal(device_product(fpc, torch, q, x, y), oracle.kronecker(q, x, y))


def test_many_zero_limbs_do_not_run_as_one_kernel(fpc, inputs):
    """N=64 with one prime: a thread's chain of L + 5 words made L = 192 slower in one kernel than in stages."""
    for limbs, one in ((4, True), (48, True), (49, False), (192, False)):
        with fpc.Plan(64, 32 * limbs, limbs, inputs.from_int(2001, limbs)) as plan:
            assert (plan.info()["kernels_per_product"] == 1) == one, limbs
