"""The tensor-core passes and top windows against the oracle, at the sizes where
their tiles, rounds and scalings change: every window size at both ends of the
index, short rounds, column counts around a tile's, cosets, odd strides."""
import numpy as np
import pytest

from conftest import kernel_names, raw_u64, to_dev, to_host

pytestmark = pytest.mark.gpu


def _ntt(log_n, cols, bitrev, inverse, ext=0, coset=0, gap=0, plan=None, seed=0):
    import torch

    import bc_ntt
    import oracle

    rng = np.random.default_rng(seed + 1000 * log_n + cols)
    n, stride = 1 << log_n, (1 << log_n) + gap
    x = raw_u64(rng, cols * stride)
    x[: min(n, 64)] = 2**64 - 1  # the largest digit sums
    d, o = to_dev(x), torch.full((cols * stride,), 7, dtype=torch.int64, device="cuda")
    if plan:
        bc_ntt.batch_ntt_with_plan(d, o, log_n, cols, stride, stride, bitrev, inverse, ext, coset, plan)
    else:
        bc_ntt.batch_ntt_internal(d.data_ptr(), o.data_ptr(), log_n, cols, stride, stride, bitrev, inverse, ext, coset)
    exp = np.asarray(oracle.batch_ntt(x, log_n, cols, stride, stride, bitrev, inverse, ext, coset))
    got = to_host(o).reshape(cols, stride)
    assert np.array_equal(got[:, :n], exp.reshape(cols, stride)[:, :n])
    assert (got[:, n:] == 7).all()


@pytest.mark.parametrize("log_n", [8, 9, 10, 11, 12])
@pytest.mark.parametrize("bitrev,inverse", [(False, False), (False, True), (True, False), (True, True)])
def test_low_windows(gpu_ctx, log_n, bitrev, inverse):
    g = 1 << (12 - log_n)  # columns of a tile
    for cols in {1, max(1, g - 1), g, g + max(1, 3 * g // 4), 2 * g + 1}:
        _ntt(log_n, cols, bitrev, inverse)
    _ntt(log_n, g, bitrev, inverse, gap=3)
    if bitrev == inverse:
        _ntt(log_n, g, bitrev, inverse, ext=2, coset=3, gap=1)


PLANS = [[(4, 8), (8, 1)], [(5, 8), (9, 1)], [(8, 8), (8, 1)], [(9, 8), (8, 1)], [(10, 4), (9, 1)], [(8, 8), (12, 1)],
         [(4, 8), (8, 8), (8, 1)], [(11, 2), (8, 1)]]


@pytest.mark.parametrize("plan", PLANS, ids=lambda p: "+".join(f"{k}.{c}" for k, c in p))
@pytest.mark.parametrize("bitrev,inverse", [(False, False), (False, True), (True, False), (True, True)])
def test_window_plans(gpu_ctx, plan, bitrev, inverse):
    log_n = sum(k for k, _ in plan)
    for cols, gap in ((1, 0), (9 if log_n < 19 else 3, 5)):
        _ntt(log_n, cols, bitrev, inverse, gap=gap, plan=plan)
        if bitrev == inverse:  # the scaling by the coset's powers, shared by the passes where all are of one kind
            _ntt(log_n, cols, bitrev, inverse, ext=1, coset=1, gap=gap, plan=plan)


@pytest.mark.parametrize("plan", [[(4, 8), (8, 1)], [(5, 8), (8, 1)], [(8, 8), (8, 1)], [(10, 4), (8, 1)],
                                  [(4, 8), (4, 8), (8, 1)], [(5, 8), (4, 8), (9, 1)]],
                         ids=lambda p: "+".join(f"{k}.{c}" for k, c in p))
@pytest.mark.parametrize("log_b", [1, 3, 4, 5])
def test_lde_top_windows(gpu_ctx, plan, log_b):
    import torch

    import bc_ntt
    import oracle

    log_n = sum(k for k, _ in plan)
    text = f"{log_n} {log_b} {len(plan)} " + " ".join(f"{k} {c}" for k, c in plan) + "\n"
    old = bc_ntt.plan_table_export()
    try:
        bc_ntt.plan_table_import(text)
        for cols in ((1, 13) if log_n + log_b < 20 else (3,)):
            n = 1 << log_n
            x = raw_u64(np.random.default_rng(log_n + cols), cols * n)
            x[:64] = 2**64 - 1
            d, o = to_dev(x), torch.zeros(cols * n << log_b, dtype=torch.int64, device="cuda")
            bc_ntt.lde(d, o, log_n, cols, log_b)
            assert np.array_equal(to_host(o), oracle.lde(x, log_n, cols, n, log_b)), cols
            # the top window runs on the tensor cores up to blowup 16, where the low one's tiles are filled
            g = 1 << (12 - plan[-1][0])
            tops = [k for k in kernel_names(lambda: bc_ntt.lde(d, o, log_n, cols, log_b)) if "top_kernel" in k]
            assert len(tops) == 1
            assert ("top_kernel_tc" in tops[0]) == (log_b <= 4 and 4 * cols >= 3 * g * -(-cols // g)), (cols, tops)
    finally:
        bc_ntt.plan_table_clear()
        if old:
            bc_ntt.plan_table_import(old)


def test_chains_in_a_graph_and_on_two_streams(gpu_ctx):
    """Kernels of one call overlap each other's start: repeated calls that read the previous call's output, two
    streams at once, and a captured graph give the canonical inputs back."""
    import torch

    import bc_ntt

    log_n, cols = 16, 16
    n = 1 << log_n
    words = raw_u64(np.random.default_rng(3), cols * n)
    x, want = to_dev(words), words % np.uint64(bc_ntt.P)

    def there_and_back(a, b):
        bc_ntt.batch_ntt_internal(a.data_ptr(), b.data_ptr(), log_n, cols, n, n, False, False, 0, 0)
        bc_ntt.batch_ntt_internal(b.data_ptr(), a.data_ptr(), log_n, cols, n, n, True, True, 0, 0)

    streams = [torch.cuda.Stream() for _ in range(2)]
    bufs = [(x.clone(), torch.empty_like(x)) for _ in streams]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, (a, b) in zip(streams, bufs):
            with torch.cuda.stream(s):
                there_and_back(a, b)
    torch.cuda.synchronize()
    for a, _ in bufs:
        assert np.array_equal(to_host(a), want)
    a, b = x.clone(), torch.empty_like(x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        there_and_back(a, b)
    for _ in range(5):
        g.replay()
    torch.cuda.synchronize()
    assert np.array_equal(to_host(a), want)
    assert bc_ntt.wait_status() == 0


@pytest.mark.parametrize("plan,log_b", [("2 8 8 8 1", 2), ("2 10 4 12 1", 1), ("2 4 8 9 1", 3)])
def test_lde_chains_in_a_graph_and_on_two_streams(gpu_ctx, plan, log_b):
    """The same for the fused LDE's kernels, the first of which leave their values in the last coset's block: both
    streams and the graph give the oracle's extension, over and over."""
    import torch

    import bc_ntt
    import oracle

    log_n = sum(int(k) for k in plan.split()[1::2])
    n, cols = 1 << log_n, 16 if log_n < 20 else 2
    old = bc_ntt.plan_table_export()
    words = [raw_u64(np.random.default_rng(s), cols * n) for s in range(2)]
    want = [np.asarray(oracle.lde(w, log_n, cols, n, log_b, threads=8)) for w in words]
    xs = [to_dev(w) for w in words]
    try:
        bc_ntt.plan_table_import(f"{log_n} {log_b} {plan}\n")
        names = kernel_names(lambda: bc_ntt.lde(xs[0], torch.empty(cols * n << log_b, dtype=torch.int64, device="cuda"),
                                                log_n, cols, log_b))
        assert len(names) == 3 and all("kernel_tc<" in k for k in names), names
        streams = [torch.cuda.Stream() for _ in xs]
        outs = [torch.zeros(cols * n << log_b, dtype=torch.int64, device="cuda") for _ in xs]
        torch.cuda.synchronize()
        for _ in range(10):
            for s, x, o in zip(streams, xs, outs):
                with torch.cuda.stream(s):
                    bc_ntt.lde(x, o, log_n, cols, log_b)
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert np.array_equal(to_host(o), w)
            o.zero_()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for x, o in zip(xs, outs):
                bc_ntt.lde(x, o, log_n, cols, log_b)
        for _ in range(3):
            g.replay()
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert np.array_equal(to_host(o), w)
        assert bc_ntt.wait_status() == 0
    finally:
        bc_ntt.plan_table_clear()
        if old:
            bc_ntt.plan_table_import(old)


@pytest.mark.parametrize("log_n,log_b", [(13, 1), (13, 2), (14, 1), (15, 3), (18, 1)])
def test_few_columns_with_tuned_plans(gpu_ctx, log_n, log_b):
    """Column counts on both sides of a low window's full tiles, where the plan in use changes."""
    import torch

    import bc_ntt
    import oracle

    old = bc_ntt.plan_table_export()
    try:
        assert bc_ntt.load_tuned_plans()
        for cols in (1, 2, 3, 5, 6, 11, 12, 17) if log_n < 16 else (1, 3, 4):
            n = 1 << log_n
            x = raw_u64(np.random.default_rng(100 * log_n + cols), cols * n)
            d, o = to_dev(x), torch.zeros(cols * n << log_b, dtype=torch.int64, device="cuda")
            bc_ntt.lde(d, o, log_n, cols, log_b)
            assert np.array_equal(to_host(o), oracle.lde(x, log_n, cols, n, log_b)), cols
    finally:
        bc_ntt.plan_table_clear()
        if old:
            bc_ntt.plan_table_import(old)


@pytest.mark.parametrize("log_n,cols,log_b,plan", [(12, 9, 0, "1 12 1"), (16, 9, 0, "2 8 8 8 1"), (14, 17, 1, "2 4 8 10 1"),
                                                   (16, 9, 3, "2 5 8 11 1"), (20, 5, 1, "3 4 8 8 8 8 1"),
                                                   (17, 16, 2, "2 8 8 9 1"), (22, 2, 1, "2 10 4 12 1")])
def test_waits_that_run_out_are_reported(gpu_ctx, log_n, cols, log_b, plan):
    """With a limit of no tries every wait for products runs out at once: the kernels end, say so, and hand their
    tensor memory on only when their products are done; with the default again, the next results are exact."""
    import torch

    import bc_ntt

    n = 1 << log_n
    x = to_dev(raw_u64(np.random.default_rng(log_n), cols * n))
    out, want = (torch.zeros(cols * n << log_b, dtype=torch.int64, device="cuda") for _ in range(2))

    def run(o):
        if log_b:
            bc_ntt.lde(x, o, log_n, cols, log_b)
        else:
            bc_ntt.batch_ntt_internal(x.data_ptr(), o.data_ptr(), log_n, cols, n, n, True, True, 0, 0)

    old = bc_ntt.plan_table_export()
    try:
        bc_ntt.plan_table_import(f"{log_n} {log_b} {plan}\n")
        run(want)
        assert bc_ntt.wait_status() == 0
        bc_ntt.set_wait_limit(0)
        for _ in range(3):
            run(out)
        assert bc_ntt.wait_status() == 1
        assert bc_ntt.wait_status() == 0
        bc_ntt.set_wait_limit()
        run(out)
        assert bc_ntt.wait_status() == 0
        assert torch.equal(out, want)
    finally:
        bc_ntt.set_wait_limit()
        bc_ntt.plan_table_clear()
        if old:
            bc_ntt.plan_table_import(old)


MODES = [(False, False), (False, True), (True, False), (True, True)]


@pytest.mark.parametrize("low", [8, 9, 10, 11, 12])
@pytest.mark.parametrize("bitrev,inverse", MODES)
def test_low_windows_below_a_top_window(gpu_ctx, low, bitrev, inverse):
    """The low windows with index prefixes, on the tensor cores but for the last pass of a natural -> bit-reversed
    inverse and the first of a scaled bit-reversed -> natural forward transform."""
    import bc_ntt

    plan, log_n, g = [(4, 8), (low, 1)], 4 + low, 1 << (12 - low)
    for cols in {1, max(1, 3 * g // 4), g, g + max(1, 3 * g // 4)}:
        _ntt(log_n, cols, bitrev, inverse, plan=plan)
        for ext in (0, 1):
            n = 1 << log_n
            d = to_dev(np.zeros(cols * n, dtype=np.uint64))
            names = kernel_names(lambda: bc_ntt.batch_ntt_with_plan(d, d, log_n, cols, n, n, bitrev, inverse, ext, ext, plan))
            filled = 4 * cols >= 3 * g * -(-cols // g)
            mixed = bitrev != inverse and (inverse or ext)
            assert any(k.startswith(f"pass_kernel_tc<{low},1") for k in names) == (filled and not mixed), (cols, ext)
    _ntt(log_n, g, bitrev, inverse, gap=3, plan=plan)
    if bitrev == inverse:
        _ntt(log_n, g, bitrev, inverse, ext=2, coset=3, gap=1, plan=plan)


def _windows(log_n, cols, bitrev, inverse, ext):
    """Windows of a plain transform's kernels, the largest first: t8 on the tensor cores, i8 on the integer kernels."""
    import torch

    import bc_ntt

    n = 1 << log_n
    d = torch.zeros(cols * n, dtype=torch.int64, device="cuda")
    names = kernel_names(lambda: bc_ntt.batch_ntt_internal(d.data_ptr(), d.data_ptr(), log_n, cols, n, n, bitrev, inverse,
                                                           ext, ext))
    return sorted((("t" if k.startswith("pass_kernel_tc") else "i") + k.split("<")[1].split(",")[0] for k in names),
                  key=lambda w: -int(w[1:]))


# calls on both sides of each rule that chooses a plan or a kernel: (log_n, columns, bitrev, inverse, coset), windows
ROUTES = [
    # one pass: forward on the integer kernels up to a size, inverse on the tensor cores where the tile is filled
    ((12, 16, 0, 0, 0), "i12"), ((12, 3000, 0, 0, 0), "t12"), ((11, 8000, 0, 0, 0), "i11"), ((12, 16, 1, 0, 0), "t12"),
    ((9, 8000, 1, 0, 0), "i9"), ((10, 400, 1, 0, 0), "i10"), ((10, 5000, 1, 0, 0), "t10"), ((12, 100, 0, 0, 1), "i12"),
    ((12, 200, 0, 0, 1), "t12"), ((12, 1, 1, 1, 0), "t12"), ((10, 2, 1, 1, 1), "i10"), ((10, 3, 1, 1, 1), "t10"),
    # low windows that the columns do or do not fill
    ((13, 16, 0, 0, 0), "t8 t5"), ((13, 5, 0, 0, 0), "i8 i5"), ((13, 3, 0, 0, 0), "i9 t4"), ((13, 1, 0, 0, 1), "i8 i5"),
    ((13, 1, 1, 1, 1), "i9 i4"), ((13, 3, 1, 1, 0), "i9 t4"), ((14, 4, 0, 0, 1), "t10 t4"), ((14, 5, 0, 0, 1), "i9 i5"),
    ((16, 3, 0, 0, 0), "t12 t4"), ((16, 5, 0, 0, 0), "t8 i8"), ((16, 5, 0, 0, 1), "t12 t4"), ((16, 16, 0, 0, 0), "t8 t8"),
    ((17, 5, 0, 0, 0), "t12 t5"), ((18, 16, 0, 0, 0), "t10 t8"), ((21, 3, 0, 0, 0), "t12 i9"), ((21, 3, 0, 0, 1), "t12 t9"),
    # a pass that keeps the integer kernel
    ((13, 12, 0, 1, 1), "i8 i5"), ((13, 12, 0, 1, 0), "i9 t4"), ((13, 12, 1, 0, 1), "i8 t5"), ((15, 3, 0, 1, 1), "i10 i5"),
    ((16, 3, 0, 1, 0), "t8 i8"), ((16, 3, 1, 0, 1), "t8 i8"), ((18, 33, 0, 1, 1), "i10 t8"), ((21, 3, 0, 1, 0), "i12 i9"),
    ((22, 3, 0, 1, 1), "i12 t10"),
]


@pytest.mark.parametrize("call,windows", ROUTES, ids=lambda x: "-".join(map(str, x)) if isinstance(x, tuple) else None)
def test_routes(gpu_ctx, call, windows):
    """The kernels that a call with built-in plans takes, and its result against the oracle's."""
    import bc_ntt

    log_n, cols, bitrev, inverse, ext = call
    old = bc_ntt.plan_table_export()
    try:
        bc_ntt.plan_table_clear()
        got = _windows(log_n, cols, bool(bitrev), bool(inverse), ext)
        assert sorted(got) == sorted(windows.split()), got
        if cols << log_n <= 1 << 21:
            _ntt(log_n, cols, bool(bitrev), bool(inverse), ext=ext, coset=ext)
    finally:
        if old:
            bc_ntt.plan_table_import(old)


def test_three_pass_routes(gpu_ctx):
    """The shipped table's three-pass plans at 21 bits: for full tiles, otherwise two passes."""
    import bc_ntt

    try:
        assert bc_ntt.load_tuned_plans()
        assert sorted(_windows(21, 16, False, False, 0)) == ["t4", "t8", "t9"]
        assert sorted(_windows(21, 12, False, False, 0)) == ["i9", "t12"]
        assert sorted(_windows(21, 16, False, True, 1)) == ["i9", "t4", "t8"]
        assert sorted(_windows(21, 12, False, True, 1)) == ["i12", "i9"]
    finally:
        bc_ntt.plan_table_clear()
