"""GPU tests of the plan table and the autotuner (bc_autotune, bc_plan_table_*)."""
import numpy as np
import pytest

import oracle
from conftest import kernel_names, raw_u64, to_dev, to_host

pytestmark = pytest.mark.gpu


def test_autotune_keeps_results_exact(gpu_ctx):
    import bc_ntt
    import torch

    bc_ntt.plan_table_clear()
    rng = np.random.default_rng(12)
    for log_n, log_b, cols in ((14, 1, 6), (17, 2, 3), (20, 0, 2), (21, 3, 2)):
        rep = bc_ntt.autotune(log_n, log_b, cols, reps=1)
        lines = rep.strip().splitlines()
        assert lines[-1].startswith("best ")
        assert len(lines) - 1 >= 8, rep  # window splits, then the launch knobs of the best one
        n = 1 << log_n
        x = raw_u64(rng, cols * n)
        if log_b:
            out = torch.empty(((1 << log_b) * cols) << log_n, dtype=torch.int64, device="cuda")
            bc_ntt.lde(to_dev(x), out, log_n, cols, log_b)
            exp = oracle.lde(x, log_n, cols, n, log_b, threads=8)
        else:
            out = torch.empty(cols * n, dtype=torch.int64, device="cuda")
            d = to_dev(x)
            bc_ntt.batch_ntt_internal(d.data_ptr(), out.data_ptr(), log_n, cols, n, n, False, False, 0, 0)
            exp = oracle.batch_ntt(x, log_n, cols, n, n, False, False, threads=8)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(to_host(out), exp, err_msg=f"log_n={log_n} blowup={1 << log_b}")
    bc_ntt.plan_table_clear()


def test_plan_table_roundtrip_and_validation(gpu_ctx):
    import bc_ntt

    bc_ntt.plan_table_clear()
    bc_ntt.plan_table_import("22 1 3 5 8 5 8 12 1\n16 0 2 8 8 8 1\n")
    text = bc_ntt.plan_table_export()
    assert "22 1 3 5 8 5 8 12 1" in text and "16 0 2 8 8 8 1" in text
    with pytest.raises(ValueError):
        bc_ntt.plan_table_import("22 1 2 10 4 11 1\n")  # bits do not sum to log_n
    with pytest.raises(ValueError):
        bc_ntt.plan_table_import("20 1 2 9 1 11 1\n")  # a run of 1 above bit 0
    # an imported three-pass plan is used and stays exact
    import torch

    rng = np.random.default_rng(3)
    x = raw_u64(rng, 2 << 22)
    out = torch.empty(4 << 22, dtype=torch.int64, device="cuda")
    bc_ntt.lde(to_dev(x), out, 22, 2, 1)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(to_host(out), oracle.lde(x, 22, 2, 1 << 22, 1, threads=8))
    bc_ntt.plan_table_clear()
    assert bc_ntt.plan_table_export() == ""


@pytest.mark.parametrize("log_n,split,integer", [(17, "5 8 12 1", False), (14, "5 8 9 1", True)])
@pytest.mark.parametrize("knobs", ["k 1 0 0 0 0", "k 32 2 0 0 0", "k 0 16 2 0 0", "k 0 0 3 0 0", "k 0 4 0 2 0",
                                   "k 0 0 0 1 3", "k 8 0 0 0 2", "k 4 2 3 2 3"])
def test_plan_knobs_stay_exact(gpu_ctx, knobs, log_n, split, integer):
    """Every launch knob the autotuner may pick -- column walks, top-window table mode and double-buffering, pass
    occupancy -- gives the oracle's result, for a fused LDE with an 8-column top window (where double-buffering
    applies) and for a plain NTT.  The first split runs on the tensor cores, which know the walks only; 5 columns do
    not fill the second one's 9-bit tiles, so that the integer kernels run with all of the knobs."""
    import bc_ntt
    import torch

    bc_ntt.plan_table_clear()
    bc_ntt.plan_table_import("".join(f"{log_n} {b} 2 {split} {knobs}\n" for b in (0, 1, 2)))
    assert knobs in bc_ntt.plan_table_export()
    rng = np.random.default_rng(31)
    cols = 5
    n = 1 << log_n
    x = raw_u64(rng, cols * n)
    d = to_dev(x)
    for log_b in (1, 2):
        out = torch.empty(((1 << log_b) * cols) << log_n, dtype=torch.int64, device="cuda")
        names = kernel_names(lambda: bc_ntt.lde(d, out, log_n, cols, log_b))
        assert len(names) == 3 and all(("kernel_tc<" in k) != integer for k in names), names
        bc_ntt.lde(d, out, log_n, cols, log_b)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(to_host(out), oracle.lde(x, log_n, cols, n, log_b, threads=8),
                                      err_msg=f"{knobs} blowup={1 << log_b}")
    out = torch.empty(cols * n, dtype=torch.int64, device="cuda")
    bc_ntt.batch_ntt_internal(d.data_ptr(), out.data_ptr(), log_n, cols, n, n, False, False, 0, 0)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(to_host(out), oracle.batch_ntt(x, log_n, cols, n, n, False, False, threads=8))
    bc_ntt.plan_table_clear()


def test_plan_knobs_validation(gpu_ctx):
    import bc_ntt

    bc_ntt.plan_table_clear()
    for bad in ("17 1 2 5 8 12 1 k 0 0 4 0 0\n", "17 1 2 5 8 12 1 k 0 0 0 3 0\n", "17 1 2 5 8 12 1 k 0 0 0 0 5\n",
                "17 1 2 5 8 12 1 k 1 2 3\n"):
        with pytest.raises(ValueError):
            bc_ntt.plan_table_import(bad)
    bc_ntt.plan_table_clear()


def test_callers_plans_run_as_they_are(gpu_ctx):
    """An imported or autotuned plan is used as it is, also for columns that do not fill its low window's tiles; only
    built-in plans and default entries may be fitted to the columns."""
    import bc_ntt
    import torch

    d = torch.zeros(16 << 13, dtype=torch.int64, device="cuda")
    out = torch.zeros(32 << 13, dtype=torch.int64, device="cuda")

    def windows(cols):
        """Window bits of the kernels of a fused LDE and of a plain transform."""
        lde = kernel_names(lambda: bc_ntt.lde(d, out, 13, cols, 1))
        ntt = kernel_names(lambda: bc_ntt.batch_ntt_internal(d.data_ptr(), out.data_ptr(), 13, cols, 1 << 13, 1 << 13,
                                                             False, False, 0, 0))
        return sorted(int(k.split("<")[1].split(",")[0]) for k in lde), sorted(
            int(k.split("<")[1].split(",")[0].rstrip(">")) for k in ntt)

    text = "13 0 2 5 8 8 1\n13 1 2 5 8 8 1\n"
    try:
        bc_ntt.plan_table_clear()
        bc_ntt.plan_table_import(text)
        for cols in (1, 5, 11, 16):  # 16 columns fill an 8-bit window's tile
            assert windows(cols) == ([5, 8, 8], [5, 8]), cols
        assert bc_ntt.plan_table_export() == text
        bc_ntt._check(bc_ntt.lib().bc_plan_table_import_defaults(text.encode()), "import_defaults")
        assert bc_ntt.plan_table_export() == text
        assert windows(16) == ([5, 8, 8], [5, 8])
        assert windows(11)[0] == [4, 9, 9]
        bc_ntt.autotune(13, 1, 5, reps=1)  # an entry measured at its column count replaces the default
        line = [x for x in bc_ntt.plan_table_export().splitlines() if x.startswith("13 1")][0].split()
        top, low = int(line[3]), int(line[5])
        assert windows(5)[0] == sorted([top, low, low])
        with pytest.raises(ValueError):
            bc_ntt._check(bc_ntt.lib().bc_plan_table_import_defaults(b"13 1 2 5 8 9 1\n"), "import_defaults")
    finally:
        bc_ntt.plan_table_clear()
