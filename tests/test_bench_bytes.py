"""bench.py's table of bytes per cell counts kernels that make one pass by what
that pass moves, not by the sum of the kernels it replaced."""
import bench


def test_one_pass_kernels_count_one_pass():
    kb = bench.KERNEL_BYTES
    # read u u0 Kx Ky, written u un
    assert kb["tea_leaf_jacobi_solve"] == 6 * 8
    # read sd u r Kx Ky, written sd u r; with the diagonal preconditioner also Mi
    assert kb["tea_leaf_ppcg_solve_inner_step"]["none"] == 8 * 8
    assert kb["tea_leaf_ppcg_solve_inner_step"]["jac_diag"] == 9 * 8


def test_instruction_counts_name_kernels_that_are_launched():
    launched = {w[7] for w in bench.WORKLOADS.values()} | set(bench.KERNEL_BYTES)
    assert {k for k, _, _ in bench.FP64_PER_CELL} <= launched
    assert not any(k == "tea_leaf_cheby_solve_calc_p" for k, _, _ in bench.FP64_PER_CELL)
